"""An epoch of several optimiser steps.

Training adds the slices of a batch's gradient as they arrive, so two trainings from equal weights and an
equal sample order are equal only as far as the last bit of a gradient carries: it may turn the BF16
rounding of a weight, and Adam's division by sqrt(v) makes whole steps of a change in a gradient near
zero.  Bounds: a step moves a parameter by lr |m^| / sqrt(v^); over the first few steps m^ is a mean of the
gradients with weights 0.9^k, v^ nearly their plain mean square, so by Cauchy-Schwarz |m^| <= 1.1 sqrt(v^) for up to
5 steps.  A training is within 1.2 lr a step of its start, two trainings within 2.4 lr of each other, and
most parameters, whose gradients are far from zero, differ by their rounding alone."""
import numpy as np
import pytest

from bonsai_gb300 import gpu as G
from oracle import guide as OG

pytestmark = pytest.mark.gpu

LR, BATCH = 1e-3, 512


@pytest.mark.parametrize("n", [129, 1025, 2048, 2500])  # 1, 3, 4 and 5 steps; the last of 129, 1, 512, 452 samples
def test_two_trainings_from_equal_weights(gpu_ctx, n):
    s = OG.random_samples(n, 21)
    p = OG.init_params(6)
    steps = -(-n // BATCH)
    out, losses = [], []
    for _ in range(2):
        g = G.Guide(gpu_ctx, batch_size=BATCH, samples_per_pass=4096, learning_rate=LR)
        try:
            g.params = p
            losses.append(g.train(s))
            out.append(g.params.astype(np.float64))
        finally:
            g.close()
    a, b = out
    moved = np.abs(a - p)
    assert 0.5 * LR <= moved.max() <= 1.2 * LR * steps
    assert (moved[p == 0.0] == 0.0).all()  # the padding stays zero
    d = np.abs(a - b)
    assert d.max() <= 2.4 * LR * steps
    assert np.median(d) <= 1e-6
    # the mean batch loss before each step: the weights' differences in second order
    assert abs(losses[0] - losses[1]) <= 1e-3 * max(abs(losses[0]), 1.0)
