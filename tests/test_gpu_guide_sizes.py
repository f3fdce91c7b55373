"""The guiding network's entry points around the 128-row tiles of its kernels: dense query and output
rows of the forward pass, and the gradient / Adam reduction, whose sums have a fixed order."""
import numpy as np
import pytest

from bonsai_gb300 import gpu as G
from oracle import guide as OG

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(gpu_ctx):
    g = G.Guide(gpu_ctx, batch_size=1024, samples_per_pass=1 << 16)
    g.params = OG.init_params(5)
    yield g
    g.close()


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 257, 4097])
def test_forward_rows(net, n):
    # against the oracle with the same BF16 roundings: what is left is the order of FP32 sums and, where
    # one flips a BF16 rounding (2^-9), its effect: 2e-3 of the output's norm
    q = OG.random_samples(n, 3)[:, :9]
    p = OG.init_params(5)
    net.params = p
    out = net.forward(q)
    ref = OG.forward(p, q, bf16_sim=True)[0][:, :OG.OUT]
    assert out.shape == (n, OG.OUT)
    assert np.linalg.norm(out - ref) <= 2e-3 * np.linalg.norm(ref)
    # a row does not depend on the rows beside it
    assert np.array_equal(net.forward(q[:1])[0], out[0])


@pytest.mark.parametrize("n", [1, 127, 129, 1024, 1025, 3000])
def test_gradient_and_steps_repeat_bit_for_bit(net, n):
    s = OG.random_samples(n, 4)
    s[:, 13] = np.maximum(s[:, 13], 1e-3)
    p = OG.init_params(5)
    net.params = p
    g0, l0 = net.gradient(s)
    g1, l1 = net.gradient(s)
    assert np.array_equal(g0, g1) and l0 == l1
    ref_g, ref_l = OG.batch_loss_grad(p, s, bf16_sim=True)
    assert np.linalg.norm(g0 - ref_g) <= 2e-2 * np.linalg.norm(ref_g)
    # the loss: FP32 terms of magnitude <= |log q| summed to 1e-6 of their sum, BF16 effects as above
    assert abs(l0 - ref_l) <= 1e-2 * max(abs(ref_l), 1.0)
    net.train(s)
    a = net.params
    net.params = p
    net.train(s)
    # the pool order of a second epoch differs, so only a single batch takes the same step
    if n <= 1024:
        assert np.allclose(a, net.params, rtol=0, atol=2e-5)
