// bg_shade_guided_full.cu - the guided shade launches of scenes with textures, an infinite light or
// emitting shapes (each resolved per scene at run time).
#include "bg_wave.cuh"

namespace bg {

int launch_shade_guided_full(const Scene& sc, const RenderParams& rp, const WaveBuffers& wb, const GuideWave& gw,
                             uint32_t b, uint32_t* err, uint32_t blocks, const ShadeFork* fork, cudaStream_t s) {
    return shade_launch<false, true, true, true, true>(sc, rp, wb, gw, b, err, nullptr, sc.cls_mask, blocks, fork, s);
}

}  // namespace bg
