// bg_shade_shapes.cu - single-scene shade launches for scenes whose light list holds emitting
// spheres or quadrics (and possibly the infinite light): variants with the general light code,
// textures resolved per scene at run time.
#include "bg_wave.cuh"

namespace bg {

int launch_shade_shapes(const Scene& sc, const RenderParams& rp, const WaveBuffers& wb, uint32_t b, uint32_t* err,
                        uint32_t blocks, const ShadeFork* fork, cudaStream_t s) {
    return shade_launch<false, false, true, true, true>(sc, rp, wb, GuideWave{}, b, err, nullptr, sc.cls_mask, blocks, fork, s);
}

}  // namespace bg
