// bg_shade_plain.cu - the shade launches of single-scene wavefront renders, in the variants for
// textured scenes and for scenes whose light list holds the infinite light.
#include "bg_wave.cuh"

namespace bg {

int launch_shade_plain(const Scene& sc, const RenderParams& rp, const WaveBuffers& wb, uint32_t b, uint32_t* err,
                       uint32_t blocks, const ShadeFork* fork, cudaStream_t s) {
    const GuideWave gw{};
    if (sc.sph_emis || sc.quad_emis) return launch_shade_shapes(sc, rp, wb, b, err, blocks, fork, s);
    if (sc.inf) {  // the light list holds the infinite light
        if (sc.ntex) return shade_launch<false, false, true, true, false>(sc, rp, wb, gw, b, err, nullptr, sc.cls_mask, blocks, fork, s);
        return shade_launch<false, false, false, true, false>(sc, rp, wb, gw, b, err, nullptr, sc.cls_mask, blocks, fork, s);
    }
    if (sc.ntex) return shade_launch<false, false, true, false, false>(sc, rp, wb, gw, b, err, nullptr, sc.cls_mask, blocks, fork, s);
    return shade_launch<false, false, false, false, false>(sc, rp, wb, gw, b, err, nullptr, sc.cls_mask, blocks, fork, s);
}

}  // namespace bg
