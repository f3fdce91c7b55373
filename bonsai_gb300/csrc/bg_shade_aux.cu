// bg_shade_aux.cu - the shade launches of guided renders (training records, network mixtures) and
// of batch renders (per-path scenes).
#include "bg_wave.cuh"

namespace bg {

int launch_shade_guided(const Scene& sc, const RenderParams& rp, const WaveBuffers& wb, const GuideWave& gw, uint32_t b,
                        uint32_t* err, uint32_t blocks, const ShadeFork* fork, cudaStream_t s) {
    if (sc.ntex || general_lights(sc)) return launch_shade_guided_full(sc, rp, wb, gw, b, err, blocks, fork, s);
    return shade_launch<false, true, false, false, false>(sc, rp, wb, gw, b, err, nullptr, sc.cls_mask, blocks, fork, s);
}

int launch_shade_batch(const SceneRender* tab, const WaveBuffers& wb, uint32_t b, uint32_t* err, uint32_t mask,
                       uint32_t blocks, const ShadeFork* fork, cudaStream_t s, bool full) {
    const Scene sc{};
    const RenderParams rp{};
    const GuideWave gw{};
    // full: textures (matte, plastic) and the infinite light's next-event estimation, per scene
    if (full) return shade_launch<true, false, true, true, true>(sc, rp, wb, gw, b, err, tab, mask, blocks, fork, s);
    return shade_launch<true, false, false, false, false>(sc, rp, wb, gw, b, err, tab, mask, blocks, fork, s);
}

}  // namespace bg
