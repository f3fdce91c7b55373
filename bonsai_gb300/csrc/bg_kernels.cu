// bg_kernels.cu - ray-query kernels and the PBRT wavefront stages.
//
// Wavefront (PBRT mode, 8-wide and 2-wide BVH):  one wave = up to `capacity` (pixel, sample) paths.
//   generate -> [extend -> bin -> shade -> shadow] x (max_depth + 1) -> film
// Queue sizes live in device memory; every stage launches a fixed persistent grid that reads its
// own work count, so the chain needs no host synchronisation and can be captured in a CUDA graph.
// Traversal stages pull rays for a warp's idle lanes from an atomic head (dynamic load balance);
// queues are compacted by whole blocks, one atomic per block and queue (BlockAppend).
//
// Renders over the reference layout (REF_COMPAT, and PBRT as a cross-check) run per path: bg_mega.cu.
#include "bg_guide.cuh"
#include "bg_guide_kernels.h"
#include "bg_kernels.h"
#include "bg_shading.cuh"
#include "bg_traverse.cuh"
#include "bg_warp.cuh"
#include "bg_wave.cuh"

namespace bg {


// ================================================================ ray queries
struct TraceSrc {
    const float4* rays;
    int2* hits;
    uint8_t* occ;
    BG_D Ray load(uint32_t i, int* skip) const {
        Ray r = load_ray(__ldg(&rays[2 * i]), __ldg(&rays[2 * i + 1]));
        r.time = 0.0f;
        *skip = -1;
        return r;
    }
    BG_D void store(uint32_t i, int prim, float t) const {
        if (occ) occ[i] = prim >= 0 ? 1 : 0;
        else hits[i] = make_int2(prim, __float_as_int(prim >= 0 ? t : INFINITY));
    }
};

// LAYOUT: 1 = reference binary layout, 2 = 2-wide, 8 = 8-wide compressed.
// Traversal kernels are compiled for 7 blocks of 128 threads per SM (72 registers): with 8 (64
// registers) they spill, with 6 (80) too few warps hide the node fetches.  Ray microbenchmark
// 12.84 ms against 14.37 with 8 and 14.05 with 6; production frame at 16 spp 106.7 / 109.1 / 110.7 ms.
#ifndef BG_MINBLOCKS
#define BG_MINBLOCKS 7
#endif
template <int LAYOUT, bool ANY>
__global__ void __launch_bounds__(128, BG_MINBLOCKS) k_trace(Scene sc, const float4* rays, uint32_t n, int2* hits, uint8_t* occ,
                                               uint32_t* err, unsigned long long* counters, uint32_t* head, int refill) {
    if constexpr (LAYOUT != 1) {
        TraceSrc src{rays, hits, ANY ? occ : nullptr};
#if BG_SMEM_STACK
        __shared__ uint2 stack8[STACK8 * 128];
#else
        uint2* stack8 = nullptr;
#endif
        if (LAYOUT == 8) traverse_queue8<ANY>(sc, n, head, src, err, refill, stack8);
        else traverse_queue<ANY>(sc, n, head, src, err, refill);
        return;
    } else {
        for (;;) {
            uint32_t base = warp_fetch(head);
            if (base >= n) break;
            uint32_t i = base + lane_id();
            if (i < n) {
                Ray ray = load_ray(__ldg(&rays[2 * i]), __ldg(&rays[2 * i + 1]));
                ray.time = 0.0f;
                int prim = ref_traverse<ANY>(sc, ray, err, counters);
                if (ANY) occ[i] = prim >= 0 ? 1 : 0;
                else hits[i] = make_int2(prim, __float_as_int(prim >= 0 ? ray.t_max : INFINITY));
            }
        }
    }
}

void launch_trace(const Scene& sc, bool ref_layout, bool any, const bg_ray* rays, size_t n, bg_hit* hits,
                  uint8_t* occluded, uint32_t* err, unsigned long long* counters, uint32_t* work_head,
                  const LaunchShape& ls, cudaStream_t s) {
    cudaMemsetAsync(work_head, 0, sizeof(uint32_t), s);
    dim3 grid(ls.sms * ls.blocks_per_sm), block(128);
    const float4* r = reinterpret_cast<const float4*>(rays);
    int2* h = reinterpret_cast<int2*>(hits);
    uint32_t nn = (uint32_t)n;
    const int layout = ref_layout ? 1 : (sc.nodes8 ? 8 : 2);
#define BG_TRACE(L, A) k_trace<L, A><<<grid, block, 0, s>>>(sc, r, nn, h, occluded, err, counters, work_head, ls.refill)
    if (layout == 1) {
        if (any) BG_TRACE(1, true);
        else BG_TRACE(1, false);
    } else if (layout == 2) {
        if (any) BG_TRACE(2, true);
        else BG_TRACE(2, false);
    } else {
        if (any) BG_TRACE(8, true);
        else BG_TRACE(8, false);
    }
#undef BG_TRACE
}

// Batch: item -> scene by binary search over the scenes' first items, then as above.
__global__ void k_generate_batch(const SceneRender* tab, uint32_t nscenes, WaveBuffers wb, uint64_t item0,
                                 uint32_t nitems) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        wb.counters[C_Q0] = nitems;
        wb.counters[C_EXT_HEAD] = 0;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nitems; i += gridDim.x * blockDim.x) {
        const uint64_t item = item0 + i;
        uint32_t lo = 0, hi = nscenes - 1;
        while (lo < hi) {  // last scene with item0 <= item
            uint32_t mid = (lo + hi + 1) >> 1;
            if (tab[mid].item0 <= item) lo = mid;
            else hi = mid - 1;
        }
        const SceneRender& sr = tab[lo];
        const uint64_t local = item - sr.item0;
        const uint64_t npix = (uint64_t)sr.rp.width * sr.rp.height;
        const uint32_t pix = (uint32_t)(local % npix);
        generate_one(sr.cam, sr.rp, wb, i, {pix % sr.rp.width, pix / sr.rp.width}, sr.rp.first_sample + (uint32_t)(local / npix));
        wb.scene_id[i] = lo;
    }
}


__global__ void k_generate(Camera cam, RenderParams rp, WaveBuffers wb, uint64_t item0, uint32_t nitems) {
    allow_next();
    generate_paths(cam, rp, wb, item0, nitems, rp.first_sample);
}

// Graph replay: the wave comes from wb.wavectl (advanced by k_wave_advance).
struct WaveItems {
    uint64_t item0;
    uint32_t n;
};
BG_D WaveItems wave_items(const WaveBuffers& wb, uint64_t total) {
    const uint64_t item0 = (uint64_t)wb.wavectl[0] * wb.capacity;
    return {item0, item0 >= total ? 0u : (uint32_t)min((uint64_t)wb.capacity, total - item0)};
}
__global__ void k_generate_ctl(Camera cam, RenderParams rp, WaveBuffers wb, uint64_t total) {
    allow_next();
    const WaveItems w = wave_items(wb, total);
    generate_paths(cam, rp, wb, w.item0, w.n, wb.wavectl[1]);
}

__global__ void k_wave_advance(WaveBuffers wb) {
    if (threadIdx.x == 0) wb.wavectl[0] += 1;
}

struct ExtendSrc {
    const uint32_t* q;
    WaveBuffers wb;
    const SceneRender* tab;
    BG_D Ray load(uint32_t i, int* skip) const {
        uint32_t slot = q[i];
        *skip = -1;
        return load_ray(wb.ray_o[slot], wb.ray_d[slot]);
    }
    BG_D const Scene* scene(uint32_t i) const { return &tab[wb.scene_id[q[i]]].sc; }
    BG_D void store(uint32_t i, int prim, float t) const { wb.hit[q[i]] = make_int2(prim, __float_as_int(t)); }
};

template <int LAYOUT, bool MULTI = false>
__global__ void __launch_bounds__(128, BG_MINBLOCKS) k_extend(Scene sc, WaveBuffers wb, uint32_t bounce, uint32_t* err,
                                                int refill, const SceneRender* tab, bool sorted) {
    allow_next();
    wait_previous();
    const uint32_t n = wb.counters[bounce & 1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&wb.ray_stats[0], (unsigned long long)n);
        wb.counters[(bounce + 1) & 1] = 0;
        wb.counters[C_SHADOW] = 0;
        wb.counters[C_SH_HEAD] = 0;
        for (int c = 0; c < NCLS; ++c) wb.counters[C_CLS + c] = 0;
    }
    ExtendSrc src{sorted ? wb.qsort : wb.queue[bounce & 1], wb, tab};
#if BG_SMEM_STACK
    __shared__ uint2 stack8[LAYOUT == 8 ? STACK8 * 128 : 1];
#else
    uint2* stack8 = nullptr;
#endif
    if (LAYOUT == 8) traverse_queue8<false, ExtendSrc, MULTI>(sc, n, &wb.counters[C_EXT_HEAD], src, err, refill, stack8);
    else traverse_queue<false>(sc, n, &wb.counters[C_EXT_HEAD], src, err, refill);
}

// ---- ray binning (BG_TUNE_SORT_RAYS): the extension queue of a bounce, counting-sorted by
// key = direction octant (3 bits) x Morton index of the origin's cell in an 8x8x8 grid over the
// scene bounds (9 bits).  Rays that leave the same region in the same octant then sit in the same
// warps and walk the same part of the tree.  hist: block-local shared-memory counts added to a
// global histogram; scan: one block turns it into bin cursors (and clears the histogram);
// scatter: each block reserves one range per (block, bin) and places its rays by local rank.
constexpr int SORT_BINS = 4096;
constexpr int SORT_K = 8;  // rays per thread per scatter chunk

BG_D uint32_t spread3(uint32_t v) {  // 3 bits -> every third bit
    return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4);
}
BG_D uint32_t ray_key(const WaveBuffers& wb, const RenderParams& rp, uint32_t slot) {
    const float4 o = wb.ray_o[slot], d = wb.ray_d[slot];
    const uint32_t oct = (d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u);
    const uint32_t cx = (uint32_t)rclamp((o.x - rp.bmin[0]) * rp.binv[0] * 8.0f, 0.0f, 7.0f);
    const uint32_t cy = (uint32_t)rclamp((o.y - rp.bmin[1]) * rp.binv[1] * 8.0f, 0.0f, 7.0f);
    const uint32_t cz = (uint32_t)rclamp((o.z - rp.bmin[2]) * rp.binv[2] * 8.0f, 0.0f, 7.0f);
    return (oct << 9) | (spread3(cx) << 2) | (spread3(cy) << 1) | spread3(cz);
}

__global__ void __launch_bounds__(256) k_sort_hist(WaveBuffers wb, RenderParams rp, uint32_t bounce) {
    __shared__ uint32_t h[SORT_BINS];
    for (int b = threadIdx.x; b < SORT_BINS; b += blockDim.x) h[b] = 0;
    __syncthreads();
    const uint32_t n = wb.counters[bounce & 1];
    const uint32_t* q = wb.queue[bounce & 1];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&h[ray_key(wb, rp, q[i])], 1u);
    __syncthreads();
    for (int b = threadIdx.x; b < SORT_BINS; b += blockDim.x)
        if (h[b]) atomicAdd(&wb.sort_hist[b], h[b]);
}

__global__ void __launch_bounds__(1024) k_sort_scan(WaveBuffers wb) {
    __shared__ uint32_t part[1024];
    constexpr int PER = SORT_BINS / 1024;
    uint32_t v[PER], sum = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        v[k] = wb.sort_hist[threadIdx.x * PER + k];
        sum += v[k];
    }
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {  // inclusive Hillis-Steele scan of the partial sums
        uint32_t x = threadIdx.x >= (unsigned)off ? part[threadIdx.x - off] : 0u;
        __syncthreads();
        part[threadIdx.x] += x;
        __syncthreads();
    }
    uint32_t base = part[threadIdx.x] - sum;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        wb.sort_hist[SORT_BINS + threadIdx.x * PER + k] = base;
        wb.sort_hist[threadIdx.x * PER + k] = 0;  // ready for the next bounce
        base += v[k];
    }
}

__global__ void __launch_bounds__(256) k_sort_scatter(WaveBuffers wb, RenderParams rp, uint32_t bounce) {
    __shared__ uint32_t h[SORT_BINS];
    const uint32_t n = wb.counters[bounce & 1];
    const uint32_t* q = wb.queue[bounce & 1];
    uint32_t* cursor = wb.sort_hist + SORT_BINS;
    const uint32_t chunk = blockDim.x * SORT_K;
    for (uint32_t c0 = blockIdx.x * chunk; c0 < n; c0 += gridDim.x * chunk) {
        for (int b = threadIdx.x; b < SORT_BINS; b += blockDim.x) h[b] = 0;
        __syncthreads();
        uint32_t key[SORT_K], rank[SORT_K], slot[SORT_K];
#pragma unroll
        for (int k = 0; k < SORT_K; ++k) {
            const uint32_t i = c0 + k * blockDim.x + threadIdx.x;
            key[k] = SORT_BINS;
            if (i < n) {
                slot[k] = q[i];
                key[k] = ray_key(wb, rp, slot[k]);
                rank[k] = atomicAdd(&h[key[k]], 1u);
            }
        }
        __syncthreads();
        for (int b = threadIdx.x; b < SORT_BINS; b += blockDim.x)
            if (h[b]) h[b] = atomicAdd(&cursor[b], h[b]);  // this block's range of bin b
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SORT_K; ++k)
            if (key[k] < SORT_BINS) {
                const uint32_t pos = h[key[k]] + rank[k];
                if (pos < n) wb.qsort[pos] = slot[k];
            }
        __syncthreads();
    }
}

// Material-key binning of this bounce's hits: one queue per material class plus misses, so each
// shade launch runs one material's code with uniform control flow.  GWK (guided waves, queries
// set): a hit of a guidable class (matte, plastic, conductor) also writes its network query at
// class * gw.cap + its queue position, for the inference that runs before shading.
constexpr uint32_t BIN_BLOCK = 512;
template <bool MULTI = false, bool GWK = false>
__global__ void __launch_bounds__(BIN_BLOCK) k_bin(Scene sc0, WaveBuffers wb, uint32_t bounce, const SceneRender* tab,
                                                   GuideWave gw = GuideWave{}, bool queries = false) {
    wait_previous();
    const uint32_t n = wb.counters[bounce & 1];
    const uint32_t* q = wb.queue[bounce & 1];
    const uint32_t stride = gridDim.x * blockDim.x;
    __shared__ BlockAppend<NCLS> append;
    if (blockIdx.x == 0 && threadIdx.x == 0) wb.counters[C_EXT_HEAD] = 0;  // for the next bounce
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        __syncthreads();
        const uint32_t i = base + threadIdx.x;
        int cls = -1;
        uint32_t slot = 0;
        if (i < n) {
            slot = q[i];
            int prim = wb.hit[slot].x;
            const Scene& sc = pick<MULTI>(sc0, MULTI ? &tab[wb.scene_id[slot]].sc : nullptr);
            cls = prim < 0 ? CLS_MISS : (int)sc.prim_cls[prim];
        }
        uint32_t qpos = 0, pos[NCLS];
        append({&wb.counters[C_CLS], &wb.counters[C_CLS + 1], &wb.counters[C_CLS + 2], &wb.counters[C_CLS + 3],
                &wb.counters[C_CLS + 4]},
               {cls == 0, cls == 1, cls == 2, cls == 3, cls == 4}, pos);
#pragma unroll
        for (int c = 0; c < NCLS; ++c) {
            if (cls == c) {
                wb.cls_queue[(size_t)c * wb.capacity + pos[c]] = slot;
                qpos = (uint32_t)c * gw.cap + pos[c];
            }
        }
        // one intersection per lane (outside the class loop, so the lanes of all three classes
        // run it together)
        if (GWK && queries && cls >= 0 && cls <= 2 && qpos - (uint32_t)cls * gw.cap < gw.cap) {
            const Ray ray = load_ray(wb.ray_o[slot], wb.ray_d[slot]);
            Isect it;
            GuideQuery gq{make_float4(0.5f, 0.5f, 0.5f, 0.0f), make_float4(0.0f, 1.0f, 0.0f, 0.0f),
                          make_float4(1.0f, 0.0f, 0.0f, 0.0f)};
            if (prim_isect<true>(sc0, wb.hit[slot].x, ray, &it)) gq = make_query(gw, it, -ray.d);
            float4* o = gw.query + 3 * (size_t)qpos;
            o[0] = gq.a;
            o[1] = gq.b;
            o[2] = gq.c;
        }
    }
}

struct ShadowSrc {
    WaveBuffers wb;
    const SceneRender* tab;
    BG_D const Scene* scene(uint32_t i) const { return &tab[wb.scene_id[wb.sh_ref[i] >> 1]].sc; }
    BG_D Ray load(uint32_t i, int* skip) const {
        float4 o = wb.sh_o[i], d = wb.sh_d[i];
        Ray ray;
        ray.o = f4xyz(o);
        ray.t_max = o.w;
        ray.d = f4xyz(d);
        ray.time = 0.0f;
        *skip = __float_as_int(d.w);
        return ray;
    }
    BG_D void store(uint32_t i, int prim, float) const {
        if (prim < 0) wb.pending[wb.sh_ref[i]].w = 1.0f;
    }
};

template <int LAYOUT, bool MULTI = false>
__global__ void __launch_bounds__(128, BG_MINBLOCKS) k_shadow(Scene sc, WaveBuffers wb, uint32_t* err, int refill,
                                                              const SceneRender* tab) {
    allow_next();
    const uint32_t n = min(wb.counters[C_SHADOW], wb.sh_capacity);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&wb.ray_stats[1], (unsigned long long)n);
    ShadowSrc src{wb, tab};
#if BG_SMEM_STACK
    __shared__ uint2 stack8[LAYOUT == 8 ? STACK8 * 128 : 1];
#else
    uint2* stack8 = nullptr;
#endif
    if (LAYOUT == 8) traverse_queue8<true, ShadowSrc, MULTI>(sc, n, &wb.counters[C_SH_HEAD], src, err, refill, stack8);
    else traverse_queue<true>(sc, n, &wb.counters[C_SH_HEAD], src, err, refill);
}

// Recording waves, once all paths have ended: the records of the paths whose last vertex left a
// light contribution pending (the others' were emitted when they ended) become training samples.
__global__ void __launch_bounds__(128) k_emit_pending(Scene sc, WaveBuffers wb, GuideWave gw, uint32_t n) {
    for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < n; base += gridDim.x * blockDim.x) {
        const uint32_t slot = base + lane_id();
        uint32_t nrec = 0, bounce = 0;
        bool lrec = false;
        RGB L = rgb(0.0f);
        if (slot < n) {
            const uint32_t state = wb.state[slot];
            if (state & ST_PENDING) {
                const float4 l4 = wb.L[slot];
                L = apply_pending(wb, slot, rgb(l4.x, l4.y, l4.z), state, sc.nlights);
                nrec = rec_count(state);
                bounce = state & 0xFFu;
                lrec = (state & ST_LREC) && wb.pending[2 * slot].w != 0.0f;
            }
        }
        emit_records(gw, wb, slot, nrec, L);
        emit_light_record(gw, bounce, slot, lrec);
    }
}

// The slots of a wave that hold thread slot i's film: [first, end), npix pixels in turn; `parts` threads share
// a pixel (film_parts).
struct FilmSpan {
    uint64_t first, end, npix;
    uint32_t parts;
};
template <bool MULTI>
BG_D FilmSpan film_span(const RenderParams& rp, const SceneRender* sr, uint64_t item0, uint32_t n) {
    FilmSpan f{0, n, (uint64_t)rp.width * rp.height, 1u};
    if (MULTI) {
        const uint64_t s0 = sr->item0, s1 = s0 + f.npix * rp.spp;
        f.first = s0 > item0 ? s0 - item0 : 0;
        f.end = min((uint64_t)n, s1 - item0);
    }
    if (rp.spp >= FILM_SPLIT) f.parts = film_parts(f.npix, f.end - f.first);
    return f;
}

// Adds a wave's paths (items item0 .. item0 + n - 1 in slots 0 .. n - 1) to the film: their radiance
// in L plus the last vertex's light contribution where its shadow rays have just resolved it, after
// the radiance sanity checks of SamplerIntegrator::render (src/base/integrator.rs:91-120;
// FilmTile::add_sample with the box filter, weight 1 to the sample's own pixel).  One thread adds all
// of the wave's samples of a pixel, in sample order and without atomics (six FP64 atomics and one
// integer one per path before: the Cornell box's contended 2^20 samples 0.12 ms of 1.86).  Where that
// leaves few threads with many samples each, `parts` threads share a pixel (film_parts): thread
// slot i takes samples i, i + width, ... (width = npix * parts), and k_film_parts adds their sums, which stay
// in slots of the ended paths' ray and throughput arrays until then.
// CTL: the wave is wb.wavectl's of `total` items.  MULTI: pixels and films of the path's scene.
template <bool MULTI, bool CTL>
__global__ void __launch_bounds__(256) k_film(Scene sc0, RenderParams rp0, FilmBuffers film0, WaveBuffers wb,
                                              uint64_t item0, uint32_t n, uint64_t total, const SceneRender* tab) {
    if (CTL) {
        const WaveItems w = wave_items(wb, total);
        item0 = w.item0;
        n = w.n;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const SceneRender* sr = MULTI ? tab + wb.scene_id[i] : nullptr;
        const FilmSpan span = film_span<MULTI>(pick<MULTI>(rp0, MULTI ? &sr->rp : nullptr), sr, item0, n);
        const uint64_t width = span.npix * span.parts;
        if (i - span.first >= width) {  // a later sample of its pixel
            if (MULTI) continue;
            break;
        }
        const uint32_t nlights = pick<MULTI>(sc0, MULTI ? &sr->sc : nullptr).nlights;
        const FilmBuffers& f = pick<MULTI>(film0, MULTI ? &sr->film : nullptr);
        double s[3] = {0.0, 0.0, 0.0}, q[3] = {0.0, 0.0, 0.0};
        float ps[3] = {0.0f, 0.0f, 0.0f};
        uint32_t cnt = 0, nan = 0;
        // four samples' loads in flight
        for (uint64_t j0 = i; j0 < span.end; j0 += 4 * width) {
            float4 l4[4];
            uint32_t st[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t j = j0 + k * width;
                if (j < span.end) {
                    l4[k] = wb.L[j];
                    st[k] = wb.state[j];
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t j = j0 + k * width;
                if (j >= span.end) break;
                RGB L = apply_pending(wb, (uint32_t)j, rgb(l4[k].x, l4[k].y, l4[k].z), st[k], nlights);
                const float y = luminance(L);
                if (is_nan(L) || y < -1e-5f || isinf(y)) {
                    L = rgb(0.0f);
                    ++nan;
                }
                const double r = L.r, g = L.g, b = L.b;
                s[0] += r;
                s[1] += g;
                s[2] += b;
                q[0] += r * r;
                q[1] += g * g;
                q[2] += b * b;
                ps[0] += L.r;
                ps[1] += L.g;
                ps[2] += L.b;
                ++cnt;
            }
        }
        if (nan) atomicAdd(f.nan_count, (unsigned long long)nan);
        if (span.parts > 1) {
            reinterpret_cast<double2*>(wb.ray_o)[i] = make_double2(s[0], s[1]);
            reinterpret_cast<double2*>(wb.ray_d)[i] = make_double2(s[2], q[0]);
            reinterpret_cast<double2*>(wb.beta)[i] = make_double2(q[1], q[2]);
            if (f.pass) {
                float* o = reinterpret_cast<float*>(wb.cls_queue) + 3 * (size_t)i;  // 5 words per slot
                o[0] = ps[0];
                o[1] = ps[1];
                o[2] = ps[2];
            }
            continue;
        }
        const size_t pix = wb.pixel[i];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f.sum[3 * pix + c] += s[c];
            f.sumsq[3 * pix + c] += q[c];
            if (f.pass) f.pass[3 * pix + c] += ps[c];
        }
        f.count[pix] += cnt;
    }
}

// Adds the sums that the threads sharing a pixel have left behind, in their order.
template <bool MULTI, bool CTL>
__global__ void __launch_bounds__(256) k_film_parts(RenderParams rp0, FilmBuffers film0, WaveBuffers wb, uint64_t item0,
                                                    uint32_t n, uint64_t total, const SceneRender* tab) {
    if (CTL) {
        const WaveItems w = wave_items(wb, total);
        item0 = w.item0;
        n = w.n;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const SceneRender* sr = MULTI ? tab + wb.scene_id[i] : nullptr;
        const FilmSpan span = film_span<MULTI>(pick<MULTI>(rp0, MULTI ? &sr->rp : nullptr), sr, item0, n);
        if (span.parts == 1 || i - span.first >= span.npix) {
            if (MULTI) continue;
            break;
        }
        const FilmBuffers& f = pick<MULTI>(film0, MULTI ? &sr->film : nullptr);
        double s[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        float ps[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll 4
        for (uint32_t p = 0; p < span.parts; ++p) {
            const size_t j = i + p * span.npix;
            const double2 a = reinterpret_cast<const double2*>(wb.ray_o)[j], b = reinterpret_cast<const double2*>(wb.ray_d)[j],
                          c = reinterpret_cast<const double2*>(wb.beta)[j];
            s[0] += a.x;
            s[1] += a.y;
            s[2] += b.x;
            s[3] += b.y;
            s[4] += c.x;
            s[5] += c.y;
            if (f.pass) {
                const float* o = reinterpret_cast<const float*>(wb.cls_queue) + 3 * j;
                ps[0] += o[0];
                ps[1] += o[1];
                ps[2] += o[2];
            }
        }
        const size_t pix = wb.pixel[i];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f.sum[3 * pix + c] += s[c];
            f.sumsq[3 * pix + c] += s[3 + c];
            if (f.pass) f.pass[3 * pix + c] += ps[c];
        }
        f.count[pix] += (uint32_t)((span.end - i + span.npix - 1) / span.npix);
    }
}

// A wave's film launches (n = the paths of a full wave); returns their number.  split: some scene's
// pixels may be shared by several threads.
template <bool MULTI, bool CTL>
static int launch_film(const Scene& sc, const RenderParams& rp, const FilmBuffers& film, const WaveBuffers& wb,
                       uint64_t item0, uint32_t n, uint64_t total, const SceneRender* tab, bool split,
                       const LaunchShape& ls, cudaStream_t s) {
    k_film<MULTI, CTL><<<ls.sms * 8, 256, 0, s>>>(sc, rp, film, wb, item0, n, total, tab);
    if (!split) return 1;
    k_film_parts<MULTI, CTL><<<ls.sms * 8, 256, 0, s>>>(rp, film, wb, item0, n, total, tab);
    return 2;
}

static int launch_bounces(const Scene& sc, const RenderParams& rp, const WaveBuffers& wb, uint32_t* err,
                          const LaunchShape& ls, cudaStream_t s, cudaEvent_t* ev, const GuideWave* gwp) {
    int launches = 0;
    dim3 grid(ls.sms * ls.blocks_per_sm), block(128);
    const dim3 bin_grid(ls.sms * 4);  // 2048 threads per SM
    const uint32_t shade_blocks = 2 * (uint32_t)ls.sms;  // one resident, one to even out the tail
    const GuideWave gw = gwp ? *gwp : GuideWave{};
    const bool guided = (gw.flags & GW_GUIDED) != 0;
    for (uint32_t b = 0; b <= rp.max_depth; ++b) {
        if (ev) cudaEventRecord(ev[4 * b + 0], s);
        const bool sorted = ls.sort_rays && b > 0 && wb.qsort;
        if (sorted) {
            k_sort_hist<<<ls.sms * 4, 256, 0, s>>>(wb, rp, b);
            k_sort_scan<<<1, 1024, 0, s>>>(wb);
            k_sort_scatter<<<ls.sms * 4, 256, 0, s>>>(wb, rp, b);
            launches += 3;
        }
        if (sc.nodes8) launch_chained(k_extend<8>, grid, block, s, sc, wb, b, err, ls.refill, nullptr, sorted);
        else launch_chained(k_extend<2>, grid, block, s, sc, wb, b, err, ls.refill, nullptr, sorted);
        const bool queries = guided && b < rp.max_depth;
        if (queries) {
            // every hit of a guidable class queues its network query; the network's mixtures are
            // ready before the shade launches
            launch_chained(k_bin<false, true>, bin_grid, BIN_BLOCK, s, sc, wb, b, nullptr, gw, true);
            launch_guide_infer(gw.wpack, gw.query, &wb.counters[C_CLS], 3, gw.cap, gw.raw, true, err, ls.sms, s);
            launches += 1;
        } else {
            launch_chained(k_bin<>, bin_grid, BIN_BLOCK, s, sc, wb, b, nullptr, GuideWave{}, false);
        }
        if (ev) cudaEventRecord(ev[4 * b + 1], s);
        if (gw.flags) launches += launch_shade_guided(sc, rp, wb, gw, b, err, shade_blocks, ls.fork, s);
        else launches += launch_shade_plain(sc, rp, wb, b, err, shade_blocks, ls.fork, s);
        if (ev) cudaEventRecord(ev[4 * b + 2], s);
        if (b < rp.max_depth) {  // the last hits sample no light
            if (sc.nodes8) k_shadow<8><<<grid, block, 0, s>>>(sc, wb, err, ls.refill, nullptr);
            else k_shadow<2><<<grid, block, 0, s>>>(sc, wb, err, ls.refill, nullptr);
            launches += 1;
        }
        if (ev) cudaEventRecord(ev[4 * b + 3], s);
        launches += 2;
    }
    return launches;
}

int launch_wave(const Scene& sc, const Camera& cam, const RenderParams& rp, const FilmBuffers& film,
                const WaveBuffers& wb, uint64_t item0, uint32_t nitems, uint32_t* err, const LaunchShape& ls,
                cudaStream_t s, cudaEvent_t* ev, const GuideWave* gw) {
    dim3 grid(ls.sms * ls.blocks_per_sm), block(128);
    k_generate<<<grid, block, 0, s>>>(cam, rp, wb, item0, nitems);
    int launches = 1 + launch_bounces(sc, rp, wb, err, ls, s, ev, gw);
    if (gw && (gw->flags & GW_RECORD)) {
        k_emit_pending<<<grid, block, 0, s>>>(sc, wb, *gw, nitems);
        launches += 1;
    }
    const bool split = rp.spp >= FILM_SPLIT && film_parts((uint64_t)rp.width * rp.height, nitems) > 1;
    return launches + launch_film<false, false>(sc, rp, film, wb, item0, nitems, 0, nullptr, split, ls, s);
}

int launch_wave_batch(const SceneRender* tab, uint32_t nscenes, uint32_t max_depth, const WaveBuffers& wb,
                      uint64_t item0, uint32_t nitems, uint32_t* err, const LaunchShape& ls, cudaStream_t s,
                      uint32_t variants) {
    dim3 grid(ls.sms * ls.blocks_per_sm), block(128);
    const Scene sc{};
    const RenderParams rp{};
    const FilmBuffers film{};
    const dim3 bin_grid(ls.sms * 4);
    k_generate_batch<<<grid, block, 0, s>>>(tab, nscenes, wb, item0, nitems);
    int launches = 1;
    for (uint32_t b = 0; b <= max_depth; ++b) {
        k_extend<8, true><<<grid, block, 0, s>>>(sc, wb, b, err, ls.refill, tab, false);
        k_bin<true><<<bin_grid, BIN_BLOCK, 0, s>>>(sc, wb, b, tab);
        launches += 2 + launch_shade_batch(tab, wb, b, err, (variants >> 2) & 15u, 2 * (uint32_t)ls.sms, ls.fork, s, (variants & 3u) != 0);
        if (b < max_depth) {
            k_shadow<8, true><<<grid, block, 0, s>>>(sc, wb, err, ls.refill, tab);
            launches += 1;
        }
    }
    return launches + launch_film<true, false>(sc, rp, film, wb, item0, nitems, 0, tab, (variants & 64u) != 0, ls, s);
}

int launch_wave_chain(const Scene& sc, const Camera& cam, const RenderParams& rp, const FilmBuffers& film,
                      const WaveBuffers& wb, uint64_t total, uint32_t* err, const LaunchShape& ls, cudaStream_t s) {
    dim3 grid(ls.sms * ls.blocks_per_sm), block(128);
    k_generate_ctl<<<grid, block, 0, s>>>(cam, rp, wb, total);
    int n = 2 + launch_bounces(sc, rp, wb, err, ls, s, nullptr, nullptr);
    const uint64_t full = std::min<uint64_t>(total, wb.capacity);
    const bool split = rp.spp >= FILM_SPLIT && film_parts((uint64_t)rp.width * rp.height, full) > 1;
    n += launch_film<false, true>(sc, rp, film, wb, 0, 0, total, nullptr, split, ls, s);
    k_wave_advance<<<1, 32, 0, s>>>(wb);
    return n;
}

// ================================================================ film
__global__ void k_resolve(FilmBuffers f) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < f.npix; p += gridDim.x * blockDim.x) {
        // merge_film_tile's rgb_to_xyz (film.rs:138-154) then write_image (film.rs:156-202)
        float r = (float)f.sum[3 * p], g = (float)f.sum[3 * p + 1], b = (float)f.sum[3 * p + 2];
        float X = 0.412453f * r + 0.357580f * g + 0.180423f * b;
        float Y = 0.212671f * r + 0.715160f * g + 0.072169f * b;
        float Z = 0.019334f * r + 0.119193f * g + 0.950227f * b;
        float o0 = 3.240479f * X - 1.537150f * Y - 0.498535f * Z;
        float o1 = -0.969256f * X + 1.875991f * Y + 0.041556f * Z;
        float o2 = 0.055648f * X - 0.204043f * Y + 1.057311f * Z;
        float w = (float)f.count[p];
        if (w != 0.0f) {
            float inv = 1.0f / w;
            o0 = fmaxf(o0 * inv, 0.0f);
            o1 = fmaxf(o1 * inv, 0.0f);
            o2 = fmaxf(o2 * inv, 0.0f);
        }
        f.rgb[3 * p] = o0;
        f.rgb[3 * p + 1] = o1;
        f.rgb[3 * p + 2] = o2;
    }
}

void launch_resolve(const FilmBuffers& film, cudaStream_t s) {
    k_resolve<<<(film.npix + 255) / 256, 256, 0, s>>>(film);
}

void launch_clear_film(const FilmBuffers& film, cudaStream_t s) {
    cudaMemsetAsync(film.sum, 0, sizeof(double) * 3 * film.npix, s);
    cudaMemsetAsync(film.sumsq, 0, sizeof(double) * 3 * film.npix, s);
    cudaMemsetAsync(film.count, 0, sizeof(uint32_t) * film.npix, s);
}

}  // namespace bg
