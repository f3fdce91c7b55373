// bg_warp.cuh - warp-level queue helpers shared by the wavefront translation units.
#pragma once
#include "bg_shapes.cuh"

namespace bg {

constexpr unsigned FULL = 0xffffffffu;

BG_D uint32_t lane_id() { return threadIdx.x & 31u; }

BG_D uint32_t warp_fetch(uint32_t* head) {
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(head, 32u);
    return __shfl_sync(FULL, base, 0);
}
// Warp-aggregated append: every lane of the warp must call it; returns the slot of lanes with pred.
BG_D uint32_t warp_append(uint32_t* counter, bool pred) {
    uint32_t mask = __ballot_sync(FULL, pred);
    if (mask == 0) return 0;
    uint32_t leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane_id() == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
    base = __shfl_sync(FULL, base, leader);
    return base + (uint32_t)__popc(mask & ((1u << lane_id()) - 1u));
}

// Appends of a whole block to NQ queues with one atomic per queue: thread t enters counters[c]'s queue
// when pred[c], at pos[c].  Every thread of the block calls it (two barriers); the struct is the block's
// shared scratch, free again after the next barrier.  Queue counters are single addresses, and a counter
// takes about one atomic per nanosecond from the whole GPU: one per warp and queue bound the binning
// and most of the shading (2^20 Cornell box paths: binning 38 us a bounce, 3 us of memory traffic).
template <int NQ>
struct BlockAppend {
    uint32_t n[NQ][32];  // per queue and warp: lanes that append, then the warp's first position
    BG_D void operator()(uint32_t* const (&counters)[NQ], const bool (&pred)[NQ], uint32_t (&pos)[NQ]) {
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31u) >> 5;
        uint32_t mask[NQ];
#pragma unroll
        for (int c = 0; c < NQ; ++c) {
            mask[c] = __ballot_sync(FULL, pred[c]);
            if (lane == 0) n[c][warp] = __popc(mask[c]);
        }
        __syncthreads();
        for (uint32_t c = warp; c < (uint32_t)NQ; c += nwarps) {  // a warp scans a queue's counts
            const uint32_t own = lane < nwarps ? n[c][lane] : 0u;
            uint32_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, incl, o);
                if (lane >= (uint32_t)o) incl += t;
            }
            uint32_t base = 0;
            if (lane == 31 && incl) {
#pragma unroll
                for (int k = 0; k < NQ; ++k)
                    if (c == (uint32_t)k) base = atomicAdd(counters[k], incl);
            }
            base = __shfl_sync(FULL, base, 31);
            if (lane < nwarps) n[c][lane] = base + incl - own;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NQ; ++c) pos[c] = n[c][warp] + __popc(mask[c] & ((1u << lane) - 1u));
    }
};

// A block's threads grouped by key (0 .. NK - 1): returns the thread whose item this thread takes, so
// that warps hold one key each but for NK - 1 borders.  Every thread of the block calls it (three
// barriers); the struct is the block's shared scratch, free again after the next barrier.
template <int NK>
struct BlockGroup {
    uint32_t n[NK][32];
    uint16_t item[1024];
    BG_D uint32_t operator()(uint32_t key) {
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
        uint32_t own = 0;
#pragma unroll
        for (int k = 0; k < NK; ++k) {
            const uint32_t mask = __ballot_sync(FULL, key == (uint32_t)k);
            if (lane == 0) n[k][warp] = __popc(mask);
            if (key == (uint32_t)k) own = __popc(mask & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (warp == 0) {  // exclusive sums, key by key
            uint32_t base = 0;
            for (int k = 0; k < NK; ++k) {
                const uint32_t c = lane < nwarps ? n[k][lane] : 0u;
                uint32_t incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, incl, o);
                    if (lane >= (uint32_t)o) incl += t;
                }
                if (lane < nwarps) n[k][lane] = base + incl - c;
                base += __shfl_sync(FULL, incl, 31);
            }
        }
        __syncthreads();
        item[n[key][warp] + own] = (uint16_t)threadIdx.x;
        __syncthreads();
        return item[threadIdx.x];
    }
};

BG_D Ray load_ray(float4 o, float4 d) {
    Ray r;
    r.o = f4xyz(o);
    r.t_max = o.w;
    r.d = f4xyz(d);
    r.time = d.w;
    return r;
}

// Chained launches (launch_chained).  A kernel's last blocks let the next kernel's start where SMs
// become free; that kernel's blocks wait for this one's end, and for its writes, before they touch memory.
BG_D void allow_next() { cudaTriggerProgrammaticLaunchCompletion(); }
BG_D void wait_previous() { cudaGridDependencySynchronize(); }

// Launches a kernel that starts with wait_previous() behind the previous kernel of its stream: its
// blocks may come to the SMs that the previous one has left while that one still ends.  Path waves:
// extension and binning (the shade launches wait for events of several streams): a 67 x 49 preview
// 388 -> 357 us, 256 x 256 x 16 Cornell paths 1.669 -> 1.647 ms; a wave of many paths gains nothing,
// nor does a batch, whose graph's launches are short already (3.43 and 3.44 ms: launched plainly).
// Tree waves: extension and shadow rays, and no launch of its own for the counters' resets: 4096 Whitted
// samples 221 -> 182 us, direct lighting of 640 x 360 x 4 9.56 -> 9.48 ms.
template <class... P, class... Args>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, Args&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace bg
