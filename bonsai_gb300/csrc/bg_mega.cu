// bg_mega.cu - PathIntegrator::radiance (src/integrators/path.rs:51-146) with one thread per path over
// the reference-layout BVH: the REF_COMPAT path and a cross-check of the wavefront in PBRT mode.
//
// The kernel is bound by instruction fetch: its code is far larger than the instruction caches and
// one thread reuses little of it.  So the threads of a block (all of an SM's) go through the bounce
// together: a bounce is a sequence of phases (closest hit; interaction, BSDF and light sample; shadow
// ray; second strategy; its ray; continuation) with a barrier between them, each phase's code is
// fetched once for 32 warps, and a thread whose path has ended starts its next one at the top of the
// loop instead of idling until its warp is done.  Cornell box 256x256, 16 spp, REF_COMPAT: 30.3 ms
// with independent threads (232 registers), 9.4 / 4.8 / 4.0 / 3.9 ms with blocks of 256 / 512 / 768 /
// 1024; 6.2 instead of 4.8 ms where spheres are tested with their intervals.
#include "bg_estimate.cuh"
#include "bg_film.cuh"
#include "bg_kernels.h"
#include "bg_shading.cuh"
#include "bg_traverse.cuh"

namespace bg {

namespace {

constexpr uint32_t MEGA_BLOCK = 1024;

// Out of line where a bounce uses them more than once: one copy in the instruction cache.
#define BG_CALL static __device__ __noinline__
template <bool ANY>
BG_CALL int mega_trace(const Scene& sc, Ray& ray, uint32_t* err) {
    return ref_traverse<ANY, false>(sc, ray, err, nullptr);
}
BG_CALL bool mega_isect(const Scene& sc, int prim, const Ray& ray, Isect* it, SurfaceGeom* g = nullptr) {
    return prim_isect(sc, prim, ray, it, g);
}
template <bool REF>
BG_CALL BxSample mega_sample(const BSDF& b, V3 wo, float u0, float u1, uint8_t type) {
    return b.sample<REF>(wo, u0, u1, type);
}
BG_CALL RGB mega_inf_radiance(const Scene& sc, V3 dir) { return inf_radiance(sc, dir); }

}  // namespace

// `rd`: the camera ray's differentials (textured scenes), which the path keeps in REF mode (the ray
// never re-spawns, F1) and only has at the first hit in PBRT mode.
template <bool REF>
__global__ void __launch_bounds__(MEGA_BLOCK, 1) k_megakernel(const __grid_constant__ Scene sc,
                                                              const __grid_constant__ Camera cam,
                                                              const __grid_constant__ RenderParams rp, FilmBuffers film,
                                                              uint32_t* err) {
    const uint64_t npix = (uint64_t)rp.width * rp.height;
    const uint64_t total = npix * rp.spp;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint64_t item = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool alive = false;
    uint32_t pix = 0, bounces = 0;
    Rng rng{0, 0, rp.seed};
    SamplerCalls calls{rp.strat, REF, 0, 0, rp.seed, 1u, 2u};
    Ray ray;
    RayDiff rd;
    RGB out = rgb(0.0f), beta = rgb(0.0f);
    bool specular_bounce = false;
    float eta_scale = 1.0f;
    const uint8_t flags = BSDF_ALL & ~BSDF_SPECULAR;
    for (;;) {
        if (!alive && item < total) {
            pix = (uint32_t)(item % npix);
            const uint32_t s = rp.first_sample + (uint32_t)(item / npix);
            item += stride;
            rng = Rng{pix, s, rp.seed};
            const CameraUs cu = camera_us(rp.strat, REF, rng, cam.lens_radius > 0.0f);
            const float fx = (float)(pix % rp.width) + cu.fx, fy = (float)(pix / rp.width) + cu.fy;
            ray = camera_ray(cam, fx, fy, cu.time, cu.lx, cu.ly);
            if (sc.ntex) rd = camera_diff(cam, fx, fy, ray, rp.diff_scale, cu.lx, cu.ly);
            calls.pix = rng.pixel;  // its calls after the camera sample's
            calls.sample = rng.sample;
            calls.k1 = 1u;
            calls.k2 = 2u;
            out = rgb(0.0f);
            beta = rgb(1.0f);
            specular_bounce = false;
            eta_scale = 1.0f;
            bounces = 0;
            alive = true;
        }
        if (!__syncthreads_or(alive)) break;
        // closest hit
        const Ray traced = ray;
        int prim = -1;
        if (alive) prim = mega_trace<false>(sc, ray, err);  // sets ray.t_max to the hit
        __syncthreads();
        // interaction, emission, BSDF, light sample
        bool nee = false, shadow = false, ended = false;
        Isect it;
        BSDF bsdf;
        float u[8], lpdf = 1.0f, scattering_pdf = 0.0f;
        uint32_t light_prim = 0;
        RGB f = rgb(0.0f), ld = rgb(0.0f);
        LightSample ls;
        Ray sr;
        if (alive) {
            bool hit = prim >= 0;
            if (hit) hit = mega_isect(sc, prim, traced, &it);
            if (bounces == 0 || specular_bounce) {
                if (hit) out = out + beta * emitted_radiance(sc, it, -ray.d);
                else if (prim < 0 && sc.inf) out = out + beta * mega_inf_radiance(sc, ray.d);
            }
            ended = !hit || bounces >= rp.max_depth;
            if (!ended) {
                TexPoint tp;
                const TexPoint* tpp = nullptr;
                if (sc.ntex && material_textured(sc.mats[prim_material(sc, it.prim)])) {
                    Isect tmp;
                    if (!mega_isect(sc, it.prim, traced, &tmp, &tp.g)) tp.g = SurfaceGeom{};
                    tp.p = it.p;
                    tp.n = it.n;
                    tp.d = compute_differentials(it.p, it.n, tp.g, (REF || bounces == 0) ? &rd : nullptr);
                    tpp = &tp;
                }
                bsdf = make_bsdf<-1, REF>(sc, it, tpp);
                const uint32_t base = DIM_BOUNCE0 + DIMS_PER_BOUNCE * bounces;
                rng.block(base, u);
                rng.block(base + 4, u + 4);
                nee = bsdf.num_components(flags) > 0 && sc.nlights > 0;
                if (nee) {
                    calls.get_1d(u[BD_LIGHT]);
                    calls.get_2d(u[BD_ULIGHT], u[BD_ULIGHT + 1]);
                    calls.get_2d(u[BD_USCAT], u[BD_USCAT + 1]);
                    const float count = (float)sc.nlights;
                    light_prim = sc.light_prims[(uint32_t)rmin(u[BD_LIGHT] * count, count - 1.0f)];
                    lpdf = 1.0f / count;
                    // estimate_direct (src/base/integrator.rs:330-437)
                    ls = light_sample_any<REF>(sc, light_prim, it, u[BD_ULIGHT], u[BD_ULIGHT + 1]);
                    if (ls.pdf > 0.0f && !is_black(ls.radiance)) {
                        f = bsdf.f<REF>(it.wo, ls.wi, flags) * abs_dot(ls.wi, it.ns);
                        scattering_pdf = bsdf.pdf<REF>(it.wo, ls.wi, flags);
                        if (!is_black(f)) {
                            sr = spawn_ray_to(it.p, it.p_err, it.n, it.time, ls.pt.p, ls.pt.p_err, ls.pt.n);
                            shadow = true;
                        }
                    }
                }
            }
        }
        __syncthreads();
        if (shadow && mega_trace<true>(sc, sr, err) < 0) {
            const float w = power_heuristic(1.0f, ls.pdf, 1.0f, scattering_pdf);
            ld = ld + f * ls.radiance * w / ls.pdf;
        }
        __syncthreads();
        // second strategy
        bool second = false;
        V3 wdir;
        float spdf = 0.0f, w2 = 1.0f;
        if (nee) {
            const BxSample bs = mega_sample<REF>(bsdf, it.wo, u[BD_USCAT], u[BD_USCAT + 1], flags);
            f = bs.f * abs_dot(bs.wi, it.ns);
            const bool sampled_specular = (bs.stype & BSDF_SPECULAR) != 0;
            // REF (F2): ray along the light sample's direction with the light half's pdf, any emitter
            wdir = REF ? ls.wi : bs.wi;
            spdf = REF ? scattering_pdf : bs.pdf;
            if (!is_black(f) && spdf > 0.0f) {
                second = true;
                if (!sampled_specular) {
                    const float p = light_pdf_any<REF>(sc, light_prim, it, wdir, nullptr);
                    if (p == 0.0f) second = false;
                    else w2 = power_heuristic(1.0f, spdf, 1.0f, p);
                }
                if (second) sr = spawn_ray(it.p, it.p_err, it.n, it.time, wdir, REF);
            }
        }
        __syncthreads();
        int lprim = -1;
        if (second) {
            Ray rr = sr;
            lprim = mega_trace<false>(sc, rr, err);
        }
        __syncthreads();
        if (second) {
            RGB li = rgb(0.0f);
            if (lprim < 0) {
                // an escaping ray sees Light::radiance: the environment map of an infinite light
                if (light_prim == LIGHT_INFINITE) li = mega_inf_radiance(sc, wdir);
            } else if (REF ? prim_emission(sc, lprim) >= 0 : lprim == (int)light_prim) {
                Isect lit;
                if (mega_isect(sc, lprim, sr, &lit)) li = emitted_radiance(sc, lit, -wdir);
            }
            if (!is_black(li)) ld = ld + f * li * w2 / spdf;
        }
        if (nee) out = out + beta * (ld / lpdf);
        __syncthreads();
        // continuation, roulette
        if (alive && !ended) {
            const V3 wo = -ray.d;
            calls.get_2d(u[BD_BSDF], u[BD_BSDF + 1]);
            const BxSample bs = mega_sample<REF>(bsdf, wo, u[BD_BSDF], u[BD_BSDF + 1], BSDF_ALL);
            if (is_black(bs.f) || bs.pdf == 0.0f) {
                ended = true;
            } else {
                beta = beta * (bs.f * abs_dot(bs.wi, it.ns) / bs.pdf);
                specular_bounce = (bs.stype & BSDF_SPECULAR) != 0;
                if ((bs.stype & BSDF_SPECULAR) && (bs.stype & BSDF_TRANSMISSION)) {
                    const float eta = bsdf.eta;
                    eta_scale *= dot(wo, it.n) > 0.0f ? eta * eta : 1.0f / (eta * eta);
                }
                // F1: REF re-intersects the same ray (t_max already at this hit); PBRT moves on
                if (!REF) ray = spawn_ray(it.p, it.p_err, it.n, it.time, bs.wi, false);
                const RGB rr_beta = beta * eta_scale;
                if (max_value(rr_beta) < rp.rr_threshold && bounces > 3) {
                    calls.get_1d(u[BD_RR]);
                    const float q = rmax(1.0f - max_value(rr_beta), 0.5f);
                    if (u[BD_RR] < q) ended = true;
                    else beta = beta / (1.0f - q);
                }
                ++bounces;
            }
        }
        if (alive && ended) {
            film_add(film, pix, out);
            alive = false;
        }
    }
}

void launch_megakernel(bool ref_compat, const Scene& sc, const Camera& cam, const RenderParams& rp,
                       const FilmBuffers& film, uint32_t* err, const LaunchShape& ls, cudaStream_t s) {
    if (ref_compat) k_megakernel<true><<<ls.sms, MEGA_BLOCK, 0, s>>>(sc, cam, rp, film, err);
    else k_megakernel<false><<<ls.sms, MEGA_BLOCK, 0, s>>>(sc, cam, rp, film, err);
}

}  // namespace bg
