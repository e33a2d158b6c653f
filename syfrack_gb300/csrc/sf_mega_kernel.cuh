// The per-pixel megakernel of the scenes that sf_path_kernel.cuh does not take (surface
// features, optics, fog, many shadow segments): one thread a path, marches in line.
// Compiled once per feature set (sf_mega*.cu): one instantiation takes a minute or more.
#pragma once
#include "sf_stages.cuh"

// The plain per-pixel integrator (pathtrace.wgsl:1203-1276): one thread per path, a
// sample of a pixel, with blocking marches. A pixel's samples run in different blocks
// (blockIdx.z): k_commit adds them in ascending order whichever ends first.
static __device__ int march_full(const DeProgram& P, March& m, uint32_t max_steps, float safety, float accept,
                                 bool absolute, DeRaw& hit, unsigned long long& evals, unsigned long long& iters) {
    int r = march_check(m, max_steps, accept);
    while (r == MARCH_CONTINUE) {
        const float3 q = m.ro + m.rd * m.t;
        DeRaw s = de_raw(P, q);
        evals++;
        iters += s.iter;
        if (needs_exact(s, m.t, safety, accept, absolute)) {
            s = de_raw_exact(P, q);
            evals++;
            iters += s.iter;
        }
        r = march_update(m, s.d, s.flags, safety, accept, absolute);
        if (r == MARCH_HIT) { hit = s; m.cand_t = m.t; return r; }
        if (r == MARCH_CONTINUE) r = march_check(m, max_steps, accept);
    }
    if (r == MARCH_HIT) {  // candidate accepted at the step budget
        const float3 q = m.ro + m.rd * m.cand_t;
        hit = de_raw(P, q);
        evals++;
        iters += hit.iter;
        if (needs_exact(hit, m.cand_t, safety, accept, absolute)) {
            hit = de_raw_exact(P, q);
            evals++;
            iters += hit.iter;
        }
    }
    return r;
}

// optical_refine_hit (optics.wgsl:7-23): up to eight Newton steps along the ray on the
// exact field from the hit at t, with a central difference of step eps (from the hit).
static __device__ float optical_refine(const DeProgram& P, float3 ro, float3 rd, float t, unsigned long long& evals,
                                       unsigned long long& iters) {
    const float eps = fmaxf(1e-5f, fminf(1e-3f, t * 1e-5f));
    for (uint32_t i = 0; i < 8u; ++i) {
        const float3 p = ro + rd * t;
        const DeRaw a = de_raw_exact(P, p);
        evals++;
        iters += a.iter;
        if (fabsf(a.d) < 1e-5f) break;
        const DeRaw b = de_raw_exact(P, p + rd * eps);
        const DeRaw c = de_raw_exact(P, p + rd * (-eps));
        evals += 2;
        iters += b.iter + c.iter;
        const float derivative = (b.d - c.d) / (2.0f * eps);
        if (fabsf(derivative) < 1e-5f) break;
        t = fmaxf(0.0f, t - fminf(fmaxf(a.d / derivative, -0.5f), 0.5f));
    }
    return t;
}

// FEAT: the surface features the kernel is built with (SF_FEAT_*; 0 for plain scenes).
template <int FEAT>
__global__ void __launch_bounds__(64) k_megakernel(const DeProgram* __restrict__ prog_g,
                                                   const DevScene* __restrict__ scene_g, PathSoA soa, DispatchGeom g,
                                                   FilmPlanes film, unsigned long long* stats) {
    __shared__ DeProgram P;
    __shared__ DevScene S;
    stage_program(P, prog_g);
    stage_pod(S, scene_g);
    stage_more_lights(scene_g);
    __syncthreads();
    uint32_t lx = blockIdx.x * 8 + (threadIdx.x & 7), ly = blockIdx.y * 8 + (threadIdx.x >> 3);
    if (lx >= g.tile_w || ly >= g.tile_h) return;
    uint32_t px = g.tile_x + lx, py = g.tile_y + ly;
    uint32_t tile_px = g.tile_w * g.tile_h, local = ly * g.tile_w + lx;
    const float accept = hit_accept(S);
    const bool absolute = hit_absolute(S);
    unsigned long long evals = 0, iters = 0, segs = 0;
    const uint32_t stream = point_stream_of(S, px, py);
    const bool optics = (FEAT & SF_FEAT_RICH) && (S.rich & SF_RICH_OPTICS) != 0u;
    for (uint32_t s = blockIdx.z; s < g.samples; s += gridDim.z) {
        uint32_t sample = g.sample_start + s;
        PathState ps;
        path_begin(S, ps, px, py, sample);
        if (optics) {  // the medium the camera ray starts in
            const DeRaw r0 = de_raw_exact(P, ps.o);
            evals++;
            iters += r0.iter;
            optics_initial_medium(S, ps, r0.d, r0.material);
        }
        float* fd = nullptr;
        float4* fa = nullptr;
        for (;;) {
            uint32_t li;
            March m;
            float t_end = nearest_emitter(S, ps.o, ps.d, S.extent, li);
            march_begin(m, ps.o, ps.d, t_end);
            DeRaw hs;
            int r = march_full(P, m, S.max_steps, S.step_scale, accept, absolute, hs, evals, iters);
            segs++;
            HitInfo h;
            h.hit = false;
            h.exhausted = r == MARCH_EXHAUSTED;
            h.light_index = SF_NO_LIGHT;
            h.steps = m.i;
            h.t = m.t_end;
            if (r == MARCH_HIT) {
                h.hit = true;
                h.t = m.cand_t;
                bool optical = false;
                if (optics && optics_enabled(material_optics(S, hs.material))) {
                    h.t = optical_refine(P, ps.o, ps.d, h.t, evals, iters);
                    hs = de_raw_exact(P, ps.o + ps.d * h.t);
                    evals++;
                    iters += hs.iter;
                    optical = optics_enabled(material_optics(S, hs.material));
                }
                h.sample = de_finalize(P, hs);
                float3 hp = ps.o + ps.d * h.t;
                const float tap_h = optical ? 1e-4f : fmaxf(h.t * S.pixel_cone * 0.5f, 1e-4f) * S.pixel_tolerance;
                float3 grad = mk3(0.f, 0.f, 0.f);
                for (uint32_t k = 0; k < 4; ++k) {
                    DeRaw d = de_raw(P, hp + tetra_offset(k) * tap_h);
                    evals++;
                    iters += d.iter;
                    grad = grad + tetra_offset(k) * d.d;
                }
                h.n = wnormalize(grad);  // as the trace kernel's taps: one rsqrt
            } else if (r == MARCH_MISS && li != SF_NO_LIGHT) {
                h.hit = true;
                h.light_index = li;
            }
            if (sample == 0 && ps.bounce == 0) {
                const size_t idx = film_index(film, px, py);
                fd = film.depth + idx;
                fa = film.aux + idx;
            } else {
                fd = nullptr;
                fa = nullptr;
            }
            // each shadow segment is traced as it is issued; its radiance lands in the
            // order the wavefront adds it (issue order, after the bounce's own terms)
            auto emit = [&](const ShadowReq& sh) {
                if (!optics) {
                    uint32_t sli;
                    March sm;
                    float st_end = nearest_emitter(S, sh.o, sh.dir, sh.t_end, sli);
                    march_begin(sm, sh.o, sh.dir, st_end);
                    DeRaw shs;
                    int sr = march_full(P, sm, S.max_steps, S.step_scale, accept, absolute, shs, evals, iters);
                    segs++;
                    if (sr == MARCH_MISS && sli == SF_NO_LIGHT) {
                        ps.L = add_rn(ps.L, sh.contrib);
                        if (sh.volume) ps.pv = add_rn(ps.pv, sh.contrib);
                    }
                    return;
                }
                // geometry_visibility_weight (lights.wgsl:263-283): dielectric surfaces pass
                // the segment weighted by 1 - opacity, up to 32 segments
                float vis = 1.0f;
                float3 origin = sh.o;
                float remaining = sh.t_end;
                bool clear = false;
                for (uint32_t i = 0; i < 32u; ++i) {
                    uint32_t sli;
                    March sm;
                    const float st_end = nearest_emitter(S, origin, sh.dir, remaining, sli);
                    march_begin(sm, origin, sh.dir, st_end);
                    DeRaw shs;
                    const int sr = march_full(P, sm, S.max_steps, S.step_scale, accept, absolute, shs, evals, iters);
                    segs++;
                    if (sr == MARCH_EXHAUSTED) break;
                    if (sr == MARCH_MISS) {
                        clear = sli == SF_NO_LIGHT;
                        break;
                    }
                    float t = sm.cand_t;
                    if (optics_enabled(material_optics(S, shs.material))) {
                        t = optical_refine(P, origin, sh.dir, t, evals, iters);
                        shs = de_raw_exact(P, origin + sh.dir * t);
                        evals++;
                        iters += shs.iter;
                    }
                    const DevOptics& o = material_optics(S, shs.material);
                    if (!optics_enabled(o)) break;
                    vis *= 1.0f - o.surface[0];
                    if (vis < 1e-6f) break;
                    const float distance = t + 1e-4f;
                    origin = origin + sh.dir * distance;
                    remaining = remaining - distance;
                    if (remaining <= 0.0f) {
                        clear = true;
                        break;
                    }
                }
                if (clear) {
                    const float3 c = sh.contrib * vis;
                    ps.L = add_rn(ps.L, c);
                    if (sh.volume) ps.pv = add_rn(ps.pv, c);
                }
            };
            int cont = bounce_body<FEAT>(S, ps, h, emit, fd, fa, sample, stream);
            if (cont != PATH_CONTINUE) break;
        }
        soa.Ls[(size_t)s * tile_px + local] = make_float4(ps.L.x, ps.L.y, ps.L.z, 1.0f);
        if (soa.pv) {  // the sample's volume part (pathtrace.wgsl:1198)
            const float3 v = path_volume(ps);
            soa.pv[(size_t)s * tile_px + local] = make_float4(v.x, v.y, v.z, 0.f);
        }
    }
    warp_stat(&stats[SF_STAT_DE_EVALS], evals);
    warp_stat(&stats[SF_STAT_DE_ITERS], iters);
    warp_stat(&stats[SF_STAT_SEGMENTS], segs);
}

template <int FEAT>
static cudaError_t launch_megakernel_feat(const DeProgram* prog, const DevScene* scene, PathSoA soa, DispatchGeom g,
                                          FilmPlanes film, unsigned long long* stats, cudaStream_t st) {
    dim3 grid((g.tile_w + 7) / 8, (g.tile_h + 7) / 8, g.samples < 65535u ? g.samples : 65535u);
    k_megakernel<FEAT><<<grid, 64, g.light_smem, st>>>(prog, scene, soa, g, film, stats);
    return cudaGetLastError();
}
