// The per-pixel integrator (pathtrace.wgsl:1203-1276) with whole paths on persistent
// lanes: a lane owns a path (a sample of a pixel) from its camera ray to its radiance and
// takes the next one, and the lanes of a warp march whatever segments they are on
// together. A lane whose segment has ended waits until PATH_BATCH lanes of its warp have
// (or none is marching), then they run what follows together: the bounce body, the next
// segment's set-up, the next path. With blocking marches, one after the other in each
// thread (k_megakernel, which keeps the scenes this kernel does not take), 7.6 lanes of
// 32 were active on average.
//
// Bounce body, march and sampling are those of the other integrators, and a bounce's
// shadow segments add their radiance in issue order after it, so films are theirs bit for
// bit. It takes scenes without finish details, textures, optics and fog whose bounces
// issue at most SF_MAX_SHADOWS shadow segments (they wait in the lane's local memory).
// Compiled once per form, as the trace kernel.
#pragma once
#include "sf_stages.cuh"
#include "sf_trace_kernel.cuh"

enum { PA_IDLE = 0, PA_MARCH = 1, PA_CAND = 2, PA_NORMAL = 3, PA_ENDED = 4, PA_DONE = 5 };
constexpr int PATH_BATCH = 8, PATH_THREADS = 128, PATH_BLOCKS = 4;

template <int FORM>
__global__ void __launch_bounds__(PATH_THREADS, PATH_BLOCKS) k_paths(const DeProgram* __restrict__ prog_g,
                                                                     const DevScene* __restrict__ scene_g, PathSoA soa,
                                                                     DispatchGeom g, FilmPlanes film,
                                                                     unsigned long long* stats, uint32_t* work) {
    __shared__ DeProgram P;
    __shared__ DevScene S;
    stage_program(P, prog_g);
    stage_pod(S, scene_g);
    stage_more_lights(scene_g);
    __syncthreads();
    const float accept = hit_accept(S);
    const bool absolute = hit_absolute(S);
    uint32_t state = PA_IDLE, path = 0, px = 0, py = 0, sample = 0, li = SF_NO_LIGHT;
    PathState ps;
    March m{};
    int end = MARCH_MISS;           // how the segment ended
    bool more = false;              // the path goes on after its shadow segments
    uint32_t sh_at = 0, sh_n = 0;   // the shadow segment marched (of sh_n), sh_n: the continuation
    ShadowReq sh[SF_MAX_SHADOWS];
    DeSampleF smp{};                // the hit's sample
    float3 grad = mk3(0.f, 0.f, 0.f);
    float hstep = 0.f;
    uint32_t tap = 0;
    unsigned long long evals = 0, iters = 0, segs = 0;

    auto check = [&]() {  // before a step of the march
        const int r = march_check(m, S.max_steps, accept);
        if (r == MARCH_CONTINUE) return;
        end = r;
        if (r == MARCH_HIT && sh_at == sh_n) {  // a candidate accepted at the step budget
            m.t = m.cand_t;
            state = PA_CAND;
        } else {
            state = PA_ENDED;
        }
    };
    auto begin = [&](float3 o, float3 d, float t_end) {
        march_begin(m, o, d, nearest_emitter(S, o, d, t_end, li));
        segs++;
        state = PA_MARCH;
        check();
    };

    while (true) {
        const uint32_t wait = __ballot_sync(FULL_MASK, state == PA_IDLE || state == PA_ENDED);
        const uint32_t marching = __ballot_sync(FULL_MASK, state >= PA_MARCH && state <= PA_NORMAL);
        if ((wait | marching) == 0u) break;
        if (wait != 0u && (__popc(wait) >= PATH_BATCH || marching == 0u)) {
            bool next = false;  // start the next segment of the path
            if (state == PA_ENDED) {
                next = true;
                if (sh_at < sh_n) {  // a shadow segment
                    if (end == MARCH_MISS && li == SF_NO_LIGHT) ps.L = add_rn(ps.L, sh[sh_at].contrib);
                    sh_at++;
                } else {
                    HitInfo h;
                    h.hit = false;
                    h.exhausted = end == MARCH_EXHAUSTED;
                    h.light_index = SF_NO_LIGHT;
                    h.steps = m.i;
                    h.t = m.t_end;
                    if (end == MARCH_HIT) {
                        h.hit = true;
                        h.t = m.t;
                        h.sample = smp;
                        h.n = wnormalize(grad);  // as the trace kernel's taps: one rsqrt
                    } else if (end == MARCH_MISS && li != SF_NO_LIGHT) {
                        h.hit = true;
                        h.light_index = li;
                    }
                    float* fd = nullptr;
                    float4* fa = nullptr;
                    if (sample == 0 && ps.bounce == 0) {
                        const size_t idx = film_index(film, px, py);
                        fd = film.depth + idx;
                        fa = film.aux + idx;
                    }
                    sh_at = sh_n = 0;
                    auto emit = [&](const ShadowReq& r) {
                        if (sh_n < SF_MAX_SHADOWS) sh[sh_n++] = r;
                    };
                    more = bounce_body<0>(S, ps, h, emit, fd, fa, sample, point_stream_of(S, px, py)) == PATH_CONTINUE;
                }
                if (sh_at == sh_n && !more) {
                    soa.Ls[path] = make_float4(ps.L.x, ps.L.y, ps.L.z, 1.0f);
                    state = PA_IDLE;
                    next = false;
                }
            }
            const uint32_t w = warp_fetch(work, state == PA_IDLE);
            if (state == PA_IDLE) {
                if (w < g.paths) {
                    // the samples of a pixel in turn, pixels column by column in bands of four rows
                    const uint32_t p = w / g.samples, s = w - p * g.samples;
                    const uint32_t band = p / (4u * g.tile_w), r = p - band * 4u * g.tile_w;
                    const uint32_t rows = min(4u, g.tile_h - 4u * band), x = r / rows;
                    const uint32_t y = 4u * band + r - x * rows;
                    px = g.tile_x + x;
                    py = g.tile_y + y;
                    sample = g.sample_start + s;
                    path = (s * g.tile_h + y) * g.tile_w + x;
                    path_begin(S, ps, px, py, sample);
                    sh_at = sh_n = 0;
                    next = true;
                } else {
                    state = PA_DONE;
                }
            }
            if (next) {
                const bool shadow = sh_at < sh_n;
                begin(shadow ? sh[sh_at].o : ps.o, shadow ? sh[sh_at].dir : ps.d, shadow ? sh[sh_at].t_end : S.extent);
            }
        }
        if (state >= PA_MARCH && state <= PA_NORMAL) {
            float3 q = m.ro + m.rd * m.t;
            if (state == PA_NORMAL) q = q + tetra_offset(tap) * hstep;
            DeRaw s = de_form<FORM>(P, P.fp, q);
            evals++;
            iters += s.iter;
            if constexpr (FORM == SF_FORM_ANY) {
                if (state != PA_NORMAL && needs_exact(s, m.t, S.step_scale, accept, absolute)) {
                    s = de_form_exact<FORM>(P, P.fp, q);
                    evals++;
                    iters += s.iter;
                }
            }
            if (state == PA_NORMAL) {
                const float3 off = tetra_offset(tap);
                grad = mk3(fmaf(off.x, s.d, grad.x), fmaf(off.y, s.d, grad.y), fmaf(off.z, s.d, grad.z));
                if (++tap == 4) state = PA_ENDED;
            } else {
                bool hit = state == PA_CAND;
                if (!hit) {
                    const int r = march_update(m, s.d, s.flags, S.step_scale, accept, absolute);
                    if (r == MARCH_CONTINUE) {
                        check();
                    } else {
                        end = r;
                        hit = r == MARCH_HIT && sh_at == sh_n;
                        if (!hit) state = PA_ENDED;
                    }
                }
                if (hit) {  // a continuation's surface at m.t: its sample, then the normal taps
                    smp = de_finalize(P, s);
                    hstep = fmaxf(m.t * S.pixel_cone * 0.5f, 1e-4f) * S.pixel_tolerance;
                    grad = mk3(0.f, 0.f, 0.f);
                    tap = 0;
                    state = PA_NORMAL;
                }
            }
        }
    }
    warp_stat(&stats[SF_STAT_DE_EVALS], evals);
    warp_stat(&stats[SF_STAT_DE_ITERS], iters);
    warp_stat(&stats[SF_STAT_SEGMENTS], segs);
}

template <int FORM>
static cudaError_t launch_paths_form(const DeProgram* prog, const DevScene* scene, PathSoA soa, DispatchGeom g,
                                     FilmPlanes film, unsigned long long* stats, uint32_t* work, cudaStream_t st) {
    const unsigned want = (g.paths + PATH_THREADS - 1) / PATH_THREADS;
    const unsigned cap = (unsigned)(sf_device_sm_count() * PATH_BLOCKS);
    k_paths<FORM><<<want < cap ? want : cap, PATH_THREADS, g.light_smem, st>>>(prog, scene, soa, g, film, stats, work);
    return cudaGetLastError();
}
