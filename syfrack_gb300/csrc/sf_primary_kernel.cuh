// Primary rays through pixel centres (control.wgsl:270-273): the relaxed march with a
// fixed-epsilon (rule 1) or cone-relative (rule 0) hit test, then a 6-tap central
// (normal_mode 0) or 4-tap tetrahedral (1) normal. Compiled once per form, as the trace
// kernel: one kernel for every graph carried the generic interpreter's 125 registers
// and 704 bytes of stack through the bundled forms too.
//
// Every lane holds one ray; a lane whose ray has ended takes the next pixel once
// PRIMARY_REGEN lanes of its warp are idle (or no lane is marching), so the ray set-up
// runs for several lanes at once and the warp keeps evaluating the DE in lockstep.
// Surface hits run their normal taps through the same DE call. Small frames are bound
// by their longest ray's chain of dependent steps (256 of them at 256x256), large ones
// by instruction issue.
#pragma once
#include "sf_trace_kernel.cuh"

enum { PR_IDLE = 0, PR_MARCH = 1, PR_NORMAL = 2, PR_DONE = 3 };
constexpr int PRIMARY_REGEN = 4, PRIMARY_THREADS = 128;

__device__ __forceinline__ float3 central_offset(uint32_t i) {
    float sgn = (i & 1u) ? -1.0f : 1.0f;
    uint32_t a = i >> 1;
    return mk3(a == 0 ? sgn : 0.f, a == 1 ? sgn : 0.f, a == 2 ? sgn : 0.f);
}

template <int FORM>
__global__ void __launch_bounds__(PRIMARY_THREADS) k_primary(const DeProgram* __restrict__ prog_g,
                                                             const DevScene* __restrict__ scene_g, PrimaryLaunch pl) {
    __shared__ DeProgram P;
    __shared__ DevScene S;
    stage_program(P, prog_g);
    stage_pod(S, scene_g);
    __syncthreads();
    const uint32_t width = pl.width, total = pl.width * pl.height, max_steps = pl.max_steps;
    const int normal_mode = pl.normal_mode;
    const float cone = S.tan_half * 2.0f / float(width);
    const float accept = pl.rule == 1 ? pl.eps : cone * S.pixel_tolerance;
    const bool absolute = pl.rule == 1;
    const uint32_t taps = normal_mode == 0 ? 6u : 4u;
    uint32_t state = PR_IDLE, pix = 0, tap = 0;
    March m{};
    float3 hp = mk3(0.f, 0.f, 0.f), grad = mk3(0.f, 0.f, 0.f);
    float hstep = 0.f, thit = 0.f;
    unsigned long long n_eval = 0, n_iter = 0, n_steps = 0;
    auto store_normal = [&](float3 n) {
        float* const q = pl.n + pix * pl.n_pixel;
        q[0] = n.x;
        q[pl.n_part] = n.y;
        q[2 * pl.n_part] = n.z;
    };
    // the ray's end: a hit at cand_t starts the normal taps, a miss writes its values
    auto end_ray = [&](bool hit) {
        pl.steps[pix] = m.i;
        n_steps += m.i;
        if (hit) {
            thit = m.cand_t;
            hp = m.ro + m.rd * thit;
            hstep = fmaxf(thit * cone * 0.5f, 1e-4f) * S.pixel_tolerance;
            grad = mk3(0.f, 0.f, 0.f);
            tap = 0;
            state = PR_NORMAL;
        } else {
            pl.t[pix] = -1.0f;
            store_normal(mk3(0.f, 0.f, 0.f));
            state = PR_IDLE;
        }
    };
    while (true) {
        const uint32_t quiet = __ballot_sync(FULL_MASK, state == PR_IDLE || state == PR_DONE);
        const uint32_t idle = quiet ? __ballot_sync(FULL_MASK, state == PR_IDLE) : 0u;
        if (quiet == FULL_MASK && idle == 0u) break;  // every lane done
        if (idle && (__popc(idle) >= PRIMARY_REGEN || quiet == FULL_MASK)) {  // warp-uniform
            const uint32_t w = warp_fetch(pl.work, state == PR_IDLE);
            if (state == PR_IDLE) {
                if (w >= total) {
                    state = PR_DONE;
                } else {
                    pix = w;
                    uint32_t px = pix % width, py = pix / width;
                    float ndcx = ((float(px) + 0.5f) / float(width)) * 2.0f - 1.0f;
                    float ndcy = ((float(py) + 0.5f) / float(pl.height)) * 2.0f - 1.0f;
                    float3 rd = normalize3(ld3(S.forward) + ld3(S.right) * (ndcx * S.tan_half) +
                                           ld3(S.up) * (-ndcy * S.tan_half / S.aspect));
                    march_begin(m, ld3(S.origin), rd, pl.t_far);
                    state = PR_MARCH;
                    const int r = march_check(m, max_steps, accept);  // an empty march
                    if (r != MARCH_CONTINUE) end_ray(r == MARCH_HIT);
                }
            }
        }
        if (state == PR_MARCH || state == PR_NORMAL) {
            const float3 qp = state == PR_NORMAL
                                  ? hp + (normal_mode == 0 ? central_offset(tap) : tetra_offset(tap)) * hstep
                                  : m.ro + m.rd * m.t;
            DeRaw s = de_form<FORM>(P, P.fp, qp);
            n_eval++;
            n_iter += s.iter;
            if constexpr (FORM == SF_FORM_ANY) {
                if (state == PR_MARCH && needs_exact(s, m.t, S.step_scale, accept, absolute)) {
                    s = de_form_exact<FORM>(P, P.fp, qp);
                    n_eval++;
                    n_iter += s.iter;
                }
            }
            if (state == PR_NORMAL) {
                grad = grad + (normal_mode == 0 ? central_offset(tap) : tetra_offset(tap)) * s.d;
                if (++tap == taps) {
                    float3 n = normalize3(grad);
                    pl.t[pix] = thit;
                    store_normal(n);
                    state = PR_IDLE;
                }
            } else {
                int r = march_update(m, s.d, s.flags, S.step_scale, accept, absolute);
                if (r == MARCH_HIT) m.cand_t = m.t;
                else if (r == MARCH_CONTINUE) r = march_check(m, max_steps, accept);  // a candidate's hit is at cand_t
                if (r != MARCH_CONTINUE) end_ray(r == MARCH_HIT);
            }
        }
    }
    warp_stat(&pl.stats[SF_STAT_DE_EVALS], n_eval);
    warp_stat(&pl.stats[SF_STAT_DE_ITERS], n_iter);
    warp_stat(&pl.stats[SF_STAT_STEPS], n_steps);
}

template <int FORM>
static cudaError_t launch_primary_form(const DeProgram* prog, const DevScene* scene, const PrimaryLaunch& pl,
                                       cudaStream_t st) {
    // one ray a lane up to 8 blocks per SM, persistent lanes beyond
    const size_t want = ((size_t)pl.width * pl.height + PRIMARY_THREADS - 1) / PRIMARY_THREADS;
    const size_t cap = (size_t)sf_device_sm_count() * 8u;
    k_primary<FORM><<<(unsigned)(want < cap ? want : cap), PRIMARY_THREADS, 0, st>>>(prog, scene, pl);
    return cudaGetLastError();
}
