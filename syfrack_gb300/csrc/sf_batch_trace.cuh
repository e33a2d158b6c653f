// The persistent trace kernel of a batch: its jobs' segments group by group (form and
// variant), so a warp's lanes run one form's code. A warp that finds a group's items
// taken goes on to the next group's while others finish theirs, so the groups share one
// launch and one tail. With the form chosen per lane in one loop, 64 mixed jobs took
// 105 ms a pass (4 blocks per SM, no quantum, regeneration 8) and 60 this way.
// GENERIC: the batch has a group of generic graphs (the interpreter's stack and calls).
#pragma once
#include "sf_trace_kernel.cuh"

template <int MIN_BLOCKS, bool GENERIC, bool OPTICS>
__global__ void __launch_bounds__(256, MIN_BLOCKS) k_trace_batch(PathSoA soa, TraceLaunch tl, unsigned long long* stats,
                                                                 BatchTable bt) {
    __shared__ uint32_t begins[SF_BATCH_MAX_JOBS];
    for (uint32_t i = threadIdx.x; i < bt.n_jobs; i += blockDim.x) begins[i] = bt.jobs[i].path_begin;
    __syncthreads();
    // every lane reads its own job's program and scene; these are only where it starts
    const DeProgram& P = *bt.jobs[0].prog;
    const DevScene& S = *bt.jobs[0].scene;
    for (uint32_t g = 0; g < bt.groups; ++g) {
        const TraceGroup group{g, bt.group_begin[g]};
        switch (bt.group_form[g]) {
        case SF_FORM_BULB:
            trace_group<SF_FORM_BULB, true, false, OPTICS>(P, S, begins, soa, tl, stats, bt, group);
            break;
        case SF_FORM_BOX:
            trace_group<SF_FORM_BOX, true, false, OPTICS>(P, S, begins, soa, tl, stats, bt, group);
            break;
        case SF_FORM_MENGER:
            trace_group<SF_FORM_MENGER, true, false, OPTICS>(P, S, begins, soa, tl, stats, bt, group);
            break;
        default:
            if constexpr (GENERIC)
                trace_group<SF_FORM_ANY, true, false, OPTICS>(P, S, begins, soa, tl, stats, bt, group);
            break;
        }
    }
}

template <bool GENERIC>
static cudaError_t launch_trace_batch(BatchTable bt, PathSoA soa, TraceLaunch tl, unsigned long long* stats, int blocks,
                                      int min_blocks, cudaStream_t st) {
    if (tl.optics) {  // a job with dielectric materials: the optics instantiation, 2 blocks per SM
        k_trace_batch<2, GENERIC, true><<<blocks, 256, 0, st>>>(soa, tl, stats, bt);
        return cudaGetLastError();
    }
    switch (min_blocks) {
    case 3: k_trace_batch<3, GENERIC, false><<<blocks, 256, 0, st>>>(soa, tl, stats, bt); break;
    case 4: k_trace_batch<4, GENERIC, false><<<blocks, 256, 0, st>>>(soa, tl, stats, bt); break;
    default: k_trace_batch<2, GENERIC, false><<<blocks, 256, 0, st>>>(soa, tl, stats, bt); break;
    }
    return cudaGetLastError();
}
