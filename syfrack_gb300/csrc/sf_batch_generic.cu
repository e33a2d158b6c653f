// The batch's trace kernel for batches with generic graphs (see sf_batch_trace.cuh).
#include "sf_batch_trace.cuh"

cudaError_t sf_launch_trace_batch_generic(BatchTable bt, PathSoA soa, TraceLaunch tl, unsigned long long* stats,
                                          int blocks, int min_blocks, cudaStream_t st) {
    return launch_trace_batch<true>(bt, soa, tl, stats, blocks, min_blocks, st);
}
