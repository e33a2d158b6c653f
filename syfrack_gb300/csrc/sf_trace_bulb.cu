// Persistent trace kernel and primary rays instantiated for the bulb form (see sf_trace_kernel.cuh,
// sf_primary_kernel.cuh).
#include "sf_primary_kernel.cuh"
#include "sf_trace_kernel.cuh"

cudaError_t sf_launch_trace_bulb(const DeProgram* prog, const DevScene* scene, PathSoA soa, TraceLaunch tl,
                               unsigned long long* stats, int blocks, int min_blocks, uint32_t light_smem, cudaStream_t st) {
    return launch_trace_form<SF_FORM_BULB>(prog, scene, soa, tl, stats, blocks, min_blocks, light_smem, st);
}
cudaError_t sf_launch_primary_bulb(const DeProgram* prog, const DevScene* scene, const PrimaryLaunch& pl, cudaStream_t st) {
    return launch_primary_form<SF_FORM_BULB>(prog, scene, pl, st);
}
