// The blocking per-pixel kernel for textured scenes (see sf_mega_kernel.cuh).
#include "sf_mega_kernel.cuh"

cudaError_t sf_launch_megakernel_textured(const DeProgram* prog, const DevScene* scene, PathSoA soa, DispatchGeom g,
                                          FilmPlanes film, unsigned long long* stats, cudaStream_t st) {
    return launch_megakernel_feat<3>(prog, scene, soa, g, film, stats, st);
}
