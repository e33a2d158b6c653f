// The blocking per-pixel kernel for scenes with finish details or optics (see sf_mega_kernel.cuh).
#include "sf_mega_kernel.cuh"

cudaError_t sf_launch_megakernel_rich(const DeProgram* prog, const DevScene* scene, PathSoA soa, DispatchGeom g,
                                      FilmPlanes film, unsigned long long* stats, cudaStream_t st) {
    return launch_megakernel_feat<1>(prog, scene, soa, g, film, stats, st);
}
