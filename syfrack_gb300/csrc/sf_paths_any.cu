// The persistent path kernel instantiated for the any form (see sf_path_kernel.cuh).
#include "sf_path_kernel.cuh"

cudaError_t sf_launch_paths_any(const DeProgram* prog, const DevScene* scene, PathSoA soa, DispatchGeom g, FilmPlanes film,
                               unsigned long long* stats, uint32_t* work, cudaStream_t st) {
    return launch_paths_form<SF_FORM_ANY>(prog, scene, soa, g, film, stats, work, st);
}
