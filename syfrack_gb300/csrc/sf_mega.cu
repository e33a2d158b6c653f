// The blocking per-pixel kernel for plain surfaces, and the choice among its builds (see
// sf_mega_kernel.cuh).
#include "sf_mega_kernel.cuh"

cudaError_t sf_launch_megakernel(const DeProgram* prog, const DevScene* scene, uint32_t rich, PathSoA soa,
                                 DispatchGeom g, FilmPlanes film, unsigned long long* stats, cudaStream_t st) {
    if (rich & SF_RICH_TEXTURE) return sf_launch_megakernel_textured(prog, scene, soa, g, film, stats, st);
    if (rich) return sf_launch_megakernel_rich(prog, scene, soa, g, film, stats, st);
    return launch_megakernel_feat<0>(prog, scene, soa, g, film, stats, st);
}
