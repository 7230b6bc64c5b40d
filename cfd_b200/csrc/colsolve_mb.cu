// colsolve_mb.cu - the warp-per-column solves of three-band channels.
#include "colsolve_launch.cuh"

namespace cfd {

cudaError_t col_prepare_mb(int m) { return prepare<true>(m, 4); }

void col_launch_mb(int mode, int m, int nsm, cudaStream_t st, const Dims& d, const Geo& g, const ColMaps& maps,
                   const ColArgs& a) {
    launch<true>(mode, m, 4, nsm, st, d, g, maps, a);
}

}  // namespace cfd
