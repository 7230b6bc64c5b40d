// colsolve.cu - instantiations and launches of the warp-per-column solves (colsolve.cuh).
#include <cudaTypedefs.h>

#include "colsolve_launch.cuh"

namespace cfd {

bool col_map(CUtensorMap* map, const void* field, int ncol, int n, int m, int cols) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &st) != cudaSuccess ||
            st != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (PFN_cuTensorMapEncodeTiled_v12000)f;
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {2 * (cuuint64_t)ncol, (cuuint64_t)n}, strides[1] = {(cuuint64_t)ncol * 16};
    const cuuint32_t box[2] = {2 * (cuuint32_t)cols, (cuuint32_t)(32 * m / col_boxes(m))}, step[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<void*>(field), dims, strides, box, step,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, cols == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

void col_meanflow(int m, cudaStream_t st, const Dims& d, const Geo& g, double beta, double bdt, double qxt, double2* u1,
                  double* scal, bool ghosts) {
    COL_SWITCH(m, { k_meanflow_warp<MR><<<1, 32, 0, st>>>(d, g, beta, bdt, qxt, u1, scal, ghosts); });
}

cudaError_t col_prepare(int m, int cols, bool mb) { return mb ? col_prepare_mb(m) : prepare<false>(m, cols); }

void col_launch(int mode, int m, int cols, bool mb, int nsm, cudaStream_t st, const Dims& d, const Geo& g,
                const ColMaps& maps, const ColArgs& a) {
    if (mb) col_launch_mb(mode, m, nsm, st, d, g, maps, a);
    else launch<false>(mode, m, cols, nsm, st, d, g, maps, a);
}

}  // namespace cfd
