// colsolve.cu - instantiations and launches of the warp-per-column solves (colsolve.cuh).
#include <algorithm>

#include <cudaTypedefs.h>

#include "colsolve.cuh"

namespace cfd {

// Run BODY with MR = the rows per lane m.
#define COL_SWITCH(m, ...)                                        \
    switch (m) {                                                  \
        case 1: { constexpr int MR = 1; __VA_ARGS__; } break;     \
        case 3: { constexpr int MR = 3; __VA_ARGS__; } break;     \
        case 5: { constexpr int MR = 5; __VA_ARGS__; } break;     \
        case 7: { constexpr int MR = 7; __VA_ARGS__; } break;     \
        case 9: { constexpr int MR = 9; __VA_ARGS__; } break;     \
        case 11: { constexpr int MR = 11; __VA_ARGS__; } break;   \
        case 13: { constexpr int MR = 13; __VA_ARGS__; } break;   \
        case 15: { constexpr int MR = 15; __VA_ARGS__; } break;   \
        case 19: { constexpr int MR = 19; __VA_ARGS__; } break;   \
        case 23: { constexpr int MR = 23; __VA_ARGS__; } break;   \
        default: break;                                           \
    }

cudaError_t col_prepare(int m) {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto* f, size_t n) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
    };
    COL_SWITCH(m, {
        set(k_col_solve<MR, 4, 7>, col_smem(MR, 4));
        set(k_col_solve<MR, 4, 1>, col_smem(MR, 4));
        set(k_col_solve<MR, 4, 2>, col_smem(MR, 4));
        if constexpr (MR <= 15) {
            set(k_col_solve<MR, 8, 7>, col_smem(MR, 8));
            set(k_col_solve<MR, 8, 1>, col_smem(MR, 8));
            set(k_col_solve<MR, 8, 2>, col_smem(MR, 8));
        }
    });
    return e;
}

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
                  CU_TENSOR_MAP_INTERLEAVE_NONE, cols == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,  CU_TENSOR_MAP_L2_PROMOTION_L2_128B,

                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

void col_launch(int mode, int m, int cols, int nsm, cudaStream_t st, const Dims& d, const Geo& g, const ColMaps& maps,
                const ColArgs& a) {
    const int grid = std::min(nsm, (d.ncol + cols - 1) / cols);
    auto run = [&](auto* f, int threads, size_t smem) { f<<<grid, threads, smem, st>>>(d, g, maps, a); };
    COL_SWITCH(m, {
        if constexpr (MR <= 15) {
            if (cols == 8) {
                const int threads = 32 * 8 * col_groups(MR, 8);
                if (mode == 7) run(k_col_solve<MR, 8, 7>, threads, col_smem(MR, 8));
                else if (mode == 1) run(k_col_solve<MR, 8, 1>, threads, col_smem(MR, 8));
                else run(k_col_solve<MR, 8, 2>, threads, col_smem(MR, 8));
                return;
            }
        }
        const int threads = 32 * 4 * col_groups(MR, 4);
        if (mode == 7) run(k_col_solve<MR, 4, 7>, threads, col_smem(MR, 4));
        else if (mode == 1) run(k_col_solve<MR, 4, 1>, threads, col_smem(MR, 4));
        else run(k_col_solve<MR, 4, 2>, threads, col_smem(MR, 4));
    });
}

}  // namespace cfd
