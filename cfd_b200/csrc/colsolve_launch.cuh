// colsolve_launch.cuh - instantiation of the warp-per-column solves, shared by colsolve.cu (one
// band) and colsolve_mb.cu (three bands).
#pragma once

#include <algorithm>

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

// m rows per lane, groups of cols columns, one band or three
template <bool MB>
static cudaError_t prepare(int m, int cols) {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto* f, size_t n) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
    };
    COL_SWITCH(m, {
        if constexpr (MR <= 15 && !MB) {
            if (cols == 8) {
                set(k_col_solve<MR, 8, 7, MB>, col_smem(MR, 8));
                set(k_col_solve<MR, 8, 1, MB>, col_smem(MR, 8));
                set(k_col_solve<MR, 8, 2, MB>, col_smem(MR, 8));
                return e;
            }
        }
        set(k_col_solve<MR, 4, 7, MB>, col_smem(MR, 4));
        set(k_col_solve<MR, 4, 1, MB>, col_smem(MR, 4));
        set(k_col_solve<MR, 4, 2, MB>, col_smem(MR, 4));
    });
    return e;
}

template <bool MB>
static void launch(int mode, int m, int cols, int nsm, cudaStream_t st, const Dims& d, const Geo& g,
                   const ColMaps& maps, const ColArgs& a) {
    const int grid = std::min(nsm, (d.ncol + cols - 1) / cols);
    auto run = [&](auto* f, int threads, size_t smem) { f<<<grid, threads, smem, st>>>(d, g, maps, a); };
    COL_SWITCH(m, {
        if constexpr (MR <= 15 && !MB) {
            if (cols == 8) {
                const int threads = 32 * 8 * col_groups(MR, 8);
                if (mode == 7) run(k_col_solve<MR, 8, 7, MB>, threads, col_smem(MR, 8));
                else if (mode == 1) run(k_col_solve<MR, 8, 1, MB>, threads, col_smem(MR, 8));
                else run(k_col_solve<MR, 8, 2, MB>, threads, col_smem(MR, 8));
                return;
            }
        }
        const int threads = 32 * 4 * col_groups(MR, 4);
        if (mode == 7) run(k_col_solve<MR, 4, 7, MB>, threads, col_smem(MR, 4));
        else if (mode == 1) run(k_col_solve<MR, 4, 1, MB>, threads, col_smem(MR, 4));
        else run(k_col_solve<MR, 4, 2, MB>, threads, col_smem(MR, 4));
    });
}

}  // namespace cfd
