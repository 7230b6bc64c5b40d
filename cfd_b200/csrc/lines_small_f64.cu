// lines_small_f64.cu - two-step kernels of the lengths below (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <>
const LineKernels<double2>* line_kernels_small<double2>(int n) {
    switch (n) {
        case 12: return line_table<double2, 4, 3, kLinesAll>();
        case 16: return line_table<double2, 4, 4, kLinesAll>();
        case 18: return line_table<double2, 6, 3, kLinesAll>();
        case 24: return line_table<double2, 4, 6, kLinesAll>();
        case 32: return line_table<double2, 4, 8, kLinesAll>();
        case 36: return line_table<double2, 6, 6, kLinesAll>();
        case 48: return line_table<double2, 8, 6, kLinesAll>();
        case 54: return line_table<double2, 6, 9, kLinesAll>();
        case 72: return line_table<double2, 8, 9, kLinesAll>();
        case 108: return line_table<double2, 12, 9, kLinesAll>();
        default: return nullptr;
    }
}

}  // namespace cfd
