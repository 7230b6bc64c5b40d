// lines_mid_f64.cu - two-step kernels of the lengths below (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <>
const LineKernels<double2>* line_kernels_mid<double2>(int n) {
    switch (n) {
        case 144: return line_table<double2, 12, 12, kLinesAll>();
        case 162: return line_table<double2, 18, 9, kLinesAll>();
        case 216: return line_table<double2, 12, 18, kLinesAll>();
        case 256: return line_table<double2, 16, 16, kLinesAll>();
        case 288: return line_table<double2, 16, 18, kLinesAll>();
        case 324: return line_table<double2, 18, 18, kLinesAll>();
        default: return nullptr;
    }
}

}  // namespace cfd
