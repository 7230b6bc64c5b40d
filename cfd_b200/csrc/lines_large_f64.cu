// lines_large_f64.cu - two-step kernels of the lengths below (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <>
const LineKernels<double2>* line_kernels_large<double2>(int n) {
    switch (n) {
        case 432: return line_table<double2, 24, 18, kLinesAll>();
        case 486: return line_table<double2, 18, 27, kLinesAll>();
        case 512: return line_table<double2, 16, 32, kLinesAll>();
        default: return nullptr;
    }
}

}  // namespace cfd
