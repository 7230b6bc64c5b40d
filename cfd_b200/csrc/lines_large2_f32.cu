// lines_large2_f32.cu - two-step kernels of the lengths below (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <>
const LineKernels<float2>* line_kernels_large2<float2>(int n) {
    switch (n) {
        case 576: return line_table<float2, 24, 24, kLinesAll>();
        case 648: return line_table<float2, 24, 27, kLinesAll>();
        default: return nullptr;
    }
}

}  // namespace cfd
