// lines_named_f32.cu - two-step kernels of the lengths below (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <>
const LineKernels<float2>* line_kernels_named<float2>(int n) {
    switch (n) {
        case 64: return line_table<float2, 8, 8, kLinesNamed>();
        case 96: return line_table<float2, 8, 12, kLinesNamed>();
        case 128: return line_table<float2, 8, 16, kLinesNamed>();
        case 192: return line_table<float2, 16, 12, kLinesNamed>();
        case 384: return line_table<float2, 16, 24, kLinesNamed>();
        case 768: return line_table<float2, 32, 24, kLinesNamed>();
        default: return nullptr;
    }
}

}  // namespace cfd
