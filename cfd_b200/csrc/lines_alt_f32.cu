// lines_alt_f32.cu - two-step kernels of the lengths below (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <>
const LineKernels<float2>* line_kernels_alt<float2>(int n) {
    switch (n) {
        case 64: return line_table<float2, 16, 4, kLinesAlt>();
        case 96: return line_table<float2, 12, 8, kLinesAlt>();
        case 128: return line_table<float2, 16, 8, kLinesAlt>();
        case 192: return line_table<float2, 12, 16, kLinesAlt>();
        case 384: return line_table<float2, 24, 16, kLinesAlt>();
        case 768: return line_table<float2, 24, 32, kLinesAlt>();
        default: return nullptr;
    }
}

}  // namespace cfd
