// lines.cu - lookup of the two-step kernels of a length (lines.cuh).
#include "lines.cuh"

namespace cfd {

template <typename T2>
static const LineKernels<T2>* find(int n, bool alt) {
    if (alt) return line_kernels_alt<T2>(n);
    const LineKernels<T2>* k = line_kernels_named<T2>(n);
    if (!k) k = line_kernels_small<T2>(n);
    if (!k) k = line_kernels_mid<T2>(n);
    if (!k) k = line_kernels_large<T2>(n);
    if (!k) k = line_kernels_large2<T2>(n);
    return k;
}

template <> const LineKernels<float2>* line_kernels<float2>(int n, bool alt) { return find<float2>(n, alt); }
template <> const LineKernels<double2>* line_kernels<double2>(int n, bool alt) { return find<double2>(n, alt); }

}  // namespace cfd
