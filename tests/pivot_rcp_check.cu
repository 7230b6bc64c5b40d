// The reciprocal of the column solves' pivots (pivot_rcp, colsolve.cuh) against 1/x: within one unit in the
// last place over normal values whose reciprocal is normal too, either sign.
#include <cstdio>

#include "../cfd_b200/csrc/colsolve.cuh"

__global__ void k_check(unsigned long long* worst) {
    unsigned long long w = 0, s = 0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
    for (int it = 0; it < 4096; ++it) {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;  // xorshift64
        unsigned long long m = s >> 12;           // 52 bits
        if (it < 8) m = (it & 1) ? 0xfffffffffffffull - it / 2 : it / 2;  // next to the powers of two
        const unsigned long long e = 23 + (s & 0x7ff) % 2000;           // 2^-1000 .. 2^999
        const double x = __longlong_as_double((long long)((s & 0x800) << 52 | e << 52 | m));
        const long long d = __double_as_longlong(cfd::pivot_rcp(x)) - __double_as_longlong(1.0 / x);
        const unsigned long long a = d < 0 ? -d : d;
        if (a > w) w = a;
    }
    atomicMax(worst, w);
}

int main() {
    unsigned long long *d, h = 0;
    if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 2;
    k_check<<<1024, 256>>>(d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    std::printf("%llu\n", h);
    return h > 1;
}
