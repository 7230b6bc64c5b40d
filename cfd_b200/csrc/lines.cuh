// lines.cuh - the two-step transform kernels of every length, as a table of kernels per length.
//
// A length N = N1*N2 has its kernels where both factors fit a thread's registers: every even
// 2^a 3^b from 12 to 768.  They are instantiated in lines_*.cu, a few lengths each, so that the
// units compile side by side.  Against the radix-by-radix kernels that lengths other than the
// named six (64, 96, 128, 192, 384, 768) ran before, microseconds a launch on B200 (z inverse, x,
// z forward): 256 x 129 x 256 FP64 232, 602, 249 -> 46, 225, 86, FP32 177, 459, 152 -> 71, 118,
// 50; 144 x 131 x 108 FP32 70, 146, 55 -> 16, 33, 13; 24 x 17(+6) x 18 FP64 4.1, 6.1, 3.9 -> 2.2,
// 3.1, 2.3.  The shared-memory passes of those kernels, and in FP64 a slot's z transform for each
// field and slot instead of one a plane, were what they spent their time on (FP32 keeps the latter at
// these lengths, since it interpolates in FP64 before the transforms).
#pragma once

#include "field_lines.cuh"
#include "xmarch.cuh"

namespace cfd {

template <typename T2>
struct LineKernels {
    using R = decltype(T2::x);
    int n1, n2;
    void (*zinv2)(Dims, Geo, const double2*, const double2*, const double2*, T2*, T2*, T2*, const T2*, int);
    void (*zinv2s)(Dims, const double2*, const double2*, const double2*, T2*, const T2*, int);
    void (*zfwd2)(Dims, const T2*, const T2*, const T2*, const T2*, T2*, T2*, T2*, T2*, const T2*, int);
    // the FP64 z kernels at 112 registers (null for FP32 and above 384 points)
    void (*zinv2s_r)(Dims, const double2*, const double2*, const double2*, T2*, const T2*, int);
    void (*zfwd2_r)(Dims, const T2*, const T2*, const T2*, const T2*, T2*, T2*, T2*, T2*, const T2*, int);
    void (*xline2)(Dims, Geo, const T2*, T2*, T2*, T2*, T2*, const T2*, int, int);
    // tuning variants of the six named lengths: 64 registers (FP32), packed rows, line pairs (FP32)
    void (*xline2_r)(Dims, Geo, const T2*, T2*, T2*, T2*, T2*, const T2*, int, int);
    void (*xline3)(Dims, Geo, const T2*, T2*, T2*, T2*, T2*, const T2*, int);
    void (*xline4)(Dims, Geo, const T2*, T2*, T2*, T2*, T2*, const T2*, int);
    // three bands: the x-line pass on planes interpolated already
    void (*xline2b)(Dims, Geo, T2*, T2*, T2*, T2*, const T2*, int, int);
    // the x-line pass marching in y, with a split of its own (null where it has none)
    void (*xmarch)(Dims, Geo, const T2*, T2*, T2*, T2*, T2*, const T2*, int, int);
    int m1, m2;
    void (*ib_zinv)(Dims, IBSrc, int, const int*, int, T2*, const T2*, int, int);
    void (*ib_xinv)(Dims, const T2*, int, R*, const int*, int, const T2*, int, IBVel);
    void (*ib_xfwd)(Dims, T2*, int, const R*, const int*, int, const T2*, int);
    void (*ib_zfwd)(Dims, const T2*, int, IBDst, int, const int*, const unsigned char*, const T2*, int);
    // the forcing of u, w and v together
    void (*ib_zin)(Dims, IBJobs, T2*, const T2*, int);
    void (*ib_force_x)(Dims, IBJobs, IBRows, IBRows, IBVels, T2*, const T2*, int);
    void (*ib_zout)(Dims, IBJobs, const T2*, const T2*, int);
    // FP64 only (field_lines.cuh): statistics (sums, or the maxima alone), plane transforms
    // [inverse, forward][8-byte, 16-byte aligned]
    void (*st_z)(Dims, Geo, StChunk, const double2*, const double2*, const double2*, const double2*, double2*,
                 const double2*, int);
    void (*st_x[2])(Dims, Geo, StChunk, const double2*, const double2*, int, int, double*, double*, int, int, int, int);
    void (*pl_cft[2][2])(double*, int, int, int, long long, const double2*, int);
    void (*pl_rft[2][2])(double*, int, int, long long, const double2*, int);
};

// The kernels of length n, null where it has none; alt: the transposed split of the six named
// lengths (only zinv2s, zfwd2, xline2, their variants, ib_zin and ib_zout).
template <typename T2> const LineKernels<T2>* line_kernels(int n, bool alt = false);

// What a context runs where cfd_tuning does not say: x-line path, radix order and rows by its x length,
// radix order and lines by its z length.  The transposed split is the default where both x and z lines
// gain by it, and at 768 points in FP64 for z alone; microseconds a launch, plain | transposed (z inverse,
// x-line, z forward; n x planes x n):
//   64 x 97    FP64 3.8 12.4 5.3 | 5.4 23.8 8.0        FP32 3.7 10.0 4.2 | 3.9 16.9 5.9
//   96 x 129   FP64 11.6 40.1 12.4 | 11.6 35.9 14.4    FP32 6.6 24.3 8.5 | 7.0 25.0 8.8
//   128 x 129  FP64 17.6 78.4 22.1 | 18.4 78.2 28.2    FP32 14.9 42.0 13.1 | 15.5 52.3 15.2
//   192 x 193  FP64 45.7 229 77.6 | 41.4 208 74.1      FP32 38.8 136 49.7 | 29.3 116 40.5
//   384 x 129  FP64 117 574 226 | 128 612 224          FP32 72.1 325 114 | 79.0 340 127
//   768 x 65   FP64 324 1730 715 | 322 1905 626        FP32 210 810 332 | 163 739 299
// (the last in 2 and 8 x rows, 4 and 8 z lines; FP32 x lines in 4 rows 818 plain).  The 64-register x-line
// (path 5) at 192 points: 119 | 109 us; the march (path 6) at 384: 470 us against 637 on 257 planes.
struct LineDefaults {
    int xpath = 1, xsplit = 1, xrows = 4, zsplit = 1, zlines = 8;
};
inline LineDefaults line_defaults(int n, bool f32) {
    LineDefaults k;
    if (f32) k.zlines = 16;
    if (n == 192) { k.xsplit = k.zsplit = 2; if (f32) k.xpath = 5; }
    if (n == 384 && f32) k.xpath = 6;
    if (n == 768) {
        k.zsplit = 2;
        k.zlines = f32 ? 8 : 4;
        if (f32) { k.xsplit = 2; k.xrows = 8; }
    }
    return k;
}

// what each unit holds (null for the lengths it does not)
template <typename T2> const LineKernels<T2>* line_kernels_named(int n);
template <typename T2> const LineKernels<T2>* line_kernels_alt(int n);
template <typename T2> const LineKernels<T2>* line_kernels_small(int n);
template <typename T2> const LineKernels<T2>* line_kernels_mid(int n);
template <typename T2> const LineKernels<T2>* line_kernels_large(int n);
template <typename T2> const LineKernels<T2>* line_kernels_large2(int n);
template <> const LineKernels<float2>* line_kernels_named<float2>(int n);
template <> const LineKernels<double2>* line_kernels_named<double2>(int n);
template <> const LineKernels<float2>* line_kernels_alt<float2>(int n);
template <> const LineKernels<double2>* line_kernels_alt<double2>(int n);
template <> const LineKernels<float2>* line_kernels_small<float2>(int n);
template <> const LineKernels<double2>* line_kernels_small<double2>(int n);
template <> const LineKernels<float2>* line_kernels_mid<float2>(int n);
template <> const LineKernels<double2>* line_kernels_mid<double2>(int n);
template <> const LineKernels<float2>* line_kernels_large<float2>(int n);
template <> const LineKernels<double2>* line_kernels_large<double2>(int n);
template <> const LineKernels<float2>* line_kernels_large2<float2>(int n);
template <> const LineKernels<double2>* line_kernels_large2<double2>(int n);
template <> const LineKernels<float2>* line_kernels<float2>(int n, bool alt);
template <> const LineKernels<double2>* line_kernels<double2>(int n, bool alt);

// Splits of the marching x-line pass: its second step holds 8 or 16 points per lane, so that the
// unpack partners kb and N2 - kb share a warp
template <int N> struct MarchSplit { static constexpr int N1 = 0, N2 = 0; };
template <> struct MarchSplit<64> { static constexpr int N1 = 8, N2 = 8; };
template <> struct MarchSplit<96> { static constexpr int N1 = 12, N2 = 8; };
template <> struct MarchSplit<128> { static constexpr int N1 = 8, N2 = 16; };
template <> struct MarchSplit<192> { static constexpr int N1 = 12, N2 = 16; };
template <> struct MarchSplit<256> { static constexpr int N1 = 16, N2 = 16; };
template <> struct MarchSplit<288> { static constexpr int N1 = 18, N2 = 16; };
template <> struct MarchSplit<384> { static constexpr int N1 = 24, N2 = 16; };
template <> struct MarchSplit<432> { static constexpr int N1 = 27, N2 = 16; };
template <> struct MarchSplit<576> { static constexpr int N1 = 36, N2 = 16; };
template <> struct MarchSplit<512> { static constexpr int N1 = 32, N2 = 16; };

// where it is built: FP32 as x-line path 6 of its lengths, FP64 where it is the default
template <typename T2> constexpr bool march_length(int n) {
    return sizeof(T2) == 8 ? true : n >= 256 && n <= 512;
}

enum { kLinesAll, kLinesNamed, kLinesAlt };

template <typename T2, int N1, int N2, int WHAT>
const LineKernels<T2>* line_table() {
    constexpr bool F32 = sizeof(T2) == 8;
    static const LineKernels<T2> k = [] {
        LineKernels<T2> t{};
        t.n1 = N1;
        t.n2 = N2;
        t.zinv2s = k_zinv2s<T2, N1, N2>;
        t.zfwd2 = k_zfwd2<T2, N1, N2>;
        t.xline2 = k_xline2<T2, N1, N2>;
        t.ib_zin = k_ib_zin<T2, N1, N2>;
        t.ib_zout = k_ib_zout<T2, N1, N2>;
        if constexpr (!F32 && N1 * N2 <= 384) {
            t.zinv2s_r = k_zinv2sd<N1, N2>;
            t.zfwd2_r = k_zfwd2d<N1, N2>;
        }
        if constexpr (F32 && WHAT != kLinesAll) t.xline2_r = k_xline2r<N1, N2>;
        if constexpr (WHAT == kLinesNamed) {
            t.xline3 = k_xline3<T2, N1, N2>;
            if constexpr (F32) t.xline4 = k_xline4<N1, N2>;
        }
        using MS = MarchSplit<N1 * N2>;
        if constexpr (WHAT != kLinesAlt && MS::N1 > 0 && march_length<T2>(N1 * N2)) {
            t.xmarch = k_xmarch<T2, MS::N1, MS::N2>;
            t.m1 = MS::N1;
            t.m2 = MS::N2;
        }
        if constexpr (WHAT != kLinesAlt) {
            t.zinv2 = k_zinv2<T2, N1, N2>;
            t.xline2b = k_xline2b<T2, N1, N2>;
            t.ib_zinv = k_ib_zinv2<T2, N1, N2>;
            t.ib_xinv = k_ib_xinv2<T2, N1, N2>;
            t.ib_xfwd = k_ib_xfwd2<T2, N1, N2>;
            t.ib_zfwd = k_ib_zfwd2<T2, N1, N2>;
            t.ib_force_x = k_ib_force_x<T2, N1, N2>;
        }
        if constexpr (WHAT != kLinesAlt && !F32) {
            t.st_z = k_st_z<N1, N2>;
            t.st_x[0] = k_st_x<N1, N2, false>;
            t.st_x[1] = k_st_x<N1, N2, true>;
            t.pl_cft[0][0] = k_pl_cft<N1, N2, +1, false>;
            t.pl_cft[0][1] = k_pl_cft<N1, N2, +1, true>;
            t.pl_cft[1][0] = k_pl_cft<N1, N2, -1, false>;
            t.pl_cft[1][1] = k_pl_cft<N1, N2, -1, true>;
            t.pl_rft[0][0] = k_pl_rft_inv<N1, N2, false>;
            t.pl_rft[0][1] = k_pl_rft_inv<N1, N2, true>;
            t.pl_rft[1][0] = k_pl_rft_fwd<N1, N2, false>;
            t.pl_rft[1][1] = k_pl_rft_fwd<N1, N2, true>;
        }
        return t;
    }();
    return &k;
}

}  // namespace cfd
