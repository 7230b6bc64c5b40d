// channel_base.cuh - sizes, grid tables and complex arithmetic shared by the channel kernels.
#pragma once

#include <cuda_runtime.h>

namespace cfd {

struct Dims {
    int ngal1, ngal2, n1, n2, nkx, ncol;
    int ju0, ju1, jv0, jv1, jp0, jp1, nyu, nyv, nyp;
    int nslot;  // nyu + nyv
    int ny;     // faces from y=-1 to y=1 (input.in ny)
    // Stored layout of the spectral fields (the wall bands' column list) as seen by a launch
    // over one band (the transform kernels of the nonlinear pass): columns per plane, per kz
    // row, and the stored kz index q + qshift of the negative modes q >= n2/2; the elements
    // per slot of the half-physical buffers; the u-slots su0..su0+nsu-1 and v-slots
    // sv0..sv0+nsv-1 (0-based within their grid) of the launch.  With one band: ncol, nkx,
    // 0, ngal2*nkx, and every slot.
    int pstride, kstride, qshift;
    long long hstride;
    int su0, nsu, sv0, nsv;
    // three bands: 1, the last v face of the bottom band (N(3,1)) and the middle band's N1, N2
    int mb, jb, n1m, n2m;
};

// stored column of spectral entry (kx i, kz q) in a launch over one band
__device__ __forceinline__ size_t scol(const Dims& d, int i, int q) {
    return (size_t)(q < d.n2 / 2 ? q : q + d.qshift) * d.kstride + i;
}

// Grid and wavenumber tables on the device (array index = j - j0 of the grid).
struct Geo {
    const double* yu;
    const double* yv;
    const double* dthdyu;
    const double* dthdyv;
    const double* dyu2i;  // [nyu][3]
    const double* dyv2i;  // [nyv][3]
    const double* kx;     // [nkx]
    const double* kz;     // [n2]
    // linear y-interpolation weights (interp_u/interp_v, FOU3D.f90:261-308):
    // v at centre j = vca[j]*v(j) + vcb[j]*v(j-1)   (index j - ju0, interior centres)
    // u at face j   = ufa[j]*u(j+1) + ufb[j]*u(j)   (index j - jv0)
    const double* vca;
    const double* vcb;
    const double* ufa;
    const double* ufb;
    double gwb, gwt, gwib, gwit;
    double gw1t, gw3b;  // three bands: gridweighting(1,2) and gridweighting(3,1)
};

// three bands: the column's mode exists in the middle band too
__device__ __forceinline__ bool mb_long(const Dims& d, int i, int q) {
    return i <= d.n1m / 2 && (q < d.n2m / 2 || q >= d.n2 - d.n2m / 2);
}

__device__ __forceinline__ int row_of(const Dims& d, int q) { return q < d.n2 / 2 ? q : q + (d.ngal2 - d.n2); }

__device__ __forceinline__ double2 dc(double a, double b) { double2 r; r.x = a; r.y = b; return r; }
__device__ __forceinline__ double2 dadd(double2 a, double2 b) { return dc(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 dsub(double2 a, double2 b) { return dc(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 dscl(double s, double2 a) { return dc(s * a.x, s * a.y); }
// (i*k) * a
__device__ __forceinline__ double2 dik(double k, double2 a) { return dc(-k * a.y, k * a.x); }

template <typename T2> __device__ __forceinline__ T2 to_t2(double2 a);
template <> __device__ __forceinline__ float2 to_t2<float2>(double2 a) { return make_float2((float)a.x, (float)a.y); }
template <> __device__ __forceinline__ double2 to_t2<double2>(double2 a) { return a; }
// max that keeps a NaN (fmax drops it), so that the reductions of the diagnostics see a
// non-finite field
__device__ __forceinline__ double nan_max(double a, double b) { return (b > a || b != b) ? b : a; }
__device__ __forceinline__ double2 to_d2(float2 a) { return dc((double)a.x, (double)a.y); }
__device__ __forceinline__ double2 to_d2(double2 a) { return a; }

}  // namespace cfd
