// field_lines.cuh - FP64 two-step transforms of the statistics pass, the CFL query and the plane
// entry points (sm_100a).
//
// Statistics (stats.f90:1-253) and dtc_calc (FOU3D.f90:516-544) reduce physical planes of u, v, w,
// the y-interpolated v and w, omega_x and p.  Interpolation in y is linear and commutes with the
// transforms, so each field is transformed in z once on its own planes (k_st_z; omega_x as a field of
// its own), and k_st_x forms the sources of a row from the transformed planes,
// transforms them in x and reduces the physical values in registers: no physical plane is stored.
// The planes go through in chunks whose transformed fields stay in L2.  The passes they replace
// (planes built, transformed in place by radix-by-radix kernels and read again by the sums) moved 17
// GB at 384 x 257(+90) x 384, 19.2 ms for a statistics call and a CFL query; here 3.7 ms, bound by the
// FP64 transforms' latency at 12 warps an SM (k_st_x 85 us, k_st_z 27 us per 16 planes).  The plane
// entry points (k_pl_cft, k_pl_rft_inv, k_pl_rft_fwd) take a line through shared memory once instead of
// once a radix: 193 planes of 192 x 192, both ways, 264 -> 82 us.
#pragma once

#include "transform_kernels.cuh"

namespace cfd {

// One chunk: u planes j0..j0+cp-1, v and p planes of the same index, and the neighbours their
// interpolations read.  Field f (u, w, v, omega_x, p) holds planes first[f]..first[f]+n[f]-1 of its
// grid (those that exist) from slot off[f] on.
struct StChunk {
    int j0, cp;
    int off[5], first[5], n[5];
};
constexpr int kStQ = 13;  // conditional quantities: U U2 W W2 UV UW, V V2 wx wx2 VW, P P2

template <int TN1, int TN2>
__global__ void __launch_bounds__(8 * (TN1 > TN2 ? TN1 : TN2), (TN1 > TN2 ? TN1 : TN2) <= 24 ? 3 : 2)
    k_st_z(Dims d, Geo g, StChunk s, const double2* __restrict__ u1, const double2* __restrict__ u2,
           const double2* __restrict__ u3, const double2* __restrict__ p, double2* __restrict__ Hs,
           const double2* __restrict__ twz, int lb) {
    constexpr int N = TN1 * TN2;
    const int f = blockIdx.y;
    const int nlines = s.n[f] * d.nkx;
    const int line0 = blockIdx.x << lb;
    if (line0 >= nlines) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* twt = reinterpret_cast<double2*>(smem_raw);
    double2* ex = twt + N;
    load_twiddles<double2, TN1, TN2>(twt, twz);
    const int b = threadIdx.x & ((1 << lb) - 1);
    const int line = min(line0 + b, nlines - 1);
    const int pl = line / d.nkx, i = line - pl * d.nkx;
    const int ny = f < 2 ? d.nyu : (f < 4 ? d.nyv : d.nyp);
    const int j = s.first[f] + pl;
    const bool live = line0 + b < nlines && j >= 0 && j < ny;
    const int jc = min(max(j, 0), ny - 1);
    const double2* src = (f == 0 ? u1 : (f == 1 ? u3 : (f < 4 ? u2 : p))) + (size_t)jc * d.ncol + i;
    double2* H = Hs + ((size_t)s.off[f] + pl) * N * d.nkx + i;
    const int r = threadIdx.x >> lb;
    __syncthreads();
    auto store = [&](int z, int, double2 v) {
        if (live) H[(size_t)z * d.nkx] = v;
    };
    if (f == 3) {  // omega_x = dw/dy - dv/dz at the face: w is differenced before its rounding by a transform
        const double2* w = u3 + (size_t)jc * d.ncol + i;
        const double dth = g.dthdyv[jc];
        auto load = [&](int e, int) -> double2 {
            const int q = zrow_q<N, TN2>(e, r);
            if (q < 0) return dc(0, 0);
            const size_t o = (size_t)q * d.nkx;
            const double2 a = dscl(dth, dsub(w[o + d.ncol], w[o]));
            // the kz = -N2/2 mode of a z derivative is zero (der_z, FOU3D.f90:388-412)
            return q == d.n2 / 2 ? a : dsub(a, dik(g.kz[q], src[o]));
        };
        two_step_lines<double2, TN1, TN2, +1>(lb, ex, twt, load, store);
        return;
    }
    auto load = [&](int e, int) -> double2 {
        const int q = zrow_q<N, TN2>(e, r);
        return q < 0 ? dc(0, 0) : src[(size_t)q * d.nkx];
    };
    two_step_lines<double2, TN1, TN2, +1>(lb, ex, twt, load, store);
}

// |a| as its bit pattern, which orders like the value and puts NaN above all: a maximum that keeps
// NaN without the FP64 unit
__device__ __forceinline__ unsigned long long mag_bits(double a) {
    return (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
}

// line slots of a k_st_x CTA, the pitch of a line's exchange, and for a pair of rows the lines
// transformed and the slots they take (a power of two: adjacent lanes in the second step)
__host__ __device__ constexpr int st_x_lines(int n1, int n2) { return (n1 > n2 ? n1 : n2) >= 16 ? 8 : 16; }
__host__ __device__ constexpr int st_x_row(int n1, int n2) { return n1 * (n2 + 1) > n1 * n2 ? n1 * (n2 + 1) + 1 : n1 * n2 + 1; }
__host__ __device__ constexpr int st_x_used(bool acc) { return acc ? 7 : 3; }
__host__ __device__ constexpr int st_x_slots(bool acc) { return acc ? 8 : 4; }

// A CTA: P row pairs of plane index jr = j0 + blockIdx.y.  A complex line is one quantity on the two rows
// of a pair (row z + i row z + 1), so that its rounding is relative to that quantity alone; lines 0.. of
// a pair:  ACC: u, w, v(centre), p, v, w(face), omega_x;  else: u, w, v.
// part[((jr*gridDim.x + blockIdx.x)*slots + l)*4 + q]: of line l, the sums of a, a^2 and a*o (o: w for
// u, u for v(centre), w(face) for v) and the maximum of |a| over the points of the CTA's rows
// (omega_x over the first N1 x N2 points, stats.f90:53-60).  With pc, on the planes of a band (its
// nbu, nbv, nbp planes from either end): pc[((pl*ngal2 + z)*kStQ + q)*dnx + ti], row z folded
// onto a tile of dnx points.
template <int TN1, int TN2, bool ACC>
__global__ void __launch_bounds__((st_x_lines(TN1, TN2) * (TN1 > TN2 ? TN1 : TN2) + 31) / 32 * 32, 2)
    k_st_x(Dims d, Geo g, StChunk s, const double2* __restrict__ Hs, const double2* __restrict__ twx, int P, int lp,
           double* __restrict__ part, double* __restrict__ pc, int dnx, int nbu, int nbv, int nbp) {
    constexpr int N = TN1 * TN2, HX = N / 3, NK = HX + 1, NU = st_x_used(ACC), NL = st_x_slots(ACC);
    constexpr int LX = st_x_row(TN1, TN2);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double red[16][NL][4];
    double2* twt = reinterpret_cast<double2*>(smem_raw);
    double2* ex = twt + N;
    load_twiddles<double2, TN1, TN2>(twt, twx);
    const int t = threadIdx.x, z0 = blockIdx.x * 2 * P, jr = s.j0 + blockIdx.y;
    __syncthreads();
    // ---- inverse N1-point DFTs, thread (line b, column n2)
    if (t < P * NU * TN2) {
        const int b = (unsigned)t / TN2, n2 = t - b * TN2;
        const int pr = b / NU, l = b - pr * NU, z = min(z0 + 2 * pr, d.ngal2 - 2);
        auto F = [&](int f, int j) { return Hs + ((size_t)(s.off[f] + j - s.first[f]) * d.ngal2 + z) * NK; };
        // a0 A0 + a1 A1 of either row
        const double2 *A0 = F(0, jr), *A1 = A0;
        double a0 = 0, a1 = 0;
        if (l < 2) {
            A0 = F(l, jr); a0 = 1.0;
        } else if (ACC && l == 2) {  // interp_v with its ghost centres (FOU3D.f90:285-308)
            int j;
            if (jr == 0) {
                j = 1; a0 = (1.0 - g.gwib) * g.vca[1]; a1 = g.gwib + (1.0 - g.gwib) * g.vcb[1];
            } else if (jr == d.nyu - 1) {
                j = jr - 1; a0 = g.gwit + (1.0 - g.gwit) * g.vca[j]; a1 = (1.0 - g.gwit) * g.vcb[j];
            } else {
                j = jr; a0 = g.vca[jr]; a1 = g.vcb[jr];
            }
            A0 = F(2, j); A1 = F(2, j - 1);
        } else if (ACC && l == 3) {
            if (jr < d.nyp) { A0 = F(4, jr); a0 = 1.0; }
        } else if (jr < d.nyv) {
            if (l == (ACC ? 4 : 2)) {
                A0 = F(2, jr); a0 = 1.0;
            } else if (l == 5) {  // w at the face
                A0 = F(1, jr + 1); a0 = g.ufa[jr]; A1 = F(1, jr); a1 = g.ufb[jr];
            } else {  // omega_x
                A0 = F(3, jr); a0 = 1.0;
            }
        }
        const bool two = a1 != 0.0;
        auto fetch = [&](int k) {
            const double2 a = dscl(a0, A0[k]);
            return two ? dadd(a, dscl(a1, A1[k])) : a;
        };
        double2 v[TN1];
#pragma unroll
        for (int n1 = 0; n1 < TN1; ++n1) {
            const int e0 = n1 * TN2, e = e0 + n2;
            const bool lo = (e0 + TN2 - 1 <= HX) || (e0 <= HX && e <= HX);
            const bool hi = (e0 >= N - HX) || (e0 + TN2 - 1 >= N - HX && e >= N - HX);
            double2 val = dc(0, 0);
            if (lo) {  // the inverse real transform ignores Im of kx = 0
                double2 a = fetch(e), c = fetch(NK + e);
                if (n1 == 0 && n2 == 0) { a.y = 0; c.y = 0; }
                val = dc(a.x - c.y, a.y + c.x);
            } else if (hi) {
                const double2 a = fetch(N - e), c = fetch(NK + N - e);
                val = dc(a.x + c.y, -a.y + c.x);
            }
            v[n1] = val;
        }
        rdft_z<TN1, +1, gap_blocks<TN1, TN2, HX>()>(v);
        double2* o = ex + (size_t)b * LX + n2;
#pragma unroll
        for (int k1 = 0; k1 < TN1; ++k1) o[k1 * (TN2 + 1)] = k1 == 0 ? v[0] : cmulc(v[k1], twt[k1 * TN2 + n2]);
    }
    __syncthreads();
    // ---- inverse N2-point DFTs -> x = k1 + N1 k2; the lines of a pair in adjacent lanes
    const int l = t & (NL - 1), rest = t / NL, pr = rest & (P - 1), k1 = min(rest >> lp, TN1 - 1);
    const bool act = t < P * NL * TN1 && l < NU;
    const int b = pr * NU + min(l, NU - 1), z = z0 + 2 * pr;
    // the lane of the line that this one is multiplied with
    const int src = (t & 31 & ~(NL - 1)) | (l == 0 ? 1 : (l == 2 ? 0 : (l == 4 ? 5 : l)));
    double2 y[TN2];
    double q[3] = {0, 0, 0};
    unsigned long long ma = 0;
    if ((t & ~31) < P * NL * TN1) {
        const double2* o = ex + (size_t)b * LX + k1 * (TN2 + 1);
#pragma unroll
        for (int n2 = 0; n2 < TN2; ++n2) y[n2] = o[n2];
        rdft<TN2, +1>(y);
        // (omega_x: N2 is even, so both rows of a pair count or neither)
        const bool wx = ACC && l == 6, in = act && z < (wx ? d.n2 : d.ngal2);
#pragma unroll
        for (int k2 = 0; k2 < TN2; ++k2) {
            const double a = y[k2].x, c = y[k2].y;
            double oa = 0.0, oc = 0.0;
            if (ACC) {
                oa = __shfl_sync(0xffffffffu, a, src);
                oc = __shfl_sync(0xffffffffu, c, src);
            }
            if (in && (!wx || k1 + TN1 * k2 < d.n1)) {
                if (ACC) {
                    q[0] += a + c;
                    q[1] += a * a + c * c;
                    q[2] += a * oa + c * oc;
                }
                ma = max(ma, max(mag_bits(a), mag_bits(c)));
            }
        }
#pragma unroll
        for (int o2 = NL; o2 < 32; o2 <<= 1) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (ACC) q[k] += __shfl_xor_sync(0xffffffffu, q[k], o2);
            ma = max(ma, __shfl_xor_sync(0xffffffffu, ma, o2));
        }
    }
    if ((t & 31) < NL) {
        double* o = red[t >> 5][t & 31];
#pragma unroll
        for (int k = 0; k < 3; ++k) o[k] = q[k];
        o[3] = __longlong_as_double((long long)ma);
    }
    __syncthreads();
    if (t < NL * 4) {
        const int lr = t >> 2, k = t & 3, nw = (blockDim.x + 31) >> 5;
        double v = red[0][lr][k];
        for (int w = 1; w < nw; ++w) v = k < 3 ? v + red[w][lr][k] : nan_max(v, red[w][lr][k]);
        part[((size_t)jr * gridDim.x + blockIdx.x) * NL * 4 + t] = v;
    }
    if constexpr (ACC) {
        auto band = [&](int ny, int nb) { return jr < ny && (jr < nb || ny - 1 - jr < nb); };
        if (pc == nullptr || !(band(d.nyu, nbu) || band(d.nyv, nbv) || band(d.nyp, nbp))) return;
        if (act)  // the exchange has been read: it takes the physical rows
#pragma unroll
            for (int k2 = 0; k2 < TN2; ++k2) ex[(size_t)b * LX + k1 + TN1 * k2] = y[k2];
        __syncthreads();
        const int ntx = N / dnx;
        for (int it = t; it < 2 * P * 3 * dnx; it += blockDim.x) {
            const int ti = it % dnx, gq = (it / dnx) % 3, row = it / (3 * dnx);
            if (z0 + row >= d.ngal2) break;
            // point x of line r of the row's pair, at 2 x
            auto line = [&](int r) { return reinterpret_cast<const double*>(ex + (size_t)((row >> 1) * NU + r) * LX + ti) + (row & 1); };
            const double *L0 = line(gq == 0 ? 0 : (gq == 1 ? 4 : 3)), *L1 = line(gq == 0 ? 1 : (gq == 1 ? 6 : 3)),
                         *L2 = line(gq == 0 ? 2 : (gq == 1 ? 5 : 3));
            double f[6] = {0, 0, 0, 0, 0, 0};
            for (int ix = 0; ix < ntx; ++ix) {
                const double m = L0[2 * ix * dnx];
                f[0] += m; f[1] += m * m;
                if (gq < 2) {  // u, w, v(centre) or v, omega_x, w(face)
                    const double n = L1[2 * ix * dnx];
                    f[2] += n; f[3] += n * n; f[4] += m * L2[2 * ix * dnx];
                    if (gq == 0) f[5] += m * n;
                }
            }
            double* o = pc + (((size_t)blockIdx.y * d.ngal2 + z0 + row) * kStQ + (gq == 0 ? 0 : (gq == 1 ? 6 : 11))) * dnx + ti;
            const int nq = gq == 0 ? 6 : (gq == 1 ? 5 : 2);
#pragma unroll
            for (int k = 0; k < 6; ++k)
                if (k < nq) o[(size_t)k * dnx] = f[k];
        }
    }
}

// ---- plane entry points ---------------------------------------------------------------
// cft (cft_buff.f:1-65): complex lines of length N in place, element stride ise and line stride isa
// in doubles, batch stride bstride; inverse (SIGN +1) unscaled, forward x 1/N.  A2: pairs lie on 16
// bytes.  grid: x = line chunk, y = batch.
template <int TN1, int TN2, int SIGN, bool A2>
__global__ void __launch_bounds__(8 * (TN1 > TN2 ? TN1 : TN2), (TN1 > TN2 ? TN1 : TN2) <= 24 ? 3 : 2)
    k_pl_cft(double* __restrict__ c, int ise, int isa, int m, long long bstride, const double2* __restrict__ tw, int lb) {
    constexpr int N = TN1 * TN2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* twt = reinterpret_cast<double2*>(smem_raw);
    double2* ex = twt + N;
    load_twiddles<double2, TN1, TN2>(twt, tw);
    const int l = (blockIdx.x << lb) + (threadIdx.x & ((1 << lb) - 1));
    const bool live = l < m;
    double* x = c + (size_t)blockIdx.y * bstride + (size_t)min(l, m - 1) * isa;
    __syncthreads();
    auto load = [&](int e, int) -> double2 {
        double* a = x + (size_t)e * ise;
        if (A2) return *reinterpret_cast<double2*>(a);
        return dc(a[0], a[1]);
    };
    auto store = [&](int e, int, double2 v) {
        if (!live) return;
        double* a = x + (size_t)e * ise;
        if (SIGN < 0) v = dscl(1.0 / N, v);
        if (A2) *reinterpret_cast<double2*>(a) = v;
        else { a[0] = v.x; a[1] = v.y; }
    };
    two_step_lines<double2, TN1, TN2, SIGN>(lb, ex, twt, load, store);
}

// rft (rft_buff.f:24-86): real lines of length N in place, stride isa doubles.  grid: x = line chunk, y =
// batch.  A stated number of CTAs per SM lets the compiler keep more loads in flight (inverse at 192
// points: 128 registers instead of 92, 193 x 192 lines 27.2 -> 24.2 us).
//
// Inverse: two lines 2b and 2b+1 a complex transform, x_a + i x_b from the Hermitian extensions of the
// half spectra (Im of modes 0 and N/2 ignored); nl transforms a CTA.
template <int TN1, int TN2, bool A2>
__global__ void __launch_bounds__((8 * (TN1 > TN2 ? TN1 : TN2) + 31) / 32 * 32, (TN1 > TN2 ? TN1 : TN2) <= 16 ? 4 : ((TN1 > TN2 ? TN1 : TN2) <= 24 ? 2 : 1))
    k_pl_rft_inv(double* __restrict__ c, int isa, int m, long long bstride, const double2* __restrict__ tw, int nl) {
    constexpr int N = TN1 * TN2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* twt = reinterpret_cast<double2*>(smem_raw);
    double2* ex = twt + N;
    load_twiddles<double2, TN1, TN2>(twt, tw);
    double* base = c + (size_t)blockIdx.y * bstride;
    const int l0 = blockIdx.x * nl;
    // (a line past the last repeats it in the transform and is not stored)
    auto line = [&](int i) { return base + (size_t)min(i, m - 1) * isa; };
    __syncthreads();
    auto load = [&](int e, int b) -> double2 {
        const int k = e <= N / 2 ? e : N - e;
        const double *xa = line(2 * (l0 + b)) + 2 * k, *xb = line(2 * (l0 + b) + 1) + 2 * k;
        double2 A, Bv;
        if (A2) { A = *reinterpret_cast<const double2*>(xa); Bv = *reinterpret_cast<const double2*>(xb); }
        else { A = dc(xa[0], xa[1]); Bv = dc(xb[0], xb[1]); }
        if (k == 0 || k == N / 2) { A.y = 0; Bv.y = 0; }
        if (e > N / 2) { A.y = -A.y; Bv.y = -Bv.y; }
        return dc(A.x - Bv.y, A.y + Bv.x);
    };
    auto store = [&](int x, int b, double2 v) {
        const int i = 2 * (l0 + b);
        if (i < m) base[(size_t)i * isa + x] = v.x;
        if (i + 1 < m) base[(size_t)(i + 1) * isa + x] = v.y;
    };
    two_step_lines<double2, TN1, TN2, +1, false>(0, ex, twt, load, store, nl);
}

// Forward: a line by itself, x 1/N, Re and Im of modes 0..N/2 with zero Im at both ends.  (Two lines in
// one complex transform share their rounding: a small line would carry that of its neighbour, and a
// NaN would spoil both.)  The N1-point DFTs of real columns are Hermitian in k1, so the second step
// takes k1 <= N1/2 only: with X_(N-k) = conj X_k its outputs are the whole half spectrum, half the
// work and the exchange of a complex line, and nothing is left to unpack: 193 x 192 lines of 192 points
// 20.5 us (28.2 in pairs), 40 x 384 of 384 25.5, 12 x 768 of 768 34.6.  TN1 is even.
__host__ __device__ constexpr int rft_rows(int n1, int n2) { return n2 > n1 / 2 + 1 ? n2 : n1 / 2 + 1; }
__host__ __device__ constexpr int rft_pitch(int n1, int n2) { return ((n1 / 2 + 1) * (n2 + 1)) | 1; }
template <int TN1, int TN2, bool A2>
__global__ void __launch_bounds__((8 * rft_rows(TN1, TN2) + 31) / 32 * 32, (TN1 > TN2 ? TN1 : TN2) <= 16 ? 4 : ((TN1 > TN2 ? TN1 : TN2) <= 24 ? 2 : 1))
    k_pl_rft_fwd(double* __restrict__ c, int isa, int m, long long bstride, const double2* __restrict__ tw, int nl) {
    static_assert(TN1 % 2 == 0, "an even first step");
    constexpr int N = TN1 * TN2, H1 = TN1 / 2 + 1, LX = rft_pitch(TN1, TN2);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* twt = reinterpret_cast<double2*>(smem_raw);  // twt[k1 * TN2 + n2], k1 < H1
    double2* ex = twt + H1 * TN2;
    for (int i = threadIdx.x; i < H1 * TN2; i += blockDim.x) twt[i] = tw[(i / TN2) * (i % TN2)];
    double* base = c + (size_t)blockIdx.y * bstride;
    const int l0 = blockIdx.x * nl, t = threadIdx.x;
    __syncthreads();
    if (t < nl * TN2) {
        const int b = t / TN2, n2 = t - b * TN2;
        // (a line past the last repeats it in the transform and is not stored)
        const double* x = base + (size_t)min(l0 + b, m - 1) * isa + n2;
        double2 v[TN1];
#pragma unroll
        for (int n1 = 0; n1 < TN1; ++n1) v[n1] = dc(x[n1 * TN2], 0.0);
        rdft<TN1, -1>(v);
        double2* o = ex + (size_t)b * LX + n2;
#pragma unroll
        for (int k1 = 0; k1 < H1; ++k1) o[k1 * (TN2 + 1)] = k1 == 0 ? v[0] : cmul(v[k1], twt[k1 * TN2 + n2]);
    }
    __syncthreads();
    if (t < nl * H1) {
        const int b = t / H1, k1 = t - b * H1;
        const double2* o = ex + (size_t)b * LX + k1 * (TN2 + 1);
        double2 y[TN2];
#pragma unroll
        for (int n2 = 0; n2 < TN2; ++n2) y[n2] = o[n2];
        rdft<TN2, -1>(y);
        if (l0 + b >= m) return;
        double* x = base + (size_t)(l0 + b) * isa;
        const bool self = k1 == 0 || k1 == TN1 / 2;  // holds both k and N - k
#pragma unroll
        for (int k2 = 0; k2 < TN2; ++k2) {
            const int e = k1 + TN1 * k2;
            const bool low = e <= N / 2;
            if (!low && self) continue;
            const int k = low ? e : N - e;
            double2 v = dscl(1.0 / N, y[k2]);
            if (!low) v.y = -v.y;
            if (k == 0 || k == N / 2) v.y = 0.0;
            if (A2) *reinterpret_cast<double2*>(x + 2 * k) = v;
            else { x[2 * k] = v.x; x[2 * k + 1] = v.y; }
        }
    }
}

}  // namespace cfd
