// colsolve.cuh - the implicit column solves of a substep on one chip pass (sm_100a).
//
// LUsolU/LUsolV (tridLU_3D_IB.f90:50-160), solveP/LUsolP (littleharsh.f90:556-611) and v_corr
// (:796-907) act on one (kx,kz) column at a time.  As three thread-per-column sweeps they move
// 448 bytes per column and plane (y and the scaled upper diagonals go through HBM and back);
// the column itself needs 128: the three right-hand sides and p read once, u, v, w, p written
// once.  So a warp takes a column, and the column stays in shared memory from the load of its
// right-hand sides to the store of the corrected velocities.
//
// One warp solves a tridiagonal system by partition: lane s holds the M rows s*M..s*M+M-1.  It
// eliminates its first M-1 rows downwards, keeping x_i = y_i - l_i X(s-1) - c_i x_(i+1) with X
// the last row of each lane, and on the way the first row in terms of X(s-1) and X(s).  The 32
// unknowns X then satisfy a tridiagonal system, one row per lane, which five steps of parallel
// cyclic reduction solve through shuffles; the back substitution is local again.  The matrices
// are diagonally dominant (strictly for the Helmholtz rows, weakly for D.G at kx = kz = 0, whose
// bottom row is pinned), as the elimination without pivoting of the reference assumes too.
//
// Four warps form a group that owns four adjacent columns: TMA brings their rows in 64-byte
// pieces (box = 4 columns x up to 256 planes, rows past the grid's end filled with zeros) and
// takes the results back.  The 64-byte swizzle and an odd M put the rows the eight lanes of a
// shared-memory phase touch, M apart, in distinct banks.  A persistent CTA runs as many groups
// as fit beside the coefficient table they share, each on its own columns with its own barriers,
// so that one group's transfers overlap another's elimination.  Where the planes lie far apart
// (col_cols) a group owns eight columns, so that a row it touches brings 128 bytes.
//
// Measured on B200, microseconds per substep against the sweeps (k_solve_uvw + k_solve_p): 323
// against 839 at 384 x 257(+90) x 384, 76 against 375 at 192 x 193(+90) x 192, 10 against 156 at
// 64 x 97(+56) x 64, 2091 against 4527 at 768 x 385(+90) x 768.  At the first size that is 0.69
// of the copy bandwidth on the 128 bytes; what is left is the latency of the elimination at the
// 12 warps an SM holds (FP64 units 22 % busy, shared memory 36 %).  An earlier form with
// the columns brought in by cp.async, one thread a 16-byte row, took 507 (L1 tag lookups of the
// 64-byte pieces), and 588 before the reduced system's matrix stopped at decoupled rows.
#pragma once

#include <cuda.h>

#include "channel_base.cuh"

namespace cfd {

// couplings of the reduced system whose products cannot change a diagonal (2^-60)
constexpr double kDecoupled = 8.67e-19;
constexpr int kColTabs = 8;  // doubles per row of the coefficient table

// rows per lane for a column of n rows, 0 where the partition does not take it
__host__ __device__ constexpr int col_rows_per_lane(int n) {
    const int m = ((n + 31) / 32) | 1;
    return m <= 15 ? m : (m <= 19 ? 19 : (m <= 23 ? 23 : 0));
}
// columns of a group, by the distance of a column's rows: each row is a page of its own from
// about 2 MB on, and the transfers are bound by the pages they touch well before that (512 x
// 512: 743 us by fours, 620 by eights; 432 x 432: 399 and 452; 768 x 768: 2960 and 2040)
__host__ __device__ constexpr int col_cols(int m, int ncol) { return m <= 15 && (long long)ncol * 16 >= 768 * 1024 ? 8 : 4; }
// whether the next columns are brought into L2 ahead: groups of eight leave an SM with one or
// two groups, which wait for them (648 x 648: 1045 us without, 983 with); by fours it pays only
// on small planes (192 x 192: 93 and 88, 384 x 384: 323 and 347)
__host__ __device__ constexpr bool col_ahead(int cols, int ncol) { return cols == 8 || (long long)ncol * 16 <= 256 * 1024; }
// groups per CTA: bounded by the registers of a lane's rows (about 12 M) and by shared memory
__host__ __device__ constexpr int col_groups(int m, int cols) {
    return cols == 4 ? (m <= 7 ? 4 : (m <= 11 ? 3 : (m <= 15 ? 2 : 1))) : (m <= 7 ? 2 : 1);
}
__host__ __device__ constexpr int col_tab_elems(int m) { return 32 * m * kColTabs; }
// bytes of a field's rows of one group (16 a column, 32 M rows) and of the CTA's shared memory:
// the groups' u, w, v rows, the table, two barriers and four words a group
__host__ __device__ constexpr int col_region(int m, int cols) { return 32 * m * cols * 16; }
__host__ __device__ constexpr size_t col_smem(int m, int cols) {
    return (size_t)col_groups(m, cols) * 3 * col_region(m, cols) + (size_t)col_tab_elems(m) * 8 + 128;
}
// boxes a region arrives in: at most 256 rows each, a multiple of 8 (the swizzle's period)
__host__ __device__ constexpr int col_boxes(int m) { return 32 * m <= 256 ? 1 : (32 * m <= 512 ? 2 : 4); }

__device__ __forceinline__ double2 shfl_up2(double2 a, int d) {
    return dc(__shfl_up_sync(0xffffffffu, a.x, d), __shfl_up_sync(0xffffffffu, a.y, d));
}
__device__ __forceinline__ double2 shfl_down2(double2 a, int d) {
    return dc(__shfl_down_sync(0xffffffffu, a.x, d), __shfl_down_sync(0xffffffffu, a.y, d));
}
// a + s*b
__device__ __forceinline__ double2 dadds(double2 a, double s, double2 b) { return dc(a.x + s * b.x, a.y + s * b.y); }

// 1/x of a pivot (normal, far from overflow) by two Newton steps from the hardware's
// approximation: within an ulp, and without the branches of the full-range division
__device__ __forceinline__ double pivot_rcp(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

// Whether couplings al, ga of at most 2^-60 cannot change any lane's f to a double, by the exponents of
// the largest and the smallest of each component: then f + al f(s-d) + ga f(s+d) is f for every lane.
// (Lanes without couplings, past the column's end, do not count.)
template <int NR>
__device__ __forceinline__ bool carries_nothing(double al, double ga, const double2 (&f)[NR]) {
    auto ex = [](double a) { return ((unsigned)__double2hiint(a) & 0x7fffffffu) >> 20; };
    const double c = fmax(fabs(al), fabs(ga));
    const unsigned ec = __reduce_max_sync(0xffffffffu, ex(c));
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NR; ++k)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const double v = i ? f[k].y : f[k].x;
            const unsigned hi = __reduce_max_sync(0xffffffffu, ex(v));
            const unsigned lo = __reduce_min_sync(0xffffffffu, c == 0.0 ? 0x7ffu : ex(v));
            ok = ok && (hi == 0 || (int)(ec + hi) - 1023 + 60 < (int)lo);
        }
    return ok;
}

// One system over the warp's column: y[k][i] holds the NR real-matrix complex right-hand sides of
// the lane's rows and receives the solution.  coef(i, a, c, s): row i reads
// (a + c + s) x(i) - a x(i-1) - c x(i+1) = y(i).  Carrying the surplus s of the diagonal through
// the elimination, as the sums of products below, instead of the diagonal leaves nothing to
// cancel: D.G at small k has s nine digits below a + c, and the partition on diagonals lost
// three times what the sequential sweep loses there.  Row 0 of the column has a = 0, its last
// row c = 0, and the rows past it a = c = 0, s = 1 and a zero right-hand side, so the shuffles
// past either end multiply by 0.
template <int M, int NR, typename Coef>
__device__ __forceinline__ void warp_tridiag(double2 (&y)[NR][M], Coef coef) {
    // x(i) = y(i) + l X(s-1) + cs x(i+1), 1 - l - cs = e; first row = A + B X(s-1) + C X(s),
    // 1 - B - C = E
    double cs[M], l[M], e = 0.0;
    double2 A[NR];
    double B = 0.0, C = 1.0, E = 0.0, a, c, s;
#pragma unroll
    for (int k = 0; k < NR; ++k) A[k] = dc(0, 0);
#pragma unroll
    for (int i = 0; i < M - 1; ++i) {
        coef(i, a, c, s);
        const double p = i > 0 ? a * l[i > 0 ? i - 1 : 0] : a;
        const double z = i > 0 ? s + a * e : s;
        const double d = pivot_rcp(c + (z + p));
        l[i] = p * d;
        cs[i] = c * d;
        e = z * d;
        B += C * l[i];
        E += C * e;
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            y[k][i] = i > 0 ? dscl(d, dadds(y[k][i], a, y[k][i > 0 ? i - 1 : 0])) : dscl(d, y[k][i]);
            A[k] = dadds(A[k], C, y[k][i]);
        }
        C *= cs[i];
    }
    constexpr int L = M > 1 ? M - 2 : 0;
    coef(M - 1, a, c, s);
    // (a sum takes its couplings together first, here and below: they are the smaller part, so one
    // rounding of the full size is left instead of two)
    double2 f[NR];
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        const double2 n = dscl(c, shfl_down2(A[k], 1));
        f[k] = dadd(y[k][M - 1], M > 1 ? dadds(n, a, y[k][L]) : n);
    }
    double al = a;
    if (M > 1) {
        al = a * l[L];
        s += a * e;
    }
    double ga = c * __shfl_down_sync(0xffffffffu, C, 1);
    s += c * __shfl_down_sync(0xffffffffu, E, 1);
    // (al + ga + s) X(s) - al X(s-d) - ga X(s+d) = f.  The rows are not scaled on the way, so f is
    // rounded once a step, until the couplings are so small that their products cannot change the
    // diagonals (at once for the Helmholtz rows of a small time step: they fall by about beta/dy^2 a
    // row).  What they still carry from row to row counts where a right-hand side is zero or small:
    // the steps left take it along, on rows scaled to a diagonal of 1, unless no lane's f would change
    // (384 x 257(+90) x 384: 335 us a substep without that test, 323 with it).
    int d = 1;
#pragma unroll 1
    for (;; d <<= 1) {
        const double r = pivot_rcp(s + (al + ga));
        if (d == 32 || __all_sync(0xffffffffu, fmax(fabs(al), fabs(ga)) * r < kDecoupled)) {
            al *= r;
            ga *= r;
#pragma unroll
            for (int k = 0; k < NR; ++k) f[k] = dscl(r, f[k]);
            break;
        }
        const double alm = __shfl_up_sync(0xffffffffu, al, d), gap = __shfl_down_sync(0xffffffffu, ga, d);
        al *= __shfl_up_sync(0xffffffffu, r, d);
        ga *= __shfl_down_sync(0xffffffffu, r, d);
#pragma unroll
        for (int k = 0; k < NR; ++k) f[k] = dadd(f[k], dadds(dscl(al, shfl_up2(f[k], d)), ga, shfl_down2(f[k], d)));
        s += al * __shfl_up_sync(0xffffffffu, s, d) + ga * __shfl_down_sync(0xffffffffu, s, d);
        al *= alm;
        ga *= gap;
    }
    if (d < 32 && carries_nothing<NR>(al, ga, f)) d = 32;
#pragma unroll 1
    for (; d < 32; d <<= 1) {
#pragma unroll
        for (int k = 0; k < NR; ++k) f[k] = dadds(dadds(f[k], al, shfl_up2(f[k], d)), ga, shfl_down2(f[k], d));
        al *= __shfl_up_sync(0xffffffffu, al, d);
        ga *= __shfl_down_sync(0xffffffffu, ga, d);
    }
#pragma unroll
    for (int k = 0; k < NR; ++k) {
        const double2 X = shfl_up2(f[k], 1);
        y[k][M - 1] = f[k];
#pragma unroll
        for (int i = M - 2; i >= 0; --i) y[k][i] = dadd(y[k][i], dadds(dscl(cs[i], y[k][i + 1]), l[i], X));
    }
}

// ---- TMA and barriers
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, int n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// true when the phase has completed; gives up after `tries` tries (kWaitTries: about a second)
constexpr int kWaitTries = 1 << 20;
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, int tries) {
    for (int k = 0; k < tries; ++k) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2, 1000;\nselp.b32 %0, 1, 0, q;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// The wait of a group's threads.  Each may find the limit by itself, so none leaves here: one that
// gives up sets *gave, and the group reads that after its next barrier and leaves as one.  Waits
// that a barrier apart may still be read take words of their own.
__device__ __forceinline__ void group_wait(unsigned bar, unsigned parity, int tries, volatile int* gave) {
    if (!mbar_wait(bar, parity, tries)) *gave = 1;
}
__device__ __forceinline__ void tma_load(unsigned dst, const CUtensorMap* m, int x, int y, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                 "l"(m), "r"(x), "r"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap* m, int x, int y, unsigned src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(m), "r"(x), "r"(y),
                 "r"(src)
                 : "memory");
}
__device__ __forceinline__ void tma_prefetch(const CUtensorMap* m, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(m), "r"(x), "r"(y) : "memory");
}

// sources and destinations of u, w, v (or psi and the divergence) and p, as [plane][column]
// tensors of doubles
struct ColMaps {
    CUtensorMap src[3], dst[3], p;
};
struct ColArgs {
    const double* tab;  // tab[(i*kColTabs + k)*32 + lane]: coefficients of row lane*M + i
    double beta;        // b dt / Re
    double dtirk;       // 1 / (dt (a+b))
    double dtrk;        // dt (a+b)
    double mean_diag;   // bottom row of D.G at kx = kz = 0
    double* err;        // set if a transfer did not arrive
    int tries;          // limit of the waits for one (kWaitTries)
    bool ahead;         // prefetch the next columns into L2 while these are solved
};

// MB: a three-band channel.  A short column (a mode of the wall bands only) is two independent
// segments, u rows 0..bu and tu..nyu-1 with v and p rows to match; the rows between are identity
// rows with zero right-hand sides, and the segments' inner ends the band-interface rows.
//
// MODE bits: 1 = the Helmholtz solves of u, v, w; 2 = solveP on the velocities, p += psi; 4 =
// v_corr.  7 is the substep's, 1 and 2 are the stage entry points' (2 stores psi and the
// divergence).
template <int M, int C, int MODE, bool MB>
__global__ void __launch_bounds__(32 * C * col_groups(M, C))
    k_col_solve(Dims d, Geo g, const __grid_constant__ ColMaps maps, ColArgs A) {
    constexpr int G = col_groups(M, C), NB = col_boxes(M), BR = 32 * M / NB, RB = col_region(M, C), PB = 16 * C;
    constexpr bool UVW = (MODE & 1) != 0, PRE = (MODE & 2) != 0, COR = (MODE & 4) != 0;
    extern __shared__ __align__(1024) unsigned char col_smem_raw[];
    const int grp = threadIdx.x / (32 * C), t = threadIdx.x - grp * 32 * C;
    const int lane = t & 31, wc = t >> 5;
    unsigned char* reg = col_smem_raw + grp * 3 * RB;  // the group's u, w, v rows
    double* stab = reinterpret_cast<double*>(col_smem_raw + G * 3 * RB);
    const unsigned sreg = smem_u32(reg);
    const unsigned bar = smem_u32(stab + col_tab_elems(M)) + 16 * grp, barp = bar + 8;
    // a wait that was given up: [phase] the columns', [2 + phase] p's
    volatile int* gave = reinterpret_cast<int*>(stab + col_tab_elems(M) + 8) + 4 * grp;
    const bool lead = t == 0;
    const int nq = (d.ncol + C - 1) / C, stride = G * gridDim.x;
    int q = blockIdx.x + grp * gridDim.x;
    if (lead) {
        mbar_init(bar, 1);
        mbar_init(barp, 1);
        for (int k = 0; k < 4; ++k) gave[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < col_tab_elems(M); i += blockDim.x) stab[i] = A.tab[i];
    __syncthreads();
    auto load = [&](int f, const CUtensorMap* m, int qq, unsigned b) {
#pragma unroll
        for (int k = 0; k < NB; ++k) tma_load(sreg + f * RB + k * BR * PB, m, 2 * C * qq, k * BR, b);
    };
    auto store = [&](int f, const CUtensorMap* m, int qq) {
#pragma unroll
        for (int k = 0; k < NB; ++k) tma_store(m, 2 * C * qq, k * BR, sreg + f * RB + k * BR * PB);
    };
    auto prefetch = [&](const CUtensorMap* m, int qq) {
#pragma unroll
        for (int k = 0; k < NB; ++k) tma_prefetch(m, 2 * C * qq, k * BR);
    };
    auto read_out = [] {  // the stores issued so far have read shared memory
        asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group.read 0;" ::: "memory");
    };
    auto publish = [] { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); };
    auto group_sync = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(grp + 1), "n"(32 * C) : "memory"); };
    if (lead && q < nq) {
        mbar_expect(bar, 3 * RB);
#pragma unroll
        for (int f = 0; f < 3; ++f) load(f, &maps.src[f], q, bar);
    }
    const double* tb = stab + lane;
    auto T = [&](int i, int k) { return tb[(i * kColTabs + k) * 32]; };
    // row row0 + i of the warp's column: PB i bytes past the address of its residue mod 8
    const int row0 = lane * M;
    auto swz = [&](int r) { return (wc ^ (C == 4 ? (r >> 1) & 3 : r & 7)) << 4; };
    unsigned char* at[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) at[k] = reg + row0 * PB + swz(row0 + k);
    auto R = [&](int f, int i) -> double2& { return *reinterpret_cast<double2*>(at[i & 7] + f * RB + i * PB); };
    auto row = [&](int f, int r) -> double2& { return *reinterpret_cast<double2*>(reg + f * RB + r * PB + swz(r)); };
    const bool top = lane == 31;  // its row M would be the region's end: never part of a column

    const int bu = d.jb + 2 - d.ju0, tu = d.ny - 2 - d.jb - d.ju0;
    unsigned phase = 0;
    bool ok = true;
    for (; q < nq; q += stride, phase ^= 1) {
        const int col = min(q * C + wc, d.ncol - 1);
        const double kxv = g.kx[col % d.nkx], kzv = g.kz[col / d.nkx];
        const double k2 = -kxv * kxv - kzv * kzv;
        const bool sh = MB && !mb_long(d, col % d.nkx, col / d.nkx);  // a short column
        // the weight of the face above p row r (0 at the ends of the column or segment)
        auto face = [&](int i, int r) { return MB && sh && r >= bu - 2 && r < tu ? 0.0 : T(i, 7); };
        group_wait(bar, phase, A.tries, gave + phase);
        if (lead) {
            if (PRE) prefetch(&maps.p, q);
            if (A.ahead && q + stride < nq)
#pragma unroll
                for (int f = 0; f < 3; ++f) prefetch(&maps.src[f], q + stride);
        }
        double2 ps[1][PRE ? M : 1];
        if (UVW) {
            {   // v: identity wall rows
                const int n = d.nyv;
                double2 y[1][M];
#pragma unroll
                for (int i = 0; i < M; ++i) y[0][i] = R(2, i);
                warp_tridiag<M, 1>(y, [&](int i, double& a, double& c, double& s) {
                    const int r = row0 + i;
                    a = A.beta * T(i, 3);
                    c = A.beta * T(i, 5);
                    s = 1.0 - A.beta * (T(i, 4) + (r > 0 && r < n - 1 ? k2 : 0.0));
                    if (MB && sh && r >= bu - 1 && r <= tu) { a = c = 0.0; s = 1.0; }
                });
#pragma unroll
                for (int i = 0; i < M; ++i) R(2, i) = y[0][i];
            }
            // u and w share the matrix: rows (0,1,gwb), interior, (gwt,1,0)
            const int n = d.nyu;
            auto coef = [&](int i, double& a, double& c, double& s) {
                const int r = row0 + i;
                a = r == n - 1 ? -g.gwt : A.beta * T(i, 0);
                c = r == 0 ? -g.gwb : A.beta * T(i, 2);
                s = r > 0 && r < n - 1 ? 1.0 - A.beta * (T(i, 1) + k2) : 1.0 - (a + c);
                if (MB && sh && r >= bu && r <= tu) {
                    a = r == bu ? -g.gw1t : 0.0;
                    c = r == tu ? -g.gw3b : 0.0;
                    s = 1.0 - (a + c);
                }
            };
            if constexpr (M <= 15) {
                double2 y[2][M];
#pragma unroll
                for (int i = 0; i < M; ++i) { y[0][i] = R(0, i); y[1][i] = R(1, i); }
                warp_tridiag<M, 2>(y, coef);
#pragma unroll
                for (int i = 0; i < M; ++i) { R(0, i) = y[0][i]; R(1, i) = y[1][i]; }
                if constexpr (PRE) {  // the divergence's share of u and w at centre row0 + i + 1
#pragma unroll
                    for (int i = 0; i < M; ++i) ps[0][i] = dadd(dik(kxv, y[0][i]), dik(kzv, y[1][i]));
                    const double2 up = shfl_down2(ps[0][0], 1);
#pragma unroll
                    for (int i = 0; i < M - 1; ++i) ps[0][i] = ps[0][i + 1];
                    ps[0][M - 1] = up;
                }
            } else {  // one at a time: both do not fit the registers
#pragma unroll 1
                for (int f = 0; f < 2; ++f) {
                    double2 y[1][M];
#pragma unroll
                    for (int i = 0; i < M; ++i) y[0][i] = R(f, i);
                    warp_tridiag<M, 1>(y, coef);
#pragma unroll
                    for (int i = 0; i < M; ++i) R(f, i) = y[0][i];
                }
            }
            __syncwarp();
        }
        if constexpr (PRE) {
            // row r of the pressure is the centre of velocity row r + 1, between faces r and r + 1
            const int n = d.nyp;
            const bool mean = col == 0;
            double2 dv[MODE == 2 ? M : 1];
            double2 vb = R(2, 0);
#pragma unroll
            for (int i = 0; i < M; ++i) {
                const int r = row0 + i;
                const bool in = i < M - 1 || !top;
                const double2 va = in ? R(2, i + 1) : vb;
                if (!(UVW && M <= 15)) ps[0][i] = in ? dadd(dik(kxv, R(0, i + 1)), dik(kzv, R(1, i + 1))) : dc(0, 0);
                double2 v = dadd(ps[0][i], dscl(T(i, 6), dsub(va, vb)));
                if (MB && sh && r > bu - 2 && r < tu) v = dc(0, 0);
                vb = va;
                if (MODE == 2) dv[i] = v;
                ps[0][i] = (r < n && !(mean && r == 0)) ? dscl(-A.dtirk, v) : dc(0, 0);
            }
            // D.G: the off-diagonals are dthdyu of the centre times dthdyv of the faces (0 at walls)
            const double dlow = __shfl_up_sync(0xffffffffu, face(M - 1, row0 + M - 1), 1);
            warp_tridiag<M, 1>(ps, [&](int i, double& a, double& c, double& s) {
                const int r = row0 + i;
                const double dt = T(i, 6);
                a = dt * (i > 0 ? face(i > 0 ? i - 1 : 0, r - 1) : (lane ? dlow : 0.0));
                c = dt * face(i, r);
                s = r < n && !(MB && sh && r > bu - 2 && r < tu) ? -k2 : 1.0;
                if (mean && r == 0) { s = A.mean_diag; c = 0.0; }
            });
            __syncwarp();
            if constexpr (MODE == 2) {
#pragma unroll
                for (int i = 0; i < M; ++i) { R(0, i) = ps[0][i]; R(1, i) = dv[i]; }
            }
        }
        if constexpr (COR) {
            // u, w of centre r take i k psi(r), the face above takes psi(r+1) - psi(r)
            const double2 pn = shfl_down2(ps[0][0], 1);  // past the top the face weight is 0
            double2 x[M];
#pragma unroll
            for (int f = 0; f < 3; ++f) {
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    if (i == M - 1 && top) break;
                    x[i] = R(f, i + 1);
                }
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    if (i == M - 1 && top) break;
                    if (f < 2) R(f, i + 1) = dsub(x[i], dik(A.dtrk * (f ? kzv : kxv), ps[0][i]));
                    else R(f, i + 1) = dsub(x[i], dscl(A.dtrk * face(i, row0 + i), dsub(i < M - 1 ? ps[0][i < M - 1 ? i + 1 : 0] : pn, ps[0][i])));
                }
            }
            __syncwarp();
            if (lane < 2) {  // ghost and wall rows
                const int e = lane ? d.nyu - 1 : 0, in = lane ? d.nyu - 2 : 1;
                const double gw = lane ? -g.gwt : -g.gwb;
                row(0, e) = dscl(gw, row(0, in));
                row(1, e) = dscl(gw, row(1, in));
                row(2, lane ? d.nyv - 1 : 0) = dc(0, 0);
            }
        }
        publish();
        group_sync();
        if (gave[phase]) {  // nothing is stored; the copies still under way end before the CTA does
            if (lead) mbar_wait(bar, phase, kWaitTries);
            ok = false;
            break;
        }
        if (lead) {
#pragma unroll
            for (int f = 0; f < (MODE == 2 ? 2 : 3); ++f) store(f, &maps.dst[f], q);
            read_out();
            if (PRE) {  // p takes the place of u
                mbar_expect(barp, RB);
                load(0, &maps.p, q, barp);
            }
            if (q + stride < nq) {
                mbar_expect(bar, 3 * RB);
                if (!PRE) load(0, &maps.src[0], q + stride, bar);
                load(1, &maps.src[1], q + stride, bar);
                load(2, &maps.src[2], q + stride, bar);
            }
        }
        if constexpr (PRE) {
            group_wait(barp, phase, A.tries, gave + 2 + phase);
#pragma unroll
            for (int i = 0; i < M; ++i) R(0, i) = dadd(R(0, i), ps[0][i]);
            publish();
            group_sync();
            if (gave[2 + phase]) {
                if (lead) {
                    mbar_wait(barp, phase, kWaitTries);
                    if (q + stride < nq) {  // (u completes the next columns' bytes)
                        load(0, &maps.src[0], q + stride, bar);
                        mbar_wait(bar, phase ^ 1, kWaitTries);
                    }
                }
                ok = false;
                break;
            }
            if (lead) {
                store(0, &maps.p, q);
                read_out();
                if (q + stride < nq) load(0, &maps.src[0], q + stride, bar);
            }
        }
    }
    if (!ok && lead) *A.err = 1.0;
    if (lead) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Mean mode at constant flow rate: flowrate_corr with LUsol0/LU_build0/LU_dec0
// (littleharsh.f90:452-484, tridLU_3D_IB.f90:320-346, 493-519, 605-622), the unit response of the
// cells between the crests and one each side (j = 0..ny) solved by the warp's partition.  One lane
// walking the column through memory took 42 us at 194 rows, the warp takes 7.5.  scal[0] = mpgx,
// scal[2] = dgx.  ghosts: extrapolate the column's ghost rows as v_corr does.
template <int M>
__global__ void __launch_bounds__(32) k_meanflow_warp(Dims d, Geo g, double beta, double bdt, double qxt,
                                                      double2* __restrict__ u1, double* __restrict__ scal, bool ghosts) {
    const int lane = threadIdx.x, n = d.ny + 1, row0 = lane * M;
    double2 x[1][M];
    double q0 = 0.0, q1 = 0.0;
    // cell width between the faces below and above centre j, for the cells between the crests
    auto width = [&](int j) { return j >= 1 && j <= n - 2 ? g.yv[j - d.jv0] - g.yv[j - 1 - d.jv0] : 0.0; };
#pragma unroll
    for (int i = 0; i < M; ++i) {
        const int j = row0 + i;
        x[0][i] = dc(j >= 1 && j <= n - 2 ? bdt : 0.0, 0.0);
        if (j >= 1 && j <= n - 2) q0 += width(j) * u1[(size_t)(j - d.ju0) * d.ncol].x;
    }
    warp_tridiag<M, 1>(x, [&](int i, double& a, double& c, double& s) {
        const int j = row0 + i;
        a = c = 0.0;
        s = 1.0;
        if (j >= 1 && j <= n - 2) {
            const double* w = g.dyu2i + 3 * (j - d.ju0);
            a = beta * w[0];
            c = beta * w[2];
            s = 1.0 - beta * ((w[0] + w[2]) + w[1]);
        } else if (j == 0) {
            c = -g.gwb;
            s = 1.0 - c;
        } else if (j == n - 1) {
            a = -g.gwt;
            s = 1.0 - a;
        }
    });
#pragma unroll
    for (int i = 0; i < M; ++i) q1 += width(row0 + i) * x[0][i].x;
    for (int o = 16; o > 0; o >>= 1) {
        q0 += __shfl_xor_sync(0xffffffffu, q0, o);
        q1 += __shfl_xor_sync(0xffffffffu, q1, o);
    }
    const double gg = (qxt - q0) / q1;
    if (lane == 0) {
        scal[0] += gg;
        scal[2] = gg;
    }
#pragma unroll
    for (int i = 0; i < M; ++i)
        if (row0 + i < n) u1[(size_t)(row0 + i - d.ju0) * d.ncol].x += gg * x[0][i].x;
    if (ghosts) {
        __syncwarp();
        if (lane == 0) {
            u1[0] = dscl(-g.gwb, u1[d.ncol]);
            u1[(size_t)(d.nyu - 1) * d.ncol] = dscl(-g.gwt, u1[(size_t)(d.nyu - 2) * d.ncol]);
        }
    }
}

// Host side (colsolve.cu; the _mb forms in colsolve_mb.cu): m rows per lane, cols columns a group
// (4 in three bands), mb three bands
cudaError_t col_prepare(int m, int cols, bool mb);  // raises the shared-memory limit of the kernels
cudaError_t col_prepare_mb(int m);
// tensor map of a field of n planes; false if it cannot be made
bool col_map(CUtensorMap* map, const void* field, int ncol, int n, int m, int cols);
void col_launch(int mode, int m, int cols, bool mb, int nsm, cudaStream_t st, const Dims& d, const Geo& g,
                const ColMaps& maps, const ColArgs& a);
// k_meanflow_warp with m rows per lane, m = col_rows_per_lane(ny + 1)
void col_meanflow(int m, cudaStream_t st, const Dims& d, const Geo& g, double beta, double bdt, double qxt, double2* u1,
                  double* scal, bool ghosts);
void col_launch_mb(int mode, int m, int nsm, cudaStream_t st, const Dims& d, const Geo& g, const ColMaps& maps,
                   const ColArgs& a);

}  // namespace cfd
