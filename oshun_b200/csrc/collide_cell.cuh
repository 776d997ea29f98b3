// Pieces of the CTA-per-cell collision kernels (collide.cu, adjoint.cu): one
// thread per momentum point (in collide.cu two from 129 points on) for the pointwise work
// and the cumulative integrals, groups of G lanes holding runs of R points for
// the tridiagonal solves.  Sums of products that end in a state are written with
// explicit roundings (rounding.cuh): the instances of few and of many cells and
// of a batch give the same bits.
#pragma once

#include <type_traits>

#include "oshun_internal.h"
#include "rounding.cuh"

namespace oshun {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// The forms: K = G R / 8 (the row's points, rounded up to the form's, over 8).
// One thread a point up to 128 points, two beyond (half the warps' scans and
// barriers: e-e substeps of 20000 cells of 184 / 200 points 354 / 444 -> 208 / 260
// us, 1433 cells of 201 points, 15 substeps, f1 and f_lm with them, 575 -> 331,
// where a warp a cell took 447; few cells, whose logarithms take a warp without
// points, 100 of 224 points 114 -> 96).  113 to 128 points take runs
// of 4 on 32 lanes: with 8 on 16 lanes two planes share a warp, but a row's
// pieces lie 64 bytes apart (20000 cells, l0 = 1, the f1 call 150 -> 101 us;
// 5000 cells, 15 planes, their call 143 -> 93; 64 cells of 48 planes 29 -> 33).
constexpr int form_lanes(int K) { return K <= 8 ? 8 : (K < 16 ? 16 : 32); }
constexpr int form_run(int K) { return 8 * K / form_lanes(K); }
constexpr int form_points(int K) { return K <= 16 ? 1 : 2; }
constexpr int form_warps(int K) { return (8 * K + 32 * form_points(K) - 1) / (32 * form_points(K)); }
// warps of one thread a point
constexpr int point_warps(int K) { return (8 * K + 31) / 32; }
// Warps of a cell's CTA: of 129 to 256 points, and unless launches of many cells
// (`many`), twice as many as the pointwise work takes, for the solves
constexpr int cell_warps(int K, bool many) { return !many && form_points(K) > 1 && K <= 32 ? point_warps(K) : form_warps(K); }
// Resident CTAs per SM up to 256 points, of 128 registers a thread; up to 128
// points more of 80 registers for launches of many cells (`many`) and for
// batches, where a lane's run is shorter than 8 points: more warps hide the FP64
// latency.  On few cells the spills cost more (256 cells of 96 points, ten e-e
// substeps: 118 us against 135).  With few planes (kManyPlanes) the many form is
// the faster one: 8000 cells of 96 points, 1D, 2 / 8 / 24 planes 138 / 187 / 307
// -> 123 / 166 / 293 us.  With several planes of one l (m0 >= 2) it depends on how
// far a row length's form spills: 15 planes, 5000 cells, 40 / 72 / 96 / 112 / 128
// points x 1.02 / 0.93 / 1.04 / 1.08 / 0.93; 48 planes x 1.07 / 0.98 / 1.11 / 1.16
// / 0.92.  From 129 points on the many form has half the warps and its CTAs hold
// more cells, whatever the planes (48 planes, 5000 cells of 136 / 192 / 256 points
// 318 / 382 / 542 -> 296 / 298 / 512 us).
constexpr int kManyPlanes = 32;
constexpr int form_blocks(int K, bool many) {
    return K > 32 ? 1 : (many && form_points(K) == 1 && form_run(K) < 8 ? 24 : 16) / cell_warps(K, many);
}
// the e-e substeps alone, one thread a point: 96 registers a thread (no spills),
// 20000 cells of 64 / 128 points 124 / 226 -> 114 / 198 us against 80 registers
constexpr int ee_blocks(int K) { return (form_points(K) > 1 ? 16 : 20) / form_warps(K); }
// the solves on a warp a cell
constexpr int solve_blocks(int K) { return K <= 32 ? 16 : 8; }
template <typename F>
cudaError_t with_form(int K, F&& go) {
    switch (K) {
        case 4: return go(std::integral_constant<int, 4>{});
        case 6: return go(std::integral_constant<int, 6>{});
        case 8: return go(std::integral_constant<int, 8>{});
        case 10: return go(std::integral_constant<int, 10>{});
        case 12: return go(std::integral_constant<int, 12>{});
        case 14: return go(std::integral_constant<int, 14>{});
        case 16: return go(std::integral_constant<int, 16>{});
        case 20: return go(std::integral_constant<int, 20>{});
        case 24: return go(std::integral_constant<int, 24>{});
        case 28: return go(std::integral_constant<int, 28>{});
        case 32: return go(std::integral_constant<int, 32>{});
        case 40: return go(std::integral_constant<int, 40>{});
        case 48: return go(std::integral_constant<int, 48>{});
        case 56: return go(std::integral_constant<int, 56>{});
        case 64: return go(std::integral_constant<int, 64>{});
        default: return cudaErrorInvalidValue;
    }
}
// Thomas pivots of harmonic order l for this lane's run of p, c'_i and
// 1/(b_i - c'_{i-1} a_i), with b_i = tri_b_i + 1 - ll1 scat_i (tri_b_0 left
// out for l > 1), as TridiagonalSolve forms them (def-Nmethods.cpp:152-159).
// c'_i = c_i / (b_i - a_i c'_{i-1}) is a linear-fractional map of c'_{i-1},
// the 2x2 matrix [[0, c_i], [-a_i, b_i]] acting on (c'_{i-1}, 1): each lane
// composes its run's matrices, a scan over the group (rescaled by powers of
// two, which leaves the maps unchanged) gives the value entering
// the run, and the lane applies the recursion inside its run.
struct M22 {
    double a, b, c, d;
};
__device__ __forceinline__ M22 m22_mul(const M22& x, const M22& y) {
    return M22{fma(x.a, y.a, x.b * y.c), fma(x.a, y.b, x.b * y.d), fma(x.c, y.a, x.d * y.c),
               fma(x.c, y.b, x.d * y.d)};
}
__device__ __forceinline__ M22 m22_rescale(M22 x) {
    const double mx = fmax(fmax(fabs(x.a), fabs(x.b)), fmax(fabs(x.c), fabs(x.d)));
    const int ex = (int)((__double_as_longlong(mx) >> 52) & 0x7ff);
    if (mx > 0.0 && ex > 0 && ex < 0x7ff) {
        const double sc = __longlong_as_double((long long)(2046 - ex) << 52);   // 2^(1023 - ex)
        x.a *= sc; x.b *= sc; x.c *= sc; x.d *= sc;
    }
    return x;
}
// the coefficients of one cell in shared memory (np each)
struct TriRows {
    double *a, *b, *c, *scat;
};
template <int G, int R>
__device__ __forceinline__ void lane_pivots(const TriRows& s, const int l, const int n, const int i0, double (&cp)[R],
                                            double (&id)[R]) {
    const int gl = threadIdx.x & (G - 1);
    const double ll1 = l * ((-0.5) * (l + 1.0));
    M22 m{1.0, 0.0, 0.0, 1.0};
#pragma unroll
    for (int e = 0; e < R; ++e) {
        const int i = i0 + e;
        id[e] = 1.0;   // b_i until the recursion below
        if (i < n) {
            const double a = s.a[i], c = s.c[i];
            const double b = add_rn(i == 0 && l > 1 ? 0.0 : s.b[i], fma_rn(-ll1, s.scat[i], 1.0));
            id[e] = b;
            m = M22{c * m.c, c * m.d, fma(-a, m.a, b * m.c), fma(-a, m.b, b * m.d)};
        }
        if (e % 8 == 7) m = m22_rescale(m);
    }
    m = m22_rescale(m);
#pragma unroll
    for (int off = 1; off < G; off <<= 1) {
        const M22 o{__shfl_up_sync(kFull, m.a, off, G), __shfl_up_sync(kFull, m.b, off, G),
                    __shfl_up_sync(kFull, m.c, off, G), __shfl_up_sync(kFull, m.d, off, G)};
        if (gl >= off) m = m22_rescale(m22_mul(m, o));
    }
    const double xb = __shfl_up_sync(kFull, m.b, 1, G), xd = __shfl_up_sync(kFull, m.d, 1, G);
    double cprev = gl == 0 ? 0.0 : xb / xd;
#pragma unroll
    for (int e = 0; e < R; ++e) {
        const int i = i0 + e;
        if (i < n) {
            const double b = id[e];
            if (i == 0) {
                id[e] = 1.0 / b;
                cprev = s.c[0] / b;
            } else {
                id[e] = 1.0 / fma_rn(-cprev, s.a[i], b);
                cprev = s.c[i] * id[e];
            }
            cp[e] = cprev;
        } else {
            id[e] = 0.0;
            cp[e] = 0.0;
        }
    }
}

// velocity tables of a thread's PT momentum points k0 .. k0+PT-1
template <int PT>
struct PointTab {
    double U4[PT], U4m[PT], U2[PT], U2m[PT], U1p[PT], U1mp[PT];   // I4, I2 terms of k; the J1 term of k + 1
    double U3[PT], Qn[PT], Pn[PT], Pm[PT];                        // Pm: Pn of k - 1
    // the parabolic fit of the first NB points: i2 = f00 A2 + (f1 - f00) B2, i4 likewise
    double A2[PT], B2[PT], A4[PT], B4[PT];
    double r, inv1r, two_v0s;   // v0^2/v1^2, 1/(1 - r), 2/v0^2
};
// A: CollideArgs or adj::CollTables
template <int PT, class A>
__device__ __forceinline__ void load_tab(const A& a, const int k0, PointTab<PT>& t) {
    const int n = a.np;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        const int k = k0 + j;
        const bool in = k < n, up = k + 1 < n;
        const int kc = in ? k : 0;
        t.U4[j] = in ? __ldg(a.U4 + kc) : 0.0;     // 0 at k = 0 (the tables start at 1)
        t.U4m[j] = in ? __ldg(a.U4m1 + kc) : 0.0;
        t.U2[j] = in ? __ldg(a.U2 + kc) : 0.0;
        t.U2m[j] = in ? __ldg(a.U2m1 + kc) : 0.0;
        t.U1p[j] = up ? __ldg(a.U1 + kc + 1) : 0.0;
        t.U1mp[j] = up ? __ldg(a.U1m1 + kc + 1) : 0.0;
        t.U3[j] = in ? __ldg(a.U3 + kc) : 1.0;
        t.Qn[j] = in ? __ldg(a.Qn + kc) : 0.0;
        t.Pn[j] = up ? __ldg(a.Pn + kc) : 0.0;
        t.Pm[j] = in && k > 0 ? __ldg(a.Pn + kc - 1) : 0.0;
    }
    // the divisions of every slope, once a cell
    const double v0 = __ldg(a.vr), v1 = __ldg(a.vr + 1);
    const double v0s = v0 * v0, v1s = v1 * v1;
    t.r = v0s / v1s;
    t.inv1r = 1.0 / (1.0 - t.r);
    t.two_v0s = 2.0 / v0s;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        const int k = k0 + j;
        t.A2[j] = t.B2[j] = t.A4[j] = t.B4[j] = 0.0;
        if (k < a.NB && k < n) {
            const double v5 = __ldg(a.V5 + k);
            t.A2[j] = t.U3[j] / 3.0;
            t.B2[j] = v5 / v1s * 0.2;
            t.A4[j] = v5 * 0.2;
            t.B4[j] = __ldg(a.V7 + k) / (v1s * 7.0);
        }
    }
}
// shared memory of one cell's CTA (doubles): tri_a, tri_b, tri_c, scat [np],
// f and G with a point of padding on both sides, the warps' totals [3][16],
// three values that one warp computes for all
__host__ __device__ inline size_t cell_smem_doubles(int np, int pts) { return 4 * (size_t)np + 2 * ((size_t)pts + 2) + 51; }
struct CellSmem {
    TriRows tri;
    double *f, *g, *tot;   // f, g: index -1 .. pts
    double* one;
};
__device__ __forceinline__ CellSmem carve_cell(double* base, int np, int pts) {
    CellSmem s;
    s.tri.a = base; s.tri.b = base + np; s.tri.c = base + 2 * np; s.tri.scat = base + 3 * np;
    s.f = base + 4 * np + 1;
    s.g = s.f + pts + 2;
    s.tot = s.g + pts + 1;
    s.one = s.tot + 48;
    return s;
}

// joins the first W warps of the CTA, which do the pointwise work
template <int W, int BAR = 1>
__device__ __forceinline__ void warps_sync() {
    asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(32 * W) : "memory");
}
// The cumulative integrals I4, I2 (k' <= k) and J1 (k' > k) of f at a thread's
// points, and the whole I4, I2 (S4, S2).  fm, fp: the neighbours.
// X: one warp more waits for the totals
template <int PT, int W, int X = 0>
__device__ __forceinline__ void cell_scans(const PointTab<PT>& t, const double (&f)[PT], const double (&fm)[PT],
                                           const double (&fp)[PT], double* tot, double (&I4)[PT], double (&I2)[PT],
                                           double (&J1)[PT], double& S4, double& S2) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s4 = 0.0, s2 = 0.0, s1 = 0.0;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        I4[j] = fma(t.U4[j], f[j], t.U4m[j] * fm[j]);
        I2[j] = fma(t.U2[j], f[j], t.U2m[j] * fm[j]);
        J1[j] = fma(t.U1p[j], fp[j], t.U1mp[j] * f[j]);
        s4 += I4[j]; s2 += I2[j]; s1 += J1[j];
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double v4 = __shfl_up_sync(kFull, s4, off);
        const double v2 = __shfl_up_sync(kFull, s2, off);
        const double v1 = __shfl_down_sync(kFull, s1, off);
        if (lane >= off) { s4 += v4; s2 += v2; }
        if (lane + off < 32) s1 += v1;
    }
    if (lane == 31) { tot[warp] = s4; tot[16 + warp] = s2; }
    if (lane == 0) tot[32 + warp] = s1;
    double r4 = __shfl_up_sync(kFull, s4, 1), r2 = __shfl_up_sync(kFull, s2, 1);
    double r1 = __shfl_down_sync(kFull, s1, 1);
    if (lane == 0) { r4 = 0.0; r2 = 0.0; }
    if (lane == 31) r1 = 0.0;
    if constexpr (X > 0) warps_sync<W + X, 2>();
    else warps_sync<W>();
    double b4 = 0.0, b2 = 0.0, b1 = 0.0;
    S4 = 0.0; S2 = 0.0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        if (w == warp) { b4 = S4; b2 = S2; }
        S4 += tot[w]; S2 += tot[16 + w];
        if (w > warp) b1 += tot[32 + w];
    }
    r4 += b4; r2 += b2; r1 += b1;
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        r4 += I4[j]; I4[j] = r4;
        r2 += I2[j]; I2[j] = r2;
    }
#pragma unroll
    for (int j = PT - 1; j >= 0; --j) {
        r1 += J1[j];
        J1[j] = r1;
    }
}
// a thread's points to shared memory, then its neighbours back
// (X: one warp more joins)
template <int PT, int W, int X = 0>
__device__ __forceinline__ void neighbours(double* buf, const int k0, const double (&v)[PT], double (&lo)[PT],
                                           double (&hi)[PT]) {
#pragma unroll
    for (int j = 0; j < PT; ++j) buf[k0 + j] = v[j];
    if constexpr (X > 0) warps_sync<W + X, 3>();
    else warps_sync<W>();
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        lo[j] = j > 0 ? v[j > 0 ? j - 1 : 0] : buf[k0 - 1];
        hi[j] = j + 1 < PT ? v[j + 1 < PT ? j + 1 : 0] : buf[k0 + PT];
    }
}

}  // namespace
}  // namespace oshun
