// The collision step's transpose (adjoint_math.h collide_cell_T) on one CTA per
// cell: one thread per momentum point, its velocity tables, the e-e stages and
// their cumulative integrals in registers; the cumulative integrals' transposes
// are scans of the same kind (suffix for prefix), joined with the block sums
// of the scalar cotangents, two barriers a transposed slope.  The solves of A
// and A^T run on the lane groups of the forward solve: with the pivots id and
// c' of A = L U, A^T y = r is z_i = r_i - c'_{i-1} z_{i-1} forward and
// y_i = (z_i - a_{i+1} y_{i+1}) id_i backward, affine maps again.  The
// arithmetic is the serial form's up to the order of the sums.
//
// The serial chain of a cell bounds it (five e-e substeps: 20 slopes forward,
// 20 again with their integrals kept, 20 transposed): one warp a cell with
// Thomas on one lane and every array in shared memory took 0.60 ms for 512
// cells of 128 points, l0 = 2 (a 20-step gradient of that run 20.2 -> 13.1 ms with this form).
#pragma once

#include "adjoint_math.h"
#include "collide_cell.cuh"

namespace oshun {
namespace adjc {

using adj::CollTables;

// one collision step: the planes of each l >= 1 with m <= min(l, mmax) share its matrix
struct StepT {
    int l0, m0, mmax, unit_planes;
    int ee, eb, nsub;
    double hsub, Dt;
    const int* plane_of;   // [(l0+1)(m0+1)]: plane of Re f_lm (Im follows)
    long long pstride;
};
constexpr int kTot = 7;   // block totals joined at once
// shared memory of a cell (doubles): a, b, c, scat and their cotangents [np],
// two point rows with padding, the warps' totals
__host__ __device__ inline size_t cell_doubles(int np, int pts) { return 8 * (size_t)np + 2 * ((size_t)pts + 2) + kTot * 8; }
struct Mem {
    TriRows tri;
    double *la, *lb, *lc, *ls;
    double *f, *g, *tot;   // f, g: index -1 .. pts
};
__device__ __forceinline__ Mem carve(double* base, int np, int pts) {
    Mem s;
    s.tri.a = base; s.tri.b = base + np; s.tri.c = base + 2 * np; s.tri.scat = base + 3 * np;
    s.la = base + 4 * np; s.lb = base + 5 * np; s.lc = base + 6 * np; s.ls = base + 7 * np;
    s.f = base + 8 * np + 1;
    s.g = s.f + pts + 2;
    s.tot = s.g + pts + 1;
    return s;
}

// a point's tables: the forward ones and those its terms of k + 1 and k take in the transpose
struct Tab {
    PointTab<1> t;
    double U4mp, U2mp, U1;   // U4m1, U2m1 of k + 1; U1 of k
};
__device__ __forceinline__ void load(const CollTables& T, const int k, Tab& t) {
    load_tab<1>(T, k, t.t);
    const bool in = k < T.np, up = k + 1 < T.np;
    t.U4mp = up ? __ldg(T.U4m1 + k + 1) : 0.0;
    t.U2mp = up ? __ldg(T.U2m1 + k + 1) : 0.0;
    t.U1 = in ? __ldg(T.U1 + k) : 0.0;
}

// joins NS block sums with the block's exclusive scans of three values: r4, r2
// over the points above, r1 over the points below
template <int NS>
__device__ __forceinline__ void suffix_scans(double* tot, const double v4, const double v2, const double v1, double& r4,
                                             double& r2, double& r1, double (&sum)[NS]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double s4 = v4, s2 = v2, s1 = v1;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double u4 = __shfl_down_sync(kFull, s4, off), u2 = __shfl_down_sync(kFull, s2, off);
        const double u1 = __shfl_up_sync(kFull, s1, off);
        if (lane + off < 32) { s4 += u4; s2 += u2; }
        if (lane >= off) s1 += u1;
    }
#pragma unroll
    for (int i = 0; i < NS; ++i)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum[i] += __shfl_xor_sync(kFull, sum[i], off);
    if (lane == 0) {
        tot[warp] = s4; tot[8 + warp] = s2;
#pragma unroll
        for (int i = 0; i < NS; ++i) tot[24 + 8 * i + warp] = sum[i];
    }
    if (lane == 31) tot[16 + warp] = s1;
    r4 = __shfl_down_sync(kFull, s4, 1); r2 = __shfl_down_sync(kFull, s2, 1);
    r1 = __shfl_up_sync(kFull, s1, 1);
    if (lane == 31) { r4 = 0.0; r2 = 0.0; }
    if (lane == 0) r1 = 0.0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NS; ++i) sum[i] = 0.0;
    for (int w = 0; w < nw; ++w) {
        if (w > warp) { r4 += tot[w]; r2 += tot[8 + w]; }
        if (w < warp) r1 += tot[16 + w];
#pragma unroll
        for (int i = 0; i < NS; ++i) sum[i] += tot[24 + 8 * i + w];
    }
}
// the transposed cumulative integrals at this point (adj::scans_T): l4, l2, l1
// its cotangents, r4, r2, r1 the exclusive scans (X4, X2: the share of the
// last point's cotangents that every point sees)
__device__ __forceinline__ double scans_T(const Tab& t, const int k, const int n, const double l4, const double l2,
                                          const double l1, const double r4, const double r2, const double r1,
                                          const double X4, const double X2) {
    double a = 0.0;
    if (k < n) {
        if (k >= 1) a += (r4 + l4 + X4) * t.t.U4[0] + (r2 + l2 + X2) * t.t.U2[0] + r1 * t.U1;
        if (k + 1 < n) a += (r4 + X4) * t.U4mp + (r2 + X2) * t.U2mp + (r1 + l1) * t.t.U1mp[0];
    }
    return a;
}

// an e-e slope with what its transpose needs
struct Slope {
    double I4, I2, J1, raw, lnee, dn, dT, fa, fb;
};
template <int W>
__device__ __forceinline__ double ee_slope(const CollTables& T, const Mem& s, const Tab& t, const int k,
                                           const double f, Slope& o) {
    const int n = T.np;
    double fin[1] = {f}, fm[1], fp[1], I4[1], I2[1], J1[1], S4, S2;
    neighbours<1, W>(s.f, k, fin, fm, fp);
    o.fa = s.f[0];
    o.fb = s.f[1];
    cell_scans<1, W>(t.t, fin, fm, fp, s.tot, I4, I2, J1, S4, S2);
    double G[1], Gm[1], Gp[1];
    if (k < T.NB) {
        const double f00 = (o.fa - o.fb * t.t.r) * t.t.inv1r, df = o.fb - f00;
        const double i2s = f00 * t.t.A2[0] + df * t.t.B2[0];
        const double i4s = f00 * t.t.A4[0] + df * t.t.B4[0];
        G[0] = f * i4s + (t.t.U3[0] * f - 3.0 * i2s) * J1[0];
    } else {
        G[0] = (I4[0] + t.t.U3[0] * J1[0]) * f - 3.0 * I2[0] * J1[0];
    }
    o.lnee = adj::log_ee_d(4.0 * adj::kPi * S2, 4.0 * adj::kPi * S4, T.density_np, &o.dn, &o.dT);
    neighbours<1, W>(s.g, k, G, Gm, Gp);
    const double D = k < n - 1 ? (G[0] - Gp[0]) * t.t.Pn[0] : G[0];
    o.raw = (k == 0 ? ((-G[0]) * t.t.two_v0s - D) : ((Gm[0] - G[0]) * t.t.Pm[0] - D)) * t.t.Qn[0];
    o.I4 = I4[0]; o.I2 = I2[0]; o.J1 = J1[0];
    return o.raw * (T.c_kpre * o.lnee);
}
// transpose of the slope's derivative at f (adj::ee_slope_T): mu -> the cotangent of f
template <int W>
__device__ __forceinline__ double ee_slope_T(const CollTables& T, const Mem& s, const Tab& t, const int k,
                                             const double f, const Slope& o,
                                             const double mu) {
    const int n = T.np;
    const double norm = T.c_kpre * o.lnee;
    double w[1] = {k < n ? mu * norm * t.t.Qn[0] : 0.0}, wm[1], wp[1];
    neighbours<1, W>(s.f, k, w, wm, wp);   // (s.g may still be read by the slope before)
    double sum[3] = {k < n ? mu * o.raw : 0.0, 0.0, 0.0};   // of the norm, f00 (the fit's f at v = 0) and f[1]
    double lf = 0.0, l4 = 0.0, l2 = 0.0, l1 = 0.0;
    if (k < n) {
        const double lD = wp[0] - w[0], lDm = w[0] - wm[0];
        double lg = k < n - 1 ? lD * t.t.Pn[0] : lD;
        if (k >= 1) lg -= lDm * t.t.Pm[0];
        else lg -= w[0] * t.t.two_v0s;
        if (k < T.NB) {
            const double f00 = (o.fa - o.fb * t.t.r) * t.t.inv1r, df = o.fb - f00;
            const double v3 = t.t.U3[0], A2 = t.t.A2[0], B2 = t.t.B2[0], A4 = t.t.A4[0], B4 = t.t.B4[0];
            const double i2s = f00 * A2 + df * B2;
            const double i4s = f00 * A4 + df * B4;
            lf = lg * (i4s + v3 * o.J1);
            const double l_i4s = lg * f, l_i2s = -3.0 * lg * o.J1;
            l1 = lg * (v3 * f - 3.0 * i2s);
            sum[1] = l_i2s * (A2 - B2) + l_i4s * (A4 - B4);
            sum[2] = l_i2s * B2 + l_i4s * B4;
        } else {
            l4 = lg * f;
            l1 = lg * (t.t.U3[0] * f - 3.0 * o.I2);
            lf = lg * (o.I4 + t.t.U3[0] * o.J1);
            l2 = -3.0 * lg * o.J1;
        }
    }
    double r4, r2, r1;
    suffix_scans<3>(s.tot, l4, l2, l1, r4, r2, r1, sum);
    if (k == 0) lf += sum[1] * t.t.inv1r;
    if (k == 1) lf += sum[2] - sum[1] * t.t.r * t.t.inv1r;
    const double l_lnee = sum[0] * T.c_kpre;
    return lf + scans_T(t, k, n, l4, l2, l1, r4, r2, r1, l_lnee * o.dT * 4.0 * adj::kPi, l_lnee * o.dn * 4.0 * adj::kPi);
}

// x = A^{-1} f and y = A^{-T} lam of every collided plane of the cell; y
// replaces lam, and -y_i x_j on the tridiagonal pattern adds up to the
// coefficients' cotangents in s.la, lb, lc, ls
template <int G, int R>
__device__ __forceinline__ void solves_T(const CollTables& T, const StepT& p, const Mem& s, const double* fl,
                                         double* laml) {
    constexpr int kSteps = G == 8 ? 3 : (G == 16 ? 4 : 5);
    const int n = T.np;
    const int gl = threadIdx.x & (G - 1), group = threadIdx.x / G, ng = blockDim.x / G;
    const int i0 = gl * R;
    const int C = p.unit_planes;
    int l = p.l0, k = group;
    auto planes_of = [&](int ll) { return 1 + 2 * min(min(ll, p.m0), p.mmax); };
    auto settle = [&]() {
        while (l >= 1) {
            const int u = (planes_of(l) + C - 1) / C;
            if (k < u) return;
            k -= u;
            --l;
        }
        l = 0;
    };
    double la[R], lb[R], lc[R], ls[R];
#pragma unroll
    for (int e = 0; e < R; ++e) { la[e] = 0.0; lb[e] = 0.0; lc[e] = 0.0; ls[e] = 0.0; }
    settle();
    while (__any_sync(kFull, l >= 1)) {
        int j0 = 0, cnt = 0;
        if (l >= 1) {
            const int nq = planes_of(l), u = (nq + C - 1) / C;
            j0 = (int)((long long)nq * k / u);
            cnt = (int)((long long)nq * (k + 1) / u) - j0;
        }
        const int most = __reduce_max_sync(kFull, cnt);
        const int lv = l >= 1 ? l : 1;
        const double ll1 = lv * ((-0.5) * (lv + 1.0));
        const long long off0 = (l >= 1 ? (long long)p.plane_of[l * (p.m0 + 1)] + j0 : 0) * p.pstride + i0;
        double id[R], cp[R], Af[kSteps], Ab[kSteps], Tf[kSteps], Tb[kSteps];
        lane_pivots<G, R>(s.tri, lv, n, i0, cp, id);
        // c' of the point below, a of the point above
        double c_in = __shfl_up_sync(kFull, cp[R - 1], 1, G);
        if (gl == 0) c_in = 0.0;
        auto a_of = [&](int i) { return i < n ? s.tri.a[i] : 0.0; };
        {
            double A = 1.0, B = 1.0, Cf = 1.0, Cb = 1.0;
#pragma unroll
            for (int e = 0; e < R; ++e) {
                const int i = i0 + e;
                if (i < n) {
                    A = (i == 0) ? 0.0 : A * (-(s.tri.a[i] * id[e]));
                    Cf = (i == 0) ? 0.0 : Cf * (-(e > 0 ? cp[e > 0 ? e - 1 : 0] : c_in));
                }
            }
#pragma unroll
            for (int e = R - 1; e >= 0; --e) {
                const int i = i0 + e;
                if (i < n) {
                    B = (i == n - 1) ? 0.0 : B * (-cp[e]);
                    Cb = (i == n - 1) ? 0.0 : Cb * (-(s.tri.a[i + 1] * id[e]));
                }
            }
#pragma unroll
            for (int t = 0, off = 1; t < kSteps; ++t, off <<= 1) {
                const double Ap = __shfl_up_sync(kFull, A, off, G), Bp = __shfl_down_sync(kFull, B, off, G);
                const double Cfp = __shfl_up_sync(kFull, Cf, off, G), Cbp = __shfl_down_sync(kFull, Cb, off, G);
                const bool up = gl >= off, dn = gl + off < G;
                Af[t] = up ? A : 0.0; Tf[t] = up ? Cf : 0.0;
                Ab[t] = dn ? B : 0.0; Tb[t] = dn ? Cb : 0.0;
                if (up) { A *= Ap; Cf *= Cfp; }
                if (dn) { B *= Bp; Cb *= Cbp; }
            }
        }
        for (int b = 0; b < most; ++b) {
            const double* g = fl + off0 + b * p.pstride;
            double* o = laml + off0 + b * p.pstride;
            double x[R], y[R];
#pragma unroll
            for (int e = 0; e < R; ++e) {
                const bool in = b < cnt && i0 + e < n;
                x[e] = in ? g[e] : 0.0;
                y[e] = in ? o[e] : 0.0;
            }
            // forward sweeps: A's elimination on x, U^T on y
            double B = 0.0, D = 0.0;
#pragma unroll
            for (int e = 0; e < R; ++e) {
                B = (x[e] - B * a_of(i0 + e)) * id[e];
                D = y[e] - (e > 0 ? cp[e > 0 ? e - 1 : 0] : c_in) * D;
            }
#pragma unroll
            for (int t = 0, off = 1; t < kSteps; ++t, off <<= 1) {
                B = fma(Af[t], __shfl_up_sync(kFull, B, off, G), B);
                D = fma(Tf[t], __shfl_up_sync(kFull, D, off, G), D);
            }
            double u = __shfl_up_sync(kFull, B, 1, G), v = __shfl_up_sync(kFull, D, 1, G);
            if (gl == 0) { u = 0.0; v = 0.0; }
#pragma unroll
            for (int e = 0; e < R; ++e) {
                const bool in = i0 + e < n;
                if (in) {
                    u = (x[e] - u * a_of(i0 + e)) * id[e];
                    v = y[e] - (e > 0 ? cp[e > 0 ? e - 1 : 0] : c_in) * v;
                }
                x[e] = in ? u : 0.0;
                y[e] = in ? v : 0.0;
            }
            // backward sweeps: U on x, L^T on y
            B = 0.0; D = 0.0;
#pragma unroll
            for (int e = R - 1; e >= 0; --e) {
                B = x[e] - cp[e] * B;
                D = (y[e] - a_of(i0 + e + 1) * D) * id[e];
            }
#pragma unroll
            for (int t = 0, off = 1; t < kSteps; ++t, off <<= 1) {
                B = fma(Ab[t], __shfl_down_sync(kFull, B, off, G), B);
                D = fma(Tb[t], __shfl_down_sync(kFull, D, off, G), D);
            }
            u = __shfl_down_sync(kFull, B, 1, G);
            v = __shfl_down_sync(kFull, D, 1, G);
            if (gl == G - 1) { u = 0.0; v = 0.0; }
            const double x_out = u;   // x of the point above this run
#pragma unroll
            for (int e = R - 1; e >= 0; --e) {
                u = x[e] - cp[e] * u;
                v = (y[e] - a_of(i0 + e + 1) * v) * id[e];
                x[e] = u;
                y[e] = v;
            }
            double x_in = __shfl_up_sync(kFull, x[R - 1], 1, G);
            if (gl == 0) x_in = 0.0;
#pragma unroll
            for (int e = 0; e < R; ++e) {
                const int i = i0 + e;
                if (b < cnt && i < n) {
                    la[e] -= y[e] * (e > 0 ? x[e > 0 ? e - 1 : 0] : x_in);
                    lc[e] -= y[e] * (e + 1 < R ? x[e + 1 < R ? e + 1 : 0] : x_out);
                    const double lbi = -y[e] * x[e];
                    if (!(i == 0 && lv > 1)) lb[e] += lbi;
                    ls[e] += -ll1 * lbi;
                    o[e] = y[e];
                }
            }
        }
        k += ng;
        settle();
    }
    // the groups' sums, in order
    for (int q = 0; q < ng; ++q) {
        if (q == group) {
#pragma unroll
            for (int e = 0; e < R; ++e) {
                const int i = i0 + e;
                if (i < n) {
                    s.la[i] = (q ? s.la[i] : 0.0) + la[e];
                    s.lb[i] = (q ? s.lb[i] : 0.0) + lb[e];
                    s.lc[i] = (q ? s.lc[i] : 0.0) + lc[e];
                    s.ls[i] = (q ? s.ls[i] : 0.0) + ls[e];
                }
            }
        }
        __syncthreads();
    }
}

// adj::collide_cell_T: lam00 / laml hold the cotangents of the outputs and
// receive those of the inputs; starts: nsub rows for the substeps' starts
template <int G, int R, int W>
__device__ __forceinline__ void collide_cell_T(const CollTables& T, const StepT& p, const double* f00_in,
                                               const double* fl_in, double* lam00, double* laml, double* smem,
                                               double* starts) {
    const int n = T.np;
    const int k = threadIdx.x, pts = blockDim.x;
    const bool in = k < n;
    const Mem s = carve(smem, n, pts);
    Tab t;
    load(T, k, t);
    if (k == 0) { s.f[-1] = 0.0; s.f[pts] = 0.0; s.g[-1] = 0.0; s.g[pts] = 0.0; }
    double f = in ? f00_in[k] : 0.0;
    double lam = in ? lam00[k] : 0.0;
    const double h = p.hsub;
    if (p.ee)
        for (int sub = 0; sub < p.nsub; ++sub) {
            if (in) starts[(long long)sub * n + k] = f;
            double fs = f, acc = 0.0;
            for (int st = 0; st < 4; ++st) {
                Slope o;
                const double d = ee_slope<W>(T, s, t, k, fs, o);
                acc = fma(st == 0 || st == 3 ? h / 6.0 : h / 3.0, d, acc);
                fs = fma(st == 2 ? h : 0.5 * h, d, f);
            }
            f += acc;
        }
    if (p.eb) {
        // coefficients (adj::reset_coeff)
        double fin[1] = {f}, fm[1], fp[1], I2[1], I0[1], J1[1], S4, S2;
        neighbours<1, W>(s.f, k, fin, fm, fp);
        cell_scans<1, W>(t.t, fin, fm, fp, s.tot, I2, I0, J1, S4, S2);
        const double Tt = S4 * (4.0 * adj::kPi), N = S2 * (4.0 * adj::kPi);
        double le_dN, le_dT, zl_dN, zl_dT;
        const double lnee = adj::log_ee_d(N, Tt, T.density_np, &le_dN, &le_dT);
        const double zl = adj::zlog_ei_d(N, Tt, T.density_np, T.Zeta, &zl_dN, &zl_dT);
        const double scale = (-1.0) * lnee * T.kpre * p.Dt;
        const double vk = in ? T.vr[k] : 1.0;
        const double i2 = I2[0] * (4.0 * adj::kPi) / (vk * vk), i0 = I0[0] * (4.0 * adj::kPi);
        const double j1m = J1[0] * (4.0 * adj::kPi * vk);
        const double t1 = i0 + (2.0 * j1m - i2) / 3.0, t2 = (i2 + j1m) / 3.0;
        double Dm = 0.0, Dp = 0.0, S = 0.0;
        const bool mid = k > 0 && k < n - 1;
        if (mid) {
            const double vp = T.vr[k + 1], vm = T.vr[k - 1];
            Dm = 1.0 / (vk * 0.5 * (vp - vm) * (vk - vm));
            Dp = 1.0 / (vk * 0.5 * (vp - vm) * (vp - vk));
            S = 1.0 / (vk * vk * (vp - vm));
        }
        if (in) {
            s.tri.scat[k] = (((k == 0) ? 0.0 : t1 * lnee) + zl * N) / t.t.U3[0] * (T.kpre * p.Dt);
            s.tri.a[k] = mid ? (t2 * Dm - t1 * S) * scale : 0.0;
            s.tri.b[k] = k == 0 ? 8.0 * adj::kPi * f * scale : mid ? (8.0 * adj::kPi * f - t2 * (Dm + Dp)) * scale : 0.0;
            s.tri.c[k] = mid ? (t2 * Dp + t1 * S) * scale : 0.0;
        }
        __syncthreads();
        solves_T<G, R>(T, p, s, fl_in, laml);
        // cotangents of the coefficients -> f00 (adj::reset_coeff_T)
        double sum[4] = {0.0, 0.0, 0.0, 0.0};   // of scale, lnee, zl, N
        double l4 = 0.0, l2 = 0.0, l1 = 0.0;
        if (in) {
            const double la = s.la[k], lb = s.lb[k], lc = s.lc[k], ls = s.ls[k];
            const double Kk = T.kpre * p.Dt / t.t.U3[0];
            double l_t1 = 0.0, l_t2 = 0.0;
            if (k > 0) {
                l_t1 += ls * Kk * lnee;
                sum[1] = ls * Kk * t1;
            }
            sum[2] = ls * Kk * N;
            sum[3] = ls * Kk * zl;
            if (k == 0) {
                lam += lb * 8.0 * adj::kPi * scale;
                sum[0] = lb * 8.0 * adj::kPi * f;
            } else if (mid) {
                lam += lb * 8.0 * adj::kPi * scale;
                l_t2 += (-lb * (Dm + Dp) + la * Dm + lc * Dp) * scale;
                l_t1 += (-la * S + lc * S) * scale;
                sum[0] = lb * (8.0 * adj::kPi * f - t2 * (Dm + Dp)) + la * (t2 * Dm - t1 * S) + lc * (t2 * Dp + t1 * S);
            }
            l4 = (-l_t1 / 3.0 + l_t2 / 3.0) * (4.0 * adj::kPi) / (vk * vk);
            l2 = l_t1 * (4.0 * adj::kPi);
            l1 = (2.0 / 3.0 * l_t1 + l_t2 / 3.0) * (4.0 * adj::kPi * vk);
        }
        double r4, r2, r1;
        suffix_scans<4>(s.tot, l4, l2, l1, r4, r2, r1, sum);
        const double l_lnee = sum[1] + sum[0] * (-1.0) * T.kpre * p.Dt;
        const double l_N = sum[3] + l_lnee * le_dN + sum[2] * zl_dN;
        const double l_T = l_lnee * le_dT + sum[2] * zl_dT;
        lam += scans_T(t, k, n, l4, l2, l1, r4, r2, r1, l_T * (4.0 * adj::kPi), l_N * (4.0 * adj::kPi));
        __syncthreads();   // the totals are read before the next slope writes them
    }
    if (p.ee)
        for (int sub = p.nsub - 1; sub >= 0; --sub) {
            // the substep's stages again, their integrals kept (adj::ee_rk4_T)
            const double fs = in ? starts[(long long)sub * n + k] : 0.0;
            double S[4];
            Slope o[4];
            S[0] = fs;
#pragma unroll
            for (int st = 0; st < 4; ++st) {
                const double d = ee_slope<W>(T, s, t, k, S[st], o[st]);
                if (st < 3) S[st < 3 ? st + 1 : 0] = fma(st == 2 ? h : 0.5 * h, d, fs);
            }
            const double out = lam;
            double a = 0.0;
#pragma unroll
            for (int st = 3; st >= 0; --st) {
                const double c = (st == 0 || st == 3 ? h / 6.0 : h / 3.0) * out + (st == 3 ? 0.0 : st == 2 ? h : 0.5 * h) * a;
                a = ee_slope_T<W>(T, s, t, k, S[st], o[st], c);
                lam += a;
            }
        }
    if (in) lam00[k] = lam;
}

}  // namespace adjc
}  // namespace oshun
