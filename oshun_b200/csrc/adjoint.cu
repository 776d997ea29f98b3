// Adjoint kernels of one small step of the 1D path with m0 = 0 (FP64), over
// the math of adjoint_math.h:
//   stage_vjp_kernel   F'(s)^T c for one RK4 stage state s (FP64 or FP32
//                      arithmetic on FP64 vectors): one CTA per cell,
//                      one thread per momentum point computes the cotangent
//                      of every f_l(x, p) (transposed G/H stencils, x
//                      advection, current) and its share of the E_x(x)
//                      cotangent, summed over the CTA in a fixed order;
//   collide_adj_kernel the collision step's transpose (reverse sweep through
//                      the e-e RK4 substeps, the transposed Thomas solves and
//                      the dependence of the tridiagonal coefficients on f00),
//                      one CTA per cell (adjoint_cell.cuh);
//   stage_vjp2_kernel  F'(s)^T c of any grid (adjoint2d.cuh), and its
//                      form without the shared-memory window;
//   rk_combine_kernel  the linear combinations of the RK4 transpose.
// State vectors use the plane layout: f00 plane, the l >= 1 planes, the 6
// field planes (for m0 = 0 and numy = 1: f[l][x][p] then E_x[x], ...).
#include "adjoint2d.cuh"
#include "adjoint_cell.cuh"
#include "adjoint_math.h"
#include "oshun_internal.h"

namespace oshun {
namespace {

using adj::Coef1;
using adj::CollTables;
using adj::Grid1;

// T: arithmetic of the transpose (double; float for the FP32 bulk form),
// the vectors stay FP64
template <typename T>
__global__ void stage_vjp_kernel(const Grid1 g, const double* __restrict__ s, const double* __restrict__ c,
                                 double* __restrict__ out) {
    const int x = blockIdx.x;
    const int k = threadIdx.x;
    const long long fsz = (long long)(g.l0 + 1) * g.nx * g.np;
    const double* Ex = s + fsz;          // field 0 of the state
    const double* cE = c + fsz;          // cotangent of the E_x slope
    __shared__ double red[8];
    double e = 0.0;
    if (k < g.np) {
        for (int l = 0; l <= g.l0; ++l)
            out[((long long)l * g.nx + x) * g.np + k] = (double)adj::vjp_f<T>(g, Ex, c, cE, l, x, k);
        e = (double)adj::vjp_E_point<T>(g, s, c, x, k);
    }
    // E_x cotangent: warp sums, then warps in order
    for (int off = 16; off > 0; off >>= 1) e += __shfl_xor_sync(0xffffffffu, e, off);
    if ((k & 31) == 0) red[k >> 5] = e;
    __syncthreads();
    if (k == 0) {
        double tot = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
        out[fsz + x] = tot;
        for (int f = 1; f < 6; ++f) out[fsz + (long long)f * g.nx + x] = 0.0;
    }
}

// the cell's field cotangents: the points' shares summed over the CTA in a fixed
// order, then the transposes of Ampere/Faraday
__device__ __forceinline__ void field_cotangents(const adj2::Grid2& g, const double* __restrict__ c,
                                                 double* __restrict__ out, const long long cell, const double (&cF)[6]) {
    __shared__ double red[6][8];
    const int k = threadIdx.x;
    const int lane = k & 31, warp = k >> 5;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        double v = cF[f];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[f][warp] = v;
    }
    __syncthreads();
    if (k == 0) {
        double F[6];
        for (int f = 0; f < 6; ++f) {
            F[f] = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) F[f] += red[f][w];
        }
        const adj2::Nbr n = adj2::nbr(g, cell);
        auto C = [&](int f, long long cc) { return adj2::fld(g, c, f, cc); };
        F[0] += g.idy * (C(5, n.yp) - C(5, n.ym));
        F[1] += -g.idx * (C(5, n.xp) - C(5, n.xm));
        F[2] += -g.idy * (C(3, n.yp) - C(3, n.ym)) + g.idx * (C(4, n.xp) - C(4, n.xm));
        F[3] += -g.idy * (C(2, n.yp) - C(2, n.ym));
        F[4] += g.idx * (C(2, n.xp) - C(2, n.xm));
        F[5] += g.idy * (C(0, n.yp) - C(0, n.ym)) - g.idx * (C(1, n.xp) - C(1, n.xm));
        double* of = out + (1 + (long long)g.nplanes) * g.pstride;
        for (int f = 0; f < 6; ++f) of[(long long)f * g.cells + cell] = F[f];
    }
}

// F'(s)^T c for any grid (adjoint2d.cuh): one CTA per cell, one thread per
// momentum point k.  The transposed momentum stencils of a target's cotangent
// c need c(k) and D = c(k+1) - c(k-1) alone, the advection v (c(x+1) - c(x-1))
// and the same in y; a thread forms these four for the target rows s-1, s, s+1
// once (a window of three rows in shared memory, its own column: no barrier)
// and source (s, M) combines the up to nine targets that it feeds.  Gathering
// every target's three momentum points and four neighbours per source from
// global memory instead took 94 us a stage (32 x 32 cells, l0 = 4, m0 = 2, np =
// 64), most of it address arithmetic and load latency; the window takes 70.
__global__ void __launch_bounds__(256) stage_vjp2_kernel(const adj2::Grid2 g, const double* __restrict__ s,
                                                         const double* __restrict__ c, double* __restrict__ out) {
    using adj2::Cx;
    extern __shared__ double win[];   // [3 rows][m0+1][8][threads]
    const long long cell = blockIdx.x;
    const int k = threadIdx.x, np = g.np, stride = blockDim.x;
    double cF[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (k < np) {
        const int m1 = g.m0 + 1;
        const adj2::Nbr nb = adj2::nbr(g, cell);
        const bool has_y = g.ny > 1;
        const double v = g.vr[k], ip = g.invp[k], wj = g.wj[k];
        const double Ex = adj2::fld(g, s, 0, cell), Ey = adj2::fld(g, s, 1, cell), Ez = adj2::fld(g, s, 2, cell);
        const double Bx = adj2::fld(g, s, 3, cell), By = adj2::fld(g, s, 4, cell), Bz = adj2::fld(g, s, 5, cell);
        const double cdEx = adj2::fld(g, c, 0, cell), cdEy = adj2::fld(g, c, 1, cell), cdEz = adj2::fld(g, c, 2, cell);
        const long long o = cell * np + k;
        auto slot = [&](int t, int m) { return win + (size_t)((t % 3) * m1 + m) * 8 * stride + k; };
        // base of harmonic (t, m) in a vector
        auto plane = [&](const double* u, int t, int m) {
            return t == 0 ? u : u + (1 + (long long)g.plane_of[t * m1 + m]) * g.pstride;
        };
        auto load_row = [&](int t) {
            const int nclean = t >= 2 ? min(t - 1, 80) : 0;   // CLEAN_LOW_PC: no cotangent below
            for (int m = 0; m <= min(t, g.m0); ++m) {
                const double* b = plane(c, t, m);
                double* w = slot(t, m);
#pragma unroll
                for (int comp = 0; comp < 2; ++comp) {
                    double cc = 0.0, D = 0.0, X = 0.0, Y = 0.0;
                    if (comp == 0 || m > 0) {
                        const double* q = b + comp * g.pstride;
                        if (k >= nclean) {
                            cc = q[o];
                            X = v * (q[nb.xp * np + k] - q[nb.xm * np + k]);
                            if (has_y) Y = v * (q[nb.yp * np + k] - q[nb.ym * np + k]);
                        }
                        // p = 0 has no G and its own H (below); the last point differences onto itself
                        const double up = k + 1 < np ? (k + 1 >= nclean ? q[o + 1] : 0.0) : -cc;
                        D = up - (k >= 2 && k - 1 >= nclean ? q[o - 1] : 0.0);
                    }
                    w[comp * stride] = cc;
                    w[(2 + comp) * stride] = D;
                    w[(4 + comp) * stride] = X;
                    w[(6 + comp) * stride] = Y;
                }
            }
        };
        load_row(0);
        for (int sl = 0; sl <= g.l0; ++sl) {
            if (sl < g.l0) load_row(sl + 1);
            for (int M = 0; M <= min(sl, g.m0); ++M) {
                const CoefLM& cf = g.coef[sl * m1 + M];
                const double ipx = ip * cf.invpax;
                // the source's value and stencils at k
                Cx f, G{0.0, 0.0}, H{0.0, 0.0};
                {
                    const double* b = plane(s, sl, M);
                    double r[2][3];
#pragma unroll
                    for (int comp = 0; comp < 2; ++comp)
                        if (comp == 0 || M > 0) {
                            const double* q = b + comp * g.pstride + o;
                            r[comp][1] = q[0];
                            r[comp][0] = k > 0 ? q[-1] : 0.0;
                            r[comp][2] = k + 1 < np ? q[1] : q[0];
                        } else {
                            r[comp][0] = r[comp][1] = r[comp][2] = 0.0;
                        }
                    f = {r[0][1], r[1][1]};
                    auto st = [&](const double* x, double& Gc, double& Hc) {
                        const double d = x[0] - x[2];
                        if (sl == 0) {
                            Gc = k == 0 ? (x[2] - (x[1] - x[2] * g.g00_s) * g.g00_inv) * g.g00_gr : d;
                        } else {
                            Hc = k == 0 ? cf.hp0 * x[2] : ipx * x[1] + d;
                            Gc = k == 0 ? 0.0 : cf.gfac * d + Hc;
                        }
                    };
                    st(r[0], G.r, H.r);
                    if (M > 0) st(r[1], G.i, H.i);
                }
                Cx acc{0.0, 0.0};
                auto cot = [&](const double* w) -> Cx { return {w[0], w[stride]}; };
                // conj(a) u
                auto add = [&](double ar, double ai, Cx u) {
                    acc.r += ar * u.r + ai * u.i;
                    acc.i += ar * u.i - ai * u.r;
                };
                // a target through G (or H) and a difference term; a = (ar + i ai) the field factor
                auto term = [&](int t, int m, bool isH, double ar, double ai, double dif, bool ydir) -> Cx {
                    const double* w = slot(t, m);
                    const Cx cc = cot(w);
                    Cx u{w[2 * stride], w[3 * stride]};
                    if (sl > 0) {
                        const double gf = isH ? 1.0 : 1.0 + cf.gfac, pi = k > 0 ? ipx : 0.0;
                        u.r = gf * u.r + pi * cc.r;
                        u.i = gf * u.i + pi * cc.i;
                    }
                    // what point 0 of the target takes from points 0 and 1
                    if (k <= 1 && t < 2) {   // (CLEAN_LOW_PC leaves point 0 of higher rows none)
                        const double e0 = sl == 0 ? (k == 0 ? -g.g00_gr * g.g00_inv : g.g00_gr * (1.0 + g.g00_inv * g.g00_s))
                                                  : (isH && k == 1 ? cf.hp0 : 0.0);
                        if (e0 != 0.0) {
                            const double* q = plane(c, t, m) + cell * np;
                            u.r += e0 * q[0];
                            if (m > 0) u.i += e0 * q[g.pstride];
                        }
                    }
                    add(ar, ai, u);
                    const double* dw = w + (ydir ? 6 : 4) * stride;
                    acc.r += dif * dw[0];
                    acc.i += dif * dw[stride];
                    return cc;
                };
                const bool up = sl + 1 <= g.l0, dn = sl >= 1;
                auto in = [&](int t, int m) { return m <= min(t, g.m0); };
                if (up) {
                    const Cx t = term(sl + 1, M, false, cf.ex_g * Ex, 0.0, cf.ax_p, false);
                    cF[0] += cf.ex_g * (t.r * G.r + t.i * G.i);
                }
                if (dn && in(sl - 1, M)) {
                    const Cx t = term(sl - 1, M, true, cf.ex_h * Ex, 0.0, cf.ax_m, false);
                    cF[0] += cf.ex_h * (t.r * H.r + t.i * H.i);
                }
                if (M + 1 <= g.m0) {
                    if (up) {
                        const Cx t = term(sl + 1, M + 1, false, cf.em_g * Ey, -cf.em_g * Ez, has_y ? cf.ay_pp : 0.0, true);
                        cF[1] += cf.em_g * (t.r * G.r + t.i * G.i);
                        cF[2] += cf.em_g * (t.r * G.i - t.i * G.r);
                    }
                    if (dn && in(sl - 1, M + 1)) {
                        const Cx t = term(sl - 1, M + 1, true, cf.em_h * Ey, -cf.em_h * Ez, has_y ? cf.ay_mp : 0.0, true);
                        cF[1] += cf.em_h * (t.r * H.r + t.i * H.i);
                        cF[2] += cf.em_h * (t.r * H.i - t.i * H.r);
                    }
                    if (dn && in(sl, M + 1)) {
                        const Cx t = cot(slot(sl, M + 1));
                        add(0.5 * Bz, 0.5 * By, t);
                        cF[5] += 0.5 * (t.r * f.r + t.i * f.i);
                        cF[4] += 0.5 * (t.i * f.r - t.r * f.i);
                    }
                }
                if (M >= 1) {
                    if (in(sl - 1, M - 1)) {
                        const Cx t = term(sl - 1, M - 1, true, cf.ep_h * Ey, cf.ep_h * Ez, has_y ? cf.ay_mm : 0.0, true);
                        cF[1] += cf.ep_h * (t.r * H.r + t.i * H.i);
                        cF[2] += cf.ep_h * (t.i * H.r - t.r * H.i);
                    }
                    if (up) {
                        const Cx t = term(sl + 1, M - 1, false, cf.ep_g * Ey, cf.ep_g * Ez, has_y ? cf.ay_pm : 0.0, true);
                        cF[1] += cf.ep_g * (t.r * G.r + t.i * G.i);
                        cF[2] += cf.ep_g * (t.i * G.r - t.r * G.i);
                    }
                    {
                        const Cx t = cot(slot(sl, M - 1));
                        add(cf.b_m * Bz, -cf.b_m * By, t);
                        cF[5] += cf.b_m * (t.r * f.r + t.i * f.i);
                        cF[4] += cf.b_m * (t.r * f.i - t.i * f.r);
                    }
                    {
                        const Cx t = cot(slot(sl, M));
                        add(0.0, -(double)M * Bx, t);
                        cF[3] += (double)M * (t.r * f.i - t.i * f.r);
                    }
                }
                // the current: dEx = sum wj Re f10, dEy = 2 sum wj Re f11, dEz = -2 sum wj Im f11
                if (sl == 1 && M == 0) acc.r += wj * cdEx;
                if (sl == 1 && M == 1) { acc.r += 2.0 * wj * cdEy; acc.i += -2.0 * wj * cdEz; }
                double* q = (sl == 0 ? out : out + (1 + (long long)g.plane_of[sl * m1 + M]) * g.pstride) + o;
                q[0] = acc.r;
                if (M > 0) q[g.pstride] = acc.i;
            }
        }
    }
    field_cotangents(g, c, out, cell, cF);
}

// The same gathered point by point from global memory (adj2::vjp_source): for
// rows whose window of targets does not fit in shared memory.
__global__ void stage_vjp2_gather_kernel(const adj2::Grid2 g, const double* __restrict__ s, const double* __restrict__ c,
                                  double* __restrict__ out) {
    const long long cell = blockIdx.x;
    const int k = threadIdx.x;
    double cF[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (k < g.np) {
        const double cdEx = adj2::fld(g, c, 0, cell), cdEy = adj2::fld(g, c, 1, cell), cdEz = adj2::fld(g, c, 2, cell);
        for (int l = 0; l <= g.l0; ++l)
            for (int M = 0; M <= (l < g.m0 ? l : g.m0); ++M) {
                adj2::Cx v = adj2::vjp_source(g, s, c, l, M, cell, k, cF);
                // the current: dEx = sum wj Re f10, dEy = 2 sum wj Re f11, dEz = -2 sum wj Im f11
                if (l == 1 && M == 0) v.r += g.wj[k] * cdEx;
                if (l == 1 && M == 1) { v.r += 2.0 * g.wj[k] * cdEy; v.i += -2.0 * g.wj[k] * cdEz; }
                if (l == 0) {
                    out[cell * g.np + k] = v.r;
                } else {
                    const long long q = g.plane_of[l * (g.m0 + 1) + M];
                    out[(1 + q) * g.pstride + cell * g.np + k] = v.r;
                    if (M > 0) out[(2 + q) * g.pstride + cell * g.np + k] = v.i;
                }
            }
    }
    field_cotangents(g, c, out, cell, cF);
}

// FP64 state vector <-> the FP32 planes and fields of an FP32-split handle
__global__ void to_fp32_kernel(const double* __restrict__ src, float* __restrict__ dst, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}
__global__ void to_fp64_kernel(const float* __restrict__ src, double* __restrict__ dst, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

// K: the form of collide_cell.cuh (nump <= 256: one thread a point).  16 warps
// an SM: the e-e sweeps, most of a cell's time, hold far fewer registers than
// the solves, which spill a little for it.  ws: the substeps' starts of every
// cell, nsub rows; shared memory for them would leave fewer CTAs an SM (600 cells
// of 64 points, 90 substeps: a step's transpose 3.34 ms against 1.96; five
// substeps 0.34 either way).
template <int K>
__global__ void __launch_bounds__(32 * point_warps(K), 16 / point_warps(K))
    collide_adj_kernel(const CollTables T, const adjc::StepT st, const double* __restrict__ y, double* __restrict__ lam,
                       double* __restrict__ ws) {
    extern __shared__ double smem[];
    const long long x = blockIdx.x;
    const int np = T.np;
    adjc::collide_cell_T<form_lanes(K), form_run(K), point_warps(K)>(
        T, st, y + x * np, y + st.pstride + x * np, lam + x * np, lam + st.pstride + x * np, smem, ws + x * st.nsub * np);
}

// out = a0 v0 + a1 v1 and, where acc is given, acc = base + v1
__global__ void rk_combine_kernel(double* out, const double* v0, double a0, const double* v1, double a1, double* acc,
                                  const double* base, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double v = v1 ? v1[i] : 0.0;
        out[i] = v1 ? a0 * v0[i] + a1 * v : a0 * v0[i];
        if (acc) acc[i] = base[i] + v;
    }
}

}  // namespace

cudaError_t launch_stage_vjp(const Grid1& g, const double* s, const double* c, double* out, cudaStream_t st,
                             bool fp32) {
    const int threads = ((g.np + 31) / 32) * 32;
    if (threads > 256) return cudaErrorInvalidValue;
    if (fp32) stage_vjp_kernel<float><<<g.nx, threads, 0, st>>>(g, s, c, out);
    else stage_vjp_kernel<double><<<g.nx, threads, 0, st>>>(g, s, c, out);
    return cudaGetLastError();
}

cudaError_t launch_convert(const double* src, float* dst, long long n, cudaStream_t st) {
    long long b = (n + 255) / 256;
    if (b > 148 * 8) b = 148 * 8;
    if (b < 1) return cudaSuccess;
    to_fp32_kernel<<<(unsigned)b, 256, 0, st>>>(src, dst, n);
    return cudaGetLastError();
}
cudaError_t launch_convert(const float* src, double* dst, long long n, cudaStream_t st) {
    long long b = (n + 255) / 256;
    if (b > 148 * 8) b = 148 * 8;
    if (b < 1) return cudaSuccess;
    to_fp64_kernel<<<(unsigned)b, 256, 0, st>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_collide_adj(const CollTables& T, int l0, int nx, const double* y, double* lam, int ee, int eb,
                               int nsub, double hsub, double Dt, double* ws, cudaStream_t st, const int* plane_of,
                               int m0, int mmax) {
    if (T.np > 256) return cudaErrorInvalidValue;
    const int K = collide_form(T.np);
    const adjc::StepT s{l0, m0, mmax, collide_unit_planes(T.np, l0, m0, mmax, 1, 1), ee, eb, nsub, hsub, Dt, plane_of,
                        (long long)nx * T.np};   // nx: the cells of the grid
    return with_form(K, [&](auto form) {
        constexpr int F = decltype(form)::value;
        if constexpr (F <= 32) {
            const size_t smem = sizeof(double) * adjc::cell_doubles(T.np, 32 * point_warps(F));
            collide_adj_kernel<F><<<nx, 32 * point_warps(F), smem, st>>>(T, s, y, lam, ws);
            return cudaGetLastError();
        }
        return cudaErrorInvalidValue;
    });
}

cudaError_t launch_stage_vjp2(const adj2::Grid2& g, const double* s, const double* c, double* out, cudaStream_t st) {
    const int threads = ((g.np + 31) / 32) * 32;
    if (threads > 256) return cudaErrorInvalidValue;
    const size_t smem = sizeof(double) * 3 * 8 * (size_t)(g.m0 + 1) * threads;
    // The window pays where the CTAs that its shared memory leaves on an SM hold
    // all cells within three waves, or are four or have five warps; else gathering,
    // with all the SM's warps, is the faster one.  A step's vjp, us, window / gather: 144 cells
    // of 64 points, l0 = m0 = 8, 957 / 1855; 1024 cells, m0 = 4, l0 = 4, 96 points (six
    // warps) 1224 / 1480, 64 points (six) 944 / 950, 128 points (four) 1795 / 1630; l0 =
    // m0 = 6, 64 points (four) 1919 / 1705, 96 points (three) 3134 / 2843, 32 points
    // (five) 1147 / 1458; m0 = 8, 32 points (four CTAs) 1769 / 2338; 391 cells of 117
    // points, l0 = 7, m0 = 4, 2.6 waves, 2119 / 2177.
    const long long fit = (228 * 1024) / (long long)(smem + 1024);
    if (smem <= 200 * 1024 && (g.cells <= 3 * fit * sm_count() || fit >= 4 || fit * (threads / 32) >= 5)) {
        const cudaError_t e = ensure_dyn_smem((const void*)stage_vjp2_kernel, smem);
        if (e != cudaSuccess) return e;
        stage_vjp2_kernel<<<(unsigned)g.cells, threads, smem, st>>>(g, s, c, out);
    } else {
        stage_vjp2_gather_kernel<<<(unsigned)g.cells, threads, 0, st>>>(g, s, c, out);
    }
    return cudaGetLastError();
}

cudaError_t launch_rk_combine(double* out, const double* v0, double a0, const double* v1, double a1, double* acc,
                              const double* base, long long n, cudaStream_t st) {
    long long b = (n + 255) / 256;
    if (b > 148 * 8) b = 148 * 8;
    rk_combine_kernel<<<(unsigned)b, 256, 0, st>>>(out, v0, a0, v1, a1, acc, base, n);
    return cudaGetLastError();
}

}  // namespace oshun
