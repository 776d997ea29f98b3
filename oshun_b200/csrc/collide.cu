// Fokker-Planck collision step, all arithmetic in FP64, one CTA or one warp per
// configuration-space cell: collide_cell_kernel (tridiagonal, rows to 512
// points; many cells: collide_ee_kernel and collide_solve_kernel),
// collide_warp_kernel (tridiagonal, longer rows) and collide_kernel (staged
// chunks, dense matrices).
//
//   1. f00 e-e, Explicit_EC_FP::loop (OSHUN-1/def-FokkerPlanck.cpp:590-625):
//      nsub RK4 substeps (RungeKutta4_ee::advance, :518-553) of Bell's
//      number/energy conserving operator (EE_isotropic_conserva::Getslope,
//      :192-267).  collide_cell_kernel: one thread a momentum point, CTA
//      scans; the others: warp 0, the cumulative integrals I4, I2 (forward)
//      and J1 (backward) as warp scans over lane-owned runs of the p axis.
//   2. Coefficients of the implicit f_lm step from the new f00,
//      Implicit_FLM_step::reset_coeff (:808-939): I2, I0, J_{-1} scans,
//      Coulomb logarithms, scattering term, the tridiagonal Alpha_Tri,
//      f00 derivatives.  Computed once per cell for every l (the reference
//      computes them in both f1_loop and flm_loop with the same f00).
//   3. (I - Dt C_l) f_lm^{n+1} = f_lm^n for every collided plane,
//      Implicit_FLM_step::advance (:943-1035):
//      tridiagonal: lane groups with rows in registers and the recursions as
//        scans, or (collide_kernel) the cell's planes staged through shared
//        memory in chunks, a thread running the reference's Thomas recursion
//        (TridiagonalSolve, OSHUN-1/def-Nmethods.cpp:142-167) on one plane;
//      dense: per l the np x np matrix is assembled in a per-CTA global
//        workspace and each warp runs the reference's Gauss-Seidel
//        (def-Nmethods.cpp:44-136: dominance test, <= 5 sweeps, prefix
//        convergence rule) on one complex right-hand side.
#include <float.h>

#include <algorithm>
#include <type_traits>

#include "collide_cell.cuh"
#include "oshun_internal.h"

namespace oshun {
namespace {

constexpr int kCollideThreads = 128;

// The three cumulative integrals of one f on one warp, interleaved:
//   I4[k] = sum_{i=1..k} U4[i] f[i] + U4m1[i] f[i-1]
//   I2[k] = sum_{i=1..k} U2[i] f[i] + U2m1[i] f[i-1]
//   J1[k] = sum_{i=k+1..n-1} U1[i] f[i] + U1m1[i] f[i-1]
// Each lane sums a contiguous run of k, keeping each term in the output
// arrays (the I4 and I2 terms at their k, the J1 term of i at i - 1, all
// inside the lane's own run), the lanes' run totals are combined by a warp
// scan, and the lane then accumulates its run again from the scanned start
// out of the kept terms; the three chains are independent and interleaved.
template <class T4, class T2, class T1>
__device__ void warp_cumsum3(double* I4, double* I2, double* J1, int n, T4 t4, T2 t2, T1 t1) {
    const int lane = threadIdx.x & 31;
    const int E = (n + 31) >> 5;
    const int b = min(lane * E, n), e = min(b + E, n);
    double l4 = 0.0, l2 = 0.0, l1 = 0.0;
    for (int k = b; k < e; ++k) {
        if (k > 0) {
            const double v4 = t4(k), v2 = t2(k);
            l4 += v4; l2 += v2;
            I4[k] = v4; I2[k] = v2;
        }
        if (k + 1 <= n - 1) {
            const double v1 = t1(k + 1);
            l1 += v1;
            J1[k] = v1;
        }
    }
    double s4 = l4, s2 = l2, s1 = l1;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double v4 = __shfl_up_sync(kFull, s4, off);
        const double v2 = __shfl_up_sync(kFull, s2, off);
        const double v1 = __shfl_down_sync(kFull, s1, off);
        if (lane >= off) { s4 += v4; s2 += v2; }
        if (lane + off < 32) s1 += v1;
    }
    double r4 = __shfl_up_sync(kFull, s4, 1), r2 = __shfl_up_sync(kFull, s2, 1);
    double r1 = __shfl_down_sync(kFull, s1, 1);
    if (lane == 0) { r4 = 0.0; r2 = 0.0; }
    if (lane == 31) r1 = 0.0;
    for (int k = b; k < e; ++k) {
        if (k > 0) { r4 += I4[k]; r2 += I2[k]; }
        I4[k] = r4;
        I2[k] = r2;
    }
    for (int k = e - 1; k >= b; --k) {
        if (k + 1 <= n - 1) r1 += J1[k];
        J1[k] = r1;
    }
    __syncwarp();
}

// Coulomb logarithms, NRL formulary as coded in OSHUN-1/def-FokkerPlanck.cpp:41-95
__device__ double log_ee(double ne, double Te, double density_np) {
    if (ne > 0.000000001) {
        Te /= (3.0 * ne);
        Te *= 511000;
        ne *= density_np;
        Te = log(Te);
        ne = log(ne);
        const double d = sub_rn(Te, 2.0);
        const double v = sub_rn(fma_rn(1.25, Te, fma_rn(-0.5, ne, 23.5)), sqrt(fma_rn(mul_rn(0.0625, d), d, 0.00001)));
        if (v > 2.0) return v;
    }
    return 2.0;
}
__device__ double zlog_ei(double ne, double Te, double density_np, double Zeta) {
    if (ne > 0.0000001) {
        Te /= (3.0 * ne);
        Te *= 511000;
        ne *= density_np;
        Te = log(Te);
        ne = log(ne);
        const double v = add_rn(fma_rn(-0.5, ne, 24.0), Te);
        if (v > 2.0) return v * Zeta;
    }
    return 2.0 * Zeta;
}

// The planes hold f - ref when a momentum profile is given (FP32 split):
// f of plane q at momentum point p, and the stored value of f.
// (FP64 planes hold f itself: no profile is read for them.)
// The profile row of plane q when the plane keeps one (FP32 planes), else null:
// looked up once per plane, so the plane loops branch once per plane
template <typename TP>
__device__ __forceinline__ const float* ref_row(const CollideArgs& a, long long q) {
    if constexpr (sizeof(TP) == sizeof(float)) return (a.pl_ref32 && __ldg(a.pl_keep + q)) ? a.pl_ref32 + q * a.np : nullptr;
    return nullptr;
}
template <typename TP>
__device__ __forceinline__ double ref_at(const CollideArgs& a, long long q, int p) {
    if constexpr (sizeof(TP) == sizeof(float))
        return (a.pl_ref32 && __ldg(a.pl_keep + q)) ? (double)__ldg(a.pl_ref32 + q * a.np + p) : 0.0;
    return 0.0;
}

struct Smem {
    double *f, *f0, *f1, *fh, *I4, *I2, *J1;            // e-e work (np each)
    double *tri_a, *tri_b, *tri_c, *scat, *df0, *ddf0;  // implicit coefficients (np each)
    double* sc;                                          // scalars: [0] dense-term scale
    double* chunk;                                       // staged planes / solver scratch
};

constexpr int kSmemArrays = 13;
constexpr int kSmemScalars = 4;

__device__ Smem carve(double* base, int np) {
    Smem s;
    s.f = base; s.f0 = base + np; s.f1 = base + 2 * np; s.fh = base + 3 * np;
    s.I4 = base + 4 * np; s.I2 = base + 5 * np; s.J1 = base + 6 * np;
    s.tri_a = base + 7 * np; s.tri_b = base + 8 * np; s.tri_c = base + 9 * np;
    s.scat = base + 10 * np; s.df0 = base + 11 * np; s.ddf0 = base + 12 * np;
    s.sc = base + kSmemArrays * np;
    s.chunk = s.sc + kSmemScalars;
    return s;
}

// e-e substeps and implicit step of one collision call: from the arguments,
// or, when a device clock is given, by the reference's clock arithmetic for a
// step ending at the clock's t (Explicit_EC_FP::loop, def-FokkerPlanck.cpp:
// 598-599; Euler_Backward, :1277, 1297), as collide_params does on the host
struct StepP {
    int nsub;
    double hsub, Dt;
};
__device__ __forceinline__ StepP step_params(const CollideArgs& a) {
    StepP p{a.nsub, a.hsub, a.Dt};
    if (a.clock) {
        const double t = a.clock[0], t_ee = a.clock[1], t_eb = a.clock[2];
        p.nsub = (int)((t - t_ee) / a.small_dt) + 1;
        p.hsub = (t - t_ee) / (double)p.nsub;
        p.Dt = t - t_eb;
    }
    return p;
}

// EE_isotropic_conserva::Getslope on warp 0: fh = C_ee(fin)
__device__ void ee_slope(const CollideArgs& a, const Smem& s, const double* fin, double* fh) {
    const int n = a.np;
    const int lane = threadIdx.x & 31;
    warp_cumsum3(s.I4, s.I2, s.J1, n, [&](int k) { return a.U4[k] * fin[k] + a.U4m1[k] * fin[k - 1]; },
                 [&](int k) { return a.U2[k] * fin[k] + a.U2m1[k] * fin[k - 1]; },
                 [&](int i) { return a.U1[i] * fin[i] + a.U1m1[i] * fin[i - 1]; });
    const double lnee = log_ee(4.0 * M_PI * s.I2[n - 1], 4.0 * M_PI * s.I4[n - 1], a.density_np);
    const double* vr = a.vr;
    const double v0s = vr[0] * vr[0], v1s = vr[1] * vr[1];
    // flux G_n (stored in I4); the first NB cells use the parabolic fit near v = 0
    for (int k = lane; k < n; k += 32) {
        double g;
        if (k < a.NB) {
            const double f00 = (fin[0] - fin[1] * v0s / v1s) / (1.0 - v0s / v1s);
            // v^3, v^5, v^7 tabulated on the host with the same pow() the reference calls
            const double v3 = a.U3[k], v5 = a.V5[k], v7 = a.V7[k];
            const double i2s = f00 * v3 / 3.0 + (fin[1] - f00) * v5 / v1s * 0.2;
            const double i4s = f00 * v5 * 0.2 + (fin[1] - f00) * v7 / (v1s * 7.0);
            g = fin[k] * i4s + (v3 * fin[k] - 3.0 * i2s) * s.J1[k];
        } else {
            double i2 = s.I2[k] * s.J1[k];
            i2 *= -3.0;
            double i4 = s.I4[k] + a.U3[k] * s.J1[k];
            i4 *= fin[k];
            g = i4 + i2;
        }
        s.I4[k] = g;
    }
    __syncwarp();
    // D_k = (G_k - G_{k+1}) P_k for k < n-1, D_{n-1} = G_{n-1}   (kept in I2)
    for (int k = lane; k < n; k += 32) s.I2[k] = (k < n - 1) ? (s.I4[k] - s.I4[k + 1]) * a.Pn[k] : s.I4[k];
    __syncwarp();
    const double norm = a.c_kpre * lnee;
    for (int k = lane; k < n; k += 32) {
        double v;
        if (k == 0) {
            v = (-1.0) * s.I4[0];
            v *= 2.0 / v0s;
            v -= s.I2[0];
            v *= a.Qn[0];
        } else {
            v = a.Qn[k] * (s.I2[k - 1] - s.I2[k]);
        }
        fh[k] = v * norm;
    }
    __syncwarp();
}

// Implicit_FLM_step::reset_coeff on warp 0 (f = f00 of the cell in smem)
__device__ void flm_reset(const CollideArgs& a, const Smem& s, const double* f) {
    const StepP sp = step_params(a);
    const int n = a.np;
    const int lane = threadIdx.x & 31;
    const double* vr = a.vr;
    double* I2 = s.I4;   // reuse the e-e work arrays
    double* I0 = s.I2;
    double* J1m = s.J1;
    warp_cumsum3(I2, I0, J1m, n, [&](int k) { return a.U4[k] * f[k] + a.U4m1[k] * f[k - 1]; },
                 [&](int k) { return a.U2[k] * f[k] + a.U2m1[k] * f[k - 1]; },
                 [&](int i) { return a.U1[i] * f[i] + a.U1m1[i] * f[i - 1]; });
    const double I2_temperature = I2[n - 1] * (4.0 * M_PI);
    const double I0_density = I0[n - 1] * (4.0 * M_PI);
    const double lnee = log_ee(I0_density, I2_temperature, a.density_np);
    const double zlnei = zlog_ei(I0_density, I2_temperature, a.density_np, a.Zeta);
    const double scale = (-1.0) * lnee * a.kpre * sp.Dt;
    if (lane == 0) s.sc[0] = scale;
    for (int k = lane; k < n; k += 32) {
        double i2 = I2[k] * (4.0 * M_PI);
        i2 /= vr[k] * vr[k];
        const double i0 = I0[k] * (4.0 * M_PI);
        const double j1m = J1m[k] * (4.0 * M_PI * vr[k]);
        const double t1 = i0 + (2.0 * j1m - i2) / 3.0;
        const double t2 = (i2 + j1m) / 3.0;
        double sc = (k == 0) ? 0.0 : t1 * lnee;
        sc += zlnei * I0_density;
        sc /= a.U3[k];
        sc *= a.kpre * sp.Dt;
        s.scat[k] = sc;
        double ta = 0.0, tb = 0.0, tc = 0.0;
        if (k == 0) {
            tb = 8.0 * M_PI * f[0] * scale;
        } else if (k < n - 1) {
            const double IvDnDm1 = 1.0 / (vr[k] * 0.5 * (vr[k + 1] - vr[k - 1]) * (vr[k] - vr[k - 1]));
            const double IvDnDp1 = 1.0 / (vr[k] * 0.5 * (vr[k + 1] - vr[k - 1]) * (vr[k + 1] - vr[k]));
            const double Ivsq2Dn = 1.0 / (vr[k] * vr[k] * (vr[k + 1] - vr[k - 1]));
            tb = (8.0 * M_PI * f[k] - t2 * (IvDnDm1 + IvDnDp1)) * scale;
            ta = (t2 * IvDnDm1 - t1 * Ivsq2Dn) * scale;
            tc = (t2 * IvDnDp1 + t1 * Ivsq2Dn) * scale;
        }
        s.tri_a[k] = ta; s.tri_b[k] = tb; s.tri_c[k] = tc;
        // raw -df/dv at n-1/2 (finished below); f0 is free once the e-e step is done
        s.f0[k] = (k >= 1) ? (f[k - 1] - f[k]) / (vr[k] - vr[k - 1]) : 0.0;
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
        double df, ddf;
        if (k == 0) {
            const double f00 = (f[0] - (vr[0] * vr[0] / (vr[1] * vr[1])) * f[1]) / (1.0 - (vr[0] * vr[0]) / (vr[1] * vr[1]));
            ddf = 2.0 * (f[1] - f00) / (vr[1] * vr[1]);
            df = ddf * vr[0];
        } else if (k < n - 1) {
            df = (f[k + 1] - f[k - 1]) / (vr[k + 1] - vr[k - 1]);
            ddf = (s.f0[k] - s.f0[k + 1]) / (0.5 * (vr[k + 1] - vr[k - 1]));
        } else {
            df = 0.0;
            ddf = s.f0[k];
        }
        if (k < n - 1) { df /= vr[k] * vr[k]; ddf /= 2.0 * vr[k]; }
        s.df0[k] = df;
        s.ddf0[k] = ddf;
    }
    __syncwarp();
}

template <typename TP>
__device__ void tridiagonal_chunks(const CollideArgs& a, const Smem& s, long long cell) {
    TP* planes = reinterpret_cast<TP*>(a.planes);
    const int* plane_l = a.plane_l;
    const int* plane_m = a.plane_m;
    const int nplanes = a.nplanes;
    const int n = a.np, ld = n + 1;
    for (int q0 = 0; q0 < nplanes; q0 += a.chunk) {
        const int nq = min(a.chunk, nplanes - q0);
        // stage: d column of plane j at chunk[j*2*ld], c' column at chunk[j*2*ld + ld]
        for (int idx = threadIdx.x; idx < nq * n; idx += blockDim.x) {
            const int j = idx / n, p = idx - j * n;
            s.chunk[(long long)j * 2 * ld + p] =
                (double)planes[(long long)(q0 + j) * a.pstride + cell * n + p] + ref_at<TP>(a, q0 + j, p);
        }
        __syncthreads();
        for (int j = threadIdx.x; j < nq; j += blockDim.x) {
            const int q = q0 + j;
            const int l = plane_l[q], m = plane_m[q];
            if (l < 1 || m > a.mmax_coll || (l == 1 ? !a.do_l1 : !a.do_lm)) continue;
            double* d = s.chunk + (long long)j * 2 * ld;
            double* c = d + ld;
            const double ll1 = l * ((-0.5) * (l + 1.0));
            // Thomas, TridiagonalSolve (def-Nmethods.cpp:150-166)
            double b0 = (l > 1 ? 0.0 : s.tri_b[0]) + (1.0 - ll1 * s.scat[0]);
            c[0] = s.tri_c[0] / b0;
            d[0] /= b0;
            for (int i = 1; i < n; ++i) {
                const double bi = s.tri_b[i] + (1.0 - ll1 * s.scat[i]);
                const double id = 1.0 / (bi - c[i - 1] * s.tri_a[i]);
                c[i] = s.tri_c[i] * id;
                d[i] = (d[i] - d[i - 1] * s.tri_a[i]) * id;
            }
            for (int i = n - 2; i > -1; --i) d[i] = d[i] - c[i] * d[i + 1];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < nq * n; idx += blockDim.x) {
            const int j = idx / n, p = idx - j * n;
            const int q = q0 + j;
            const int l = plane_l[q], m = plane_m[q];
            if (l < 1 || m > a.mmax_coll || (l == 1 ? !a.do_l1 : !a.do_lm)) continue;
            planes[(long long)q * a.pstride + cell * n + p] = (TP)(s.chunk[(long long)j * 2 * ld + p] - ref_at<TP>(a, q, p));
        }
        __syncthreads();
    }
}

// dense path: assemble Alpha for harmonic order el in the CTA workspace
__device__ void dense_assemble(const CollideArgs& a, const Smem& s, double* A, int el) {
    const int n = a.np;
    const double* vr = a.vr;
    const double LL = el;
    const double A1 = (LL + 1.0) * (LL + 2.0) / ((2.0 * LL + 1.0) * (2.0 * LL + 3.0));
    const double A2 = (-1.0) * (LL - 1.0) * LL / ((2.0 * LL + 1.0) * (2.0 * LL - 1.0));
    const double B1 = (-1.0) * (0.5 * LL * (LL + 1.0) + (LL + 1.0)) / ((2.0 * LL + 1.0) * (2.0 * LL + 3.0));
    const double B2 = ((-0.5) * LL * (LL + 1.0) + (LL + 2.0)) / ((2.0 * LL + 1.0) * (2.0 * LL + 3.0));
    const double B3 = (0.5 * LL * (LL + 1.0) + (LL - 1.0)) / ((2.0 * LL + 1.0) * (2.0 * LL - 1.0));
    const double B4 = (0.5 * LL * (LL + 1.0) - LL) / ((2.0 * LL + 1.0) * (2.0 * LL - 1.0));
    const double ll1 = el * ((-0.5) * (el + 1.0));
    const double sc = s.sc[0];  // (-1) lnee kpre Dt (def-FokkerPlanck.cpp:973)
    for (long long idx = threadIdx.x; idx < (long long)n * n; idx += blockDim.x) {
        const int i = (int)(idx / n), j = (int)(idx - (long long)i * n);
        double v = 0.0;
        if (i == j) v = s.tri_b[i];
        else if (j == i - 1) v = s.tri_a[i];
        else if (j == i + 1) v = s.tri_c[i];
        if (i == 0 && j == 0 && el > 1) v = 0.0;
        if (i < n - 1 && j < n - 1) {
            double t1 = A1 * s.ddf0[i] + B1 * s.df0[i]; t1 *= sc;
            double t2 = A1 * s.ddf0[i] + B2 * s.df0[i]; t2 *= sc;
            double t3 = A2 * s.ddf0[i] + B3 * s.df0[i]; t3 *= sc;
            double t4 = A2 * s.ddf0[i] + B4 * s.df0[i]; t4 *= sc;
            // same accumulation order as the reference row loop (def-FokkerPlanck.cpp:981-998)
            if (j == 0) {
                v += t1 * (2.0 * M_PI * pow(vr[0] / vr[i], el + 2) * vr[0] * vr[0] * (vr[1] - vr[0]));
                v += t3 * (2.0 * M_PI * pow(vr[0] / vr[i], el) * vr[0] * vr[0] * (vr[1] - vr[0]));
            }
            if (j >= 1 && j < i) {
                v += t1 * (2.0 * M_PI * pow(vr[j] / vr[i], el + 2) * vr[j] * vr[j] * (vr[j + 1] - vr[j - 1]));
                v += t3 * (2.0 * M_PI * pow(vr[j] / vr[i], el) * vr[j] * vr[j] * (vr[j + 1] - vr[j - 1]));
            }
            if (j == i) {
                // the reference reads vr[-1] at i = 0 (def-FokkerPlanck.cpp:989-990), a
                // denormal malloc header word; 0 here
                const double vlow = i > 0 ? vr[i - 1] : 0.0;
                v += t1 * (2.0 * M_PI * vr[i] * vr[i] * (vr[i] - vlow));
                v += t3 * (2.0 * M_PI * vr[i] * vr[i] * (vr[i] - vlow));
                v += t2 * (2.0 * M_PI * vr[i] * vr[i] * (vr[i + 1] - vr[i]));
                v += t4 * (2.0 * M_PI * vr[i] * vr[i] * (vr[i + 1] - vr[i]));
            }
            if (j > i) {
                v += t2 * (2.0 * M_PI * pow(vr[j] / vr[i], -el - 1) * vr[j] * vr[j] * (vr[j + 1] - vr[j - 1]));
                v += t4 * (2.0 * M_PI * pow(vr[j] / vr[i], -el + 1) * vr[j] * vr[j] * (vr[j + 1] - vr[j - 1]));
            }
        }
        if (i == j) v += 1.0 - ll1 * s.scat[i];
        A[idx] = v;
    }
}

// Gauss_Seidel on one warp; x: complex (re at xr, im at xi) in smem, initial
// guess = b.  Returns false (x untouched) when the dominance test fails.
__device__ void dense_gauss_seidel(const double* A, int n, const double* inv, double* xr, double* xi,
                                   const double* br, const double* bi, double* ovr, double* ovi) {
    const int lane = threadIdx.x & 31;
    const double tol = 1.0e-1;
    int iteration = 0, conv = 0;
    while ((iteration++ < 5) && (conv < n)) {
        for (int k = lane; k < n; k += 32) { ovr[k] = xr[k]; ovi[k] = xi[k]; }
        __syncwarp();
        for (int i = 0; i < n; ++i) {
            const double* row = A + (long long)i * n;
            double sr = 0.0, si = 0.0;
            for (int j = lane; j < n; j += 32) {
                if (j == i) continue;
                const double aij = row[j];
                sr += aij * xr[j];
                si += aij * xi[j];
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                sr += __shfl_xor_sync(kFull, sr, off);
                si += __shfl_xor_sync(kFull, si, off);
            }
            if (lane == 0) {
                xr[i] = inv[i] * (br[i] - sr);
                xi[i] = inv[i] * (bi[i] - si);
            }
            __syncwarp();
        }
        // prefix convergence test |dx_i| < tol |x_i + 20 DBL_MIN|
        conv = n;
        for (int base = 0; base < n; base += 32) {
            const int k = base + lane;
            bool ok = true;
            if (k < n) {
                const double dr = ovr[k] - xr[k], di = ovi[k] - xi[k];
                ok = hypot(dr, di) < tol * hypot(xr[k] + 20.0 * DBL_MIN, xi[k]);
            }
            const unsigned bad = __ballot_sync(kFull, !ok);
            if (bad) { conv = base + __ffs(bad) - 1; break; }
        }
        __syncwarp();
    }
}

template <typename TP>
__device__ void dense_solves(const CollideArgs& a, const Smem& s, long long cell, double* A, double* scratch) {
    TP* planes = reinterpret_cast<TP*>(a.planes);
    const int* plane_of = a.plane_of;
    const int n = a.np;
    const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    // per warp: x re/im, b re/im, old re/im (6n); shared: inv diag (n), dominance flag
    double* inv = scratch;
    int* dominant = reinterpret_cast<int*>(scratch + n);
    double* wbase = scratch + n + 2 + warp * 6 * n;
    double *xr = wbase, *xi = wbase + n, *br = wbase + 2 * n, *bi = wbase + 3 * n, *ovr = wbase + 4 * n,
           *ovi = wbase + 5 * n;
    for (int el = 1; el <= a.l0; ++el) {
        if (el == 1 ? !a.do_l1 : !a.do_lm) continue;
        dense_assemble(a, s, A, el);
        __syncthreads();
        if (threadIdx.x == 0) *dominant = 1;
        __syncthreads();
        // dominance: sequential signed row sums as in the reference
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            double row = 0.0;
            for (int j = 0; j < n; ++j) row += A[(long long)i * n + j];
            if (!(row < 2.0 * A[(long long)i * n + i])) atomicExch(dominant, 0);
            inv[i] = 1.0 / A[(long long)i * n + i];
        }
        __syncthreads();
        const int mtop = min(el, a.mmax_coll);
        if (*dominant) {
            for (int m = warp; m <= mtop; m += nwarps) {
                const long long q = plane_of[el * (a.m0 + 1) + m];
                const TP* pr_ = planes + q * a.pstride + cell * n;
                const TP* pi_ = planes + (q + 1) * a.pstride + cell * n;
                for (int k = threadIdx.x & 31; k < n; k += 32) {
                    br[k] = (double)pr_[k] + ref_at<TP>(a, q, k);
                    bi[k] = m > 0 ? (double)pi_[k] + ref_at<TP>(a, q + 1, k) : 0.0;
                    xr[k] = br[k];
                    xi[k] = bi[k];
                }
                __syncwarp();
                dense_gauss_seidel(A, n, inv, xr, xi, br, bi, ovr, ovi);
                TP* wr = planes + q * a.pstride + cell * n;
                TP* wi = planes + (q + 1) * a.pstride + cell * n;
                for (int k = threadIdx.x & 31; k < n; k += 32) {
                    wr[k] = (TP)(xr[k] - ref_at<TP>(a, q, k));
                    if (m > 0) wi[k] = (TP)(xi[k] - ref_at<TP>(a, q + 1, k));
                }
                __syncwarp();
            }
        } else if (threadIdx.x == 0) {
            atomicOr(a.status, 1);
            atomicAdd(a.status + 1, mtop + 1);
        }
        __syncthreads();
    }
}

// Opt-in backward-Euler e-e step (OSHUN_FLAG_IMPLICIT_EE; not a reference
// scheme) on one warp, f00 of the cell in s.f.  The explicit operator of
// EE_isotropic_conserva (def-FokkerPlanck.cpp:201-267) is
//   C(f)_k = c_kpre lnee Qn_k (D_{k-1} - D_k),  D_k = P_k (G_k - G_{k+1}),
//   G_j = A_j f_j - B_j  (A = I4 + v^3 J1, B = 3 I2 J1; the low-v fit's
//   i4s, i2s for j < NB); row 0 Qn_0 (-(2/v_0^2) G_0 - D_0), D_{n-1} = G_{n-1}.
// One step g - D C(g) = f over the whole e-e interval D, by Picard sweeps,
// each a tridiagonal solve with the coefficients of the previous iterate x
// (the first from f): on each face the B difference becomes a drag on g,
// B_{k+1} - B_k = gam_k ((1 - w) g_k + w g_{k+1}), gam_k = (B_{k+1} - B_k) /
// ((1 - w) x_k + w x_{k+1}), w = 1/2, or 0 / 1 (upwind) where 1/2 would give
// the face a coefficient of the wrong sign; likewise B_0 = (B_0 / x_0) g_0.
// Every sweep's matrix is then an M-matrix (f stays positive for any D),
// and at convergence (g = x) the operator is the explicit one exactly, so
// the step converges to the explicit scheme as D -> 0.
// face k (between points k and k+1): D_k = al g_k + be g_{k+1} + cs; the
// B difference stays explicit (cs) where the iterate is not positive there
__device__ __forceinline__ void ee_face(double Ak, double Ak1, double Bk, double Bk1, double xk, double xk1,
                                        double P, double& al, double& be, double& cs) {
    const double dB = Bk1 - Bk;
    const double h = 0.5 * (xk + xk1);
    cs = 0.0;
    if (!(h > 0.0)) { al = P * Ak; be = -P * Ak1; cs = P * dB; return; }
    double w = 0.5;
    double gam = dB / h;
    if (Ak + 0.5 * gam < 0.0) w = 1.0;
    else if (0.5 * gam > Ak1) w = 0.0;
    if (w != 0.5) {
        const double hw = (1.0 - w) * xk + w * xk1;
        if (!(hw > 0.0)) { al = P * Ak; be = -P * Ak1; cs = P * dB; return; }
        gam = dB / hw;
    }
    al = P * (Ak + gam * (1.0 - w));
    be = P * (gam * w - Ak1);
}
__device__ void ee_implicit_step(const CollideArgs& a, const Smem& s) {
    const StepP sp = step_params(a);
    const double D = a.clock ? (a.clock[0] - a.clock[1]) : sp.hsub * (double)sp.nsub;
    const int n = a.np;
    const int lane = threadIdx.x & 31;
    const double* vr = a.vr;
    const double v0s = vr[0] * vr[0], v1s = vr[1] * vr[1];
    double* x = s.f1;    // iterate
    double* A = s.f0;    // A_j, then the Thomas c'
    double* B = s.fh;    // B_j
    double* al = s.tri_a;
    double* be = s.tri_c;
    double* tb = s.tri_b;
    double* cs = s.scat;   // explicit face parts
    for (int k = lane; k < n; k += 32) x[k] = s.f[k];
    __syncwarp();
    for (int sweep = 0; sweep < a.ee_implicit; ++sweep) {
        warp_cumsum3(s.I4, s.I2, s.J1, n, [&](int k) { return a.U4[k] * x[k] + a.U4m1[k] * x[k - 1]; },
                     [&](int k) { return a.U2[k] * x[k] + a.U2m1[k] * x[k - 1]; },
                     [&](int i) { return a.U1[i] * x[i] + a.U1m1[i] * x[i - 1]; });
        const double lnee = log_ee(4.0 * M_PI * s.I2[n - 1], 4.0 * M_PI * s.I4[n - 1], a.density_np);
        const double dn = D * a.c_kpre * lnee;
        const double fz = (x[0] - x[1] * v0s / v1s) / (1.0 - v0s / v1s);
        for (int k = lane; k < n; k += 32) {
            const double j1 = s.J1[k], v3 = a.U3[k];
            double i4 = s.I4[k], i2 = s.I2[k];
            if (k < a.NB) {
                i2 = fz * v3 / 3.0 + (x[1] - fz) * a.V5[k] / v1s * 0.2;
                i4 = fz * a.V5[k] * 0.2 + (x[1] - fz) * a.V7[k] / (v1s * 7.0);
            }
            A[k] = i4 + v3 * j1;
            B[k] = 3.0 * i2 * j1;
        }
        __syncwarp();
        for (int k = lane; k < n - 1; k += 32)
            ee_face(A[k], A[k + 1], B[k], B[k + 1], x[k], x[k + 1], a.Pn[k], al[k], be[k], cs[k]);
        __syncwarp();
        const bool imp0 = x[0] > 0.0;
        const double a0 = imp0 ? A[0] - B[0] / x[0] : A[0];
        const double b0 = imp0 ? 0.0 : B[0];
        double* rhs = s.I2;   // free once A and B are formed
        for (int k = lane; k < n; k += 32) {
            const double q = a.Qn[k];
            double d0, c0;
            if (k == 0) { d0 = -q * ((2.0 / v0s) * a0 + al[0]); c0 = q * ((2.0 / v0s) * b0 - cs[0]); }
            else if (k < n - 1) { d0 = q * (be[k - 1] - al[k]); c0 = q * (cs[k - 1] - cs[k]); }
            else { d0 = q * (be[k - 1] - A[k]); c0 = q * cs[k - 1]; }
            tb[k] = 1.0 - dn * d0;
            rhs[k] = s.f[k] + dn * c0;
        }
        __syncwarp();
        if (lane == 0) {
            // Thomas: sub-diagonal -dn Qn_k al_{k-1}, super-diagonal dn Qn_k be_k;
            // c' into A, d' then the solution into x
            double sup = dn * a.Qn[0] * be[0];
            double cp = sup / tb[0];
            double dp = rhs[0] / tb[0];
            A[0] = cp; x[0] = dp;
            for (int k = 1; k < n; ++k) {
                const double sub = -dn * a.Qn[k] * al[k - 1];
                sup = k < n - 1 ? dn * a.Qn[k] * be[k] : 0.0;
                const double id = 1.0 / (tb[k] - sub * cp);
                cp = sup * id;
                dp = (rhs[k] - sub * dp) * id;
                A[k] = cp; x[k] = dp;
            }
            for (int k = n - 2; k >= 0; --k) x[k] -= A[k] * x[k + 1];
        }
        __syncwarp();
    }
    for (int k = lane; k < n; k += 32) s.f[k] = x[k];
    __syncwarp();
}

// e-e RK4 substeps of Explicit_EC_FP::loop on one warp (f00 of the cell in s.f)
__device__ void ee_substeps(const CollideArgs& a, const Smem& s) {
    const StepP sp = step_params(a);
    const int n = a.np;
    const int lane = threadIdx.x & 31;
    for (int sub = 0; sub < sp.nsub; ++sub) {
        const double h = sp.hsub;
        for (int k = lane; k < n; k += 32) { s.f0[k] = s.f[k]; s.f1[k] = s.f[k]; }
        __syncwarp();
        ee_slope(a, s, s.f1, s.fh);
        for (int k = lane; k < n; k += 32) {
            double t = s.fh[k] * (0.5 * h);
            s.f1[k] += t; t *= 1.0 / 3.0; s.f[k] += t;
        }
        __syncwarp();
        ee_slope(a, s, s.f1, s.fh);
        for (int k = lane; k < n; k += 32) {
            s.f1[k] = s.f0[k];
            double t = s.fh[k] * (0.5 * h);
            s.f1[k] += t; t *= 2.0 / 3.0; s.f[k] += t;
        }
        __syncwarp();
        ee_slope(a, s, s.f1, s.fh);
        for (int k = lane; k < n; k += 32) {
            double t = s.fh[k] * h;
            s.f0[k] += t; t *= 1.0 / 3.0; s.f[k] += t;
        }
        __syncwarp();
        ee_slope(a, s, s.f0, s.fh);
        for (int k = lane; k < n; k += 32) s.f[k] += s.fh[k] * (h / 6.0);
        __syncwarp();
    }
}

// the backward-Euler e-e step alone, one warp per cell (the collision
// kernels then run with do_ee = 0)
__global__ void __launch_bounds__(32) ee_implicit_kernel(const CollideArgs a) {
    extern __shared__ double smem[];
    const int n = a.np;
    const Smem s = carve(smem, n);
    const int lane = threadIdx.x & 31;
    for (long long cell = blockIdx.x; cell < a.cells; cell += gridDim.x) {
        for (int k = lane; k < n; k += 32) s.f[k] = a.f00[cell * n + k];
        __syncwarp();
        ee_implicit_step(a, s);
        for (int k = lane; k < n; k += 32) a.f00[cell * n + k] = s.f[k];
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kCollideThreads) collide_kernel(const CollideArgs a) {
    extern __shared__ double smem[];
    const int n = a.np;
    Smem s = carve(smem, n);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    for (long long cell = blockIdx.x; cell < a.cells; cell += gridDim.x) {
        // f00 of the cell
        for (int k = threadIdx.x; k < n; k += blockDim.x) s.f[k] = a.f00[cell * n + k];
        __syncthreads();
        if (warp == 0 && a.do_ee) {
            ee_substeps(a, s);
            for (int k = lane; k < n; k += 32) a.f00[cell * n + k] = s.f[k];
        }
        if (a.do_l1 || a.do_lm) {
            if (warp == 0) flm_reset(a, s, s.f);
            __syncthreads();
            if (a.if_tridiagonal) {
                if (a.planes_fp32) tridiagonal_chunks<float>(a, s, cell);
                else tridiagonal_chunks<double>(a, s, cell);
            } else {
                double* A = a.dense_ws + (long long)blockIdx.x * n * n;
                if (a.planes_fp32) dense_solves<float>(a, s, cell, A, s.chunk);
                else dense_solves<double>(a, s, cell, A, s.chunk);
            }
        }
        __syncthreads();
    }
}

__device__ __forceinline__ bool collided(const CollideArgs& a, int l, int m) {
    return l >= 1 && m <= a.mmax_coll && (l == 1 ? a.do_l1 : a.do_lm);
}

// Tridiagonal collision step, one warp per cell (1-warp CTAs, one CTA per
// cell), no CTA-wide barriers:
//   1. f00 e-e substeps, reset_coeff, and the Thomas pivots of every l --
//      c'_i and 1/(b_i - c'_{i-1} a_i), with b_0 kept for the reference's
//      d_0/b_0 -- one lane per l (TridiagonalSolve, def-Nmethods.cpp:152-159).
//   2. every collided plane of the cell: the row is loaded coalesced into
//      shared memory and both recurrences of TridiagonalSolve run with lanes
//      over momentum.  Each lane owns a contiguous run of p; the value
//      entering its run comes from a warp scan of the affine maps
//      d'_i = (d_i - a_i d'_{i-1}) id_i (forward) and x_i = d'_i - c'_i x_{i+1}
//      (backward); inside the run the lane applies the reference's recursion.
template <typename TP>
__global__ void __launch_bounds__(32) collide_warp_kernel(const CollideArgs a) {
    extern __shared__ double smem[];
    const int n = a.np;
    const int l0 = a.l0;
    const int lane = threadIdx.x & 31;
    TP* planes = reinterpret_cast<TP*>(a.planes);
    const bool solve = a.do_l1 || a.do_lm;
    Smem s = carve(smem, n);
    double* cp = s.chunk;                    // [l0][n]
    double* idv = cp + (size_t)l0 * n;       // [l0][n]
    double* row = idv + (size_t)l0 * n;      // [n]
    const int E = (n + 31) >> 5;
    const int rb = min(lane * E, n), re = min(rb + E, n);

    for (long long cell = blockIdx.x; cell < a.cells; cell += gridDim.x) {
        for (int k = lane; k < n; k += 32) s.f[k] = a.f00[cell * n + k];
        __syncwarp();
        if (a.do_ee) {
            ee_substeps(a, s);
            for (int k = lane; k < n; k += 32) a.f00[cell * n + k] = s.f[k];
        }
        if (!solve) continue;
        flm_reset(a, s, s.f);
        for (int l = 1 + lane; l <= l0; l += 32) {
            if (!(l == 1 ? a.do_l1 : a.do_lm)) continue;
            const double ll1 = l * ((-0.5) * (l + 1.0));
            double* cpl = cp + (size_t)(l - 1) * n;
            double* idl = idv + (size_t)(l - 1) * n;
            const double b0 = (l > 1 ? 0.0 : s.tri_b[0]) + (1.0 - ll1 * s.scat[0]);
            double cprev = s.tri_c[0] / b0;
            cpl[0] = cprev;
            idl[0] = b0;
            for (int i = 1; i < n; ++i) {
                const double bi = s.tri_b[i] + (1.0 - ll1 * s.scat[i]);
                const double id = 1.0 / (bi - cprev * s.tri_a[i]);
                cprev = s.tri_c[i] * id;
                cpl[i] = cprev;
                idl[i] = id;
            }
        }
        __syncwarp();
        const double* tri_a = s.tri_a;
        for (int q = 0; q < a.nplanes; ++q) {
            const int l = a.plane_l[q], m = a.plane_m[q];
            if (!collided(a, l, m)) continue;
            const double* cpl = cp + (size_t)(l - 1) * n;
            const double* idl = idv + (size_t)(l - 1) * n;
            TP* g = planes + (long long)q * a.pstride + cell * n;
            for (int k = lane; k < n; k += 32) row[k] = (double)g[k] + ref_at<TP>(a, q, k);
            __syncwarp();
            // forward: compose this lane's maps x -> A x + B over [rb, re)
            double A = 1.0, B = 0.0;
            for (int i = rb; i < re; ++i) {
                double Ai, Bi;
                if (i == 0) { Ai = 0.0; Bi = row[0] / idl[0]; }
                else { Ai = -(tri_a[i] * idl[i]); Bi = row[i] * idl[i]; }
                B = Ai * B + Bi;
                A = Ai * A;
            }
            // inclusive scan of the maps over the lanes (earlier lanes first)
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const double Ap = __shfl_up_sync(kFull, A, off), Bp = __shfl_up_sync(kFull, B, off);
                if (lane >= off) { B = A * Bp + B; A = A * Ap; }
            }
            double din = __shfl_up_sync(kFull, B, 1);   // d' just before this lane's run
            if (rb < re) {
                double d = din;
                for (int i = rb; i < re; ++i) {
                    if (i == 0) d = row[0] / idl[0];
                    else d = (row[i] - d * tri_a[i]) * idl[i];
                    row[i] = d;
                }
            }
            __syncwarp();
            // backward: x_i = d'_i - c'_i x_{i+1}, x_{n-1} = d'_{n-1}
            A = 1.0; B = 0.0;
            for (int i = re - 1; i >= rb; --i) {
                double Ai, Bi;
                if (i == n - 1) { Ai = 0.0; Bi = row[i]; }
                else { Ai = -cpl[i]; Bi = row[i]; }
                B = Ai * B + Bi;
                A = Ai * A;
            }
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const double Ap = __shfl_down_sync(kFull, A, off), Bp = __shfl_down_sync(kFull, B, off);
                if (lane + off < 32) { B = A * Bp + B; A = A * Ap; }
            }
            double xin = __shfl_down_sync(kFull, B, 1);  // x just after this lane's run
            if (rb < re) {
                double x = xin;
                for (int i = re - 1; i >= rb; --i) {
                    if (i == n - 1) x = row[i];
                    else x = row[i] - cpl[i] * x;
                    row[i] = x;
                }
            }
            __syncwarp();
            for (int k = lane; k < n; k += 32) g[k] = (TP)(row[k] - ref_at<TP>(a, q, k));
            __syncwarp();
        }
    }
}

// Tridiagonal collision step for nump <= 512, one CTA per cell (of many cells,
// launch_cell: the e-e substeps so and the rest on a warp a cell):
//   1. f00 e-e substeps and the coefficients of reset_coeff with one thread
//      per momentum point (two from 129 points on): f, the RK4 stages and the
//      point's velocity tables in registers, the three cumulative integrals as
//      warp scans joined through the warps' totals, neighbours through shared
//      memory, three barriers a slope.
//   2. the collided planes, by groups of G lanes (8 for rows of up to 64
//      points, 16 up to 112, else 32) so that a lane's run of p is 4 to 8
//      points long and a warp solves 32/G planes at once: a group takes units
//      of up to unit_planes planes of one l, forms that l's Thomas pivots for
//      each lane's run (lane_pivots; TridiagonalSolve, def-Nmethods.cpp:
//      152-159) and solves its planes one after the other, rows in registers,
//      the next plane's rows loading meanwhile.  Both recurrences of
//      TridiagonalSolve -- d'_i = (d_i - a_i d'_{i-1}) / (b_i - c'_{i-1} a_i)
//      forward, x_i = d'_i - c'_i x_{i+1} backward -- are affine maps of the
//      previous value.  Each lane composes its run, a scan over the group gives
//      the value entering the run, and the lane applies the recursion inside
//      its run.  The maps' multipliers depend on l only, so their composition
//      and scan are done once per unit and only the offsets are scanned per
//      plane.

// EE_isotropic_conserva::Getslope (def-FokkerPlanck.cpp:192-267): fh = C_ee(fin)
// X: a warp that holds no points takes the logarithm (cell_ee_log)
template <int PT, int W, int X>
__device__ __forceinline__ void cell_ee_slope(const CollideArgs& a, const CellSmem& s, const PointTab<PT>& t,
                                              const int k0, const double (&fin)[PT], double (&fh)[PT]) {
    const int n = a.np;
    double fm[PT], fp[PT], I4[PT], I2[PT], J1[PT], S4, S2;
    neighbours<PT, W>(s.f, k0, fin, fm, fp);
    const double fa = s.f[0], fb = s.f[1];
    cell_scans<PT, W, X>(t, fin, fm, fp, s.tot, I4, I2, J1, S4, S2);
    // the logarithm of the whole cell on the last warp (the first has the fit below): every warp
    // of its own would spend as many FP64 instructions on it as on all the rest of the slope
    if (X == 0 && (int)threadIdx.x >= 32 * (W - 1)) {
        const double norm = a.c_kpre * log_ee(4.0 * M_PI * S2, 4.0 * M_PI * S4, a.density_np);
        if ((threadIdx.x & 31) == 0) s.one[0] = norm;
    }
    // flux G_n; the first NB cells use the parabolic fit near v = 0
    double G[PT], Gm[PT], Gp[PT];
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (k0 + j < a.NB) {
            const double f00 = mul_rn(fma_rn(-fb, t.r, fa), t.inv1r), df = sub_rn(fb, f00);
            const double i2s = fma_rn(df, t.B2[j], mul_rn(f00, t.A2[j]));
            const double i4s = fma_rn(df, t.B4[j], mul_rn(f00, t.A4[j]));
            G[j] = fma_rn(fin[j], i4s, mul_rn(fma_rn(t.U3[j], fin[j], mul_rn(-3.0, i2s)), J1[j]));
        } else {
            const double i2 = mul_rn(-3.0, mul_rn(I2[j], J1[j]));
            G[j] = fma_rn(fma_rn(t.U3[j], J1[j], I4[j]), fin[j], i2);
        }
    }
    neighbours<PT, W, X>(s.g, k0, G, Gm, Gp);
    const double norm = s.one[0];
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        const int k = k0 + j;
        // D_k = (G_k - G_{k+1}) P_k for k < n-1, D_{n-1} = G_{n-1}
        const double D = k < n - 1 ? mul_rn(sub_rn(G[j], Gp[j]), t.Pn[j]) : G[j];
        const double v = k == 0 ? fma_rn(-G[j], t.two_v0s, -D) : fma_rn(sub_rn(Gm[j], G[j]), t.Pm[j], -D);
        fh[j] = mul_rn(mul_rn(v, t.Qn[j]), norm);
    }
}

// the collided planes of the cell over the CTA's groups of G lanes: units in
// order of falling l, group g takes units g, g + groups, ...
template <typename TP, int G, int R>
__device__ __forceinline__ void cell_solves(const CollideArgs& a, const TriRows& s, const long long cell) {
    constexpr int kSteps = G == 8 ? 3 : (G == 16 ? 4 : 5);
    const int n = a.np;
    const int gl = threadIdx.x & (G - 1);
    const int ng = blockDim.x / G;
    TP* planes = reinterpret_cast<TP*>(a.planes);
    const int i0 = gl * R;   // first p of this lane's run
    const int C = a.unit_planes;
    auto nplanes_of = [&](int l) { return collided(a, l, 0) ? 1 + 2 * min(min(l, a.m0), a.mmax_coll) : 0; };
    // this group's unit: k-th of order l; l = 0: none left
    int l = a.l0, k = threadIdx.x / G;
    auto settle = [&]() {
        while (l >= 1) {
            const int u = (nplanes_of(l) + C - 1) / C;
            if (k < u) return;
            k -= u;
            --l;
        }
        l = 0;
    };
    // the planes of one l split evenly over its units
    auto split = [&](int& first, int& count) {
        const int nq = nplanes_of(l), u = (nq + C - 1) / C;
        first = (int)((long long)nq * k / u);
        count = (int)((long long)nq * (k + 1) / u) - first;
    };
    // a lane's run in the widest pieces that divide it, where the rows start on such a boundary and are whole numbers
    // of them: 8-byte accesses 64 bytes apart (128 points) take a tag look-up for every second lane (5000 cells of 128
    // points in runs of 8, 48 planes, the planes' call alone: 0.266 -> 0.217 ms)
    constexpr int VW = R * sizeof(TP) % 16 == 0 ? 16 / (int)sizeof(TP) : (R % 2 == 0 ? 2 : 1);
    struct alignas(VW * sizeof(TP)) Pack { TP v[VW]; };
    const bool vec = n % VW == 0 && ((reinterpret_cast<uintptr_t>(planes) | (uintptr_t)(a.pstride * sizeof(TP))) & (sizeof(Pack) - 1)) == 0;
    double ta[R];
#pragma unroll
    for (int e = 0; e < R; ++e) ta[e] = (i0 + e < n) ? s.a[i0 + e] : 0.0;
    settle();
    while (__any_sync(kFull, l >= 1)) {
        int j0 = 0, cnt = 0;
        if (l >= 1) split(j0, cnt);
        const int most = __reduce_max_sync(kFull, cnt);
        const long long q0 = l >= 1 ? (long long)a.plane_of[l * (a.m0 + 1)] + j0 : 0;
        TP* g = planes + q0 * a.pstride + cell * n + i0;
        // rows as stored: the next plane's loads stay in flight during this plane's solve
        TP raw[R];
        auto load = [&](int b) {
            if (VW > 1 && vec) {
#pragma unroll
                for (int e = 0; e < R; e += VW) {
                    Pack v{};
                    if (b < cnt && i0 + e < n) v = *reinterpret_cast<const Pack*>(g + b * a.pstride + e);
#pragma unroll
                    for (int w = 0; w < VW; ++w) raw[e + w] = v.v[w];
                }
                return;
            }
#pragma unroll
            for (int e = 0; e < R; ++e) raw[e] = (b < cnt && i0 + e < n) ? g[b * a.pstride + e] : TP(0);
        };
        load(0);
        // per-l constants: pivots of this lane's run and the scan multipliers
        double id[R], cp[R], Af[kSteps], Ab[kSteps];
        lane_pivots<G, R>(s, l >= 1 ? l : 1, n, i0, cp, id);
        {
            double A = 1.0, B = 1.0;
#pragma unroll
            for (int e = 0; e < R; ++e) {
                const int i = i0 + e;
                if (i < n) A = (i == 0) ? 0.0 : A * (-(ta[e] * id[e]));
            }
#pragma unroll
            for (int e = R - 1; e >= 0; --e) {
                const int i = i0 + e;
                if (i < n) B = (i == n - 1) ? 0.0 : B * (-cp[e]);
            }
#pragma unroll
            for (int t = 0, off = 1; t < kSteps; ++t, off <<= 1) {
                const double Ap = __shfl_up_sync(kFull, A, off, G);
                const double Bp = __shfl_down_sync(kFull, B, off, G);
                Af[t] = gl >= off ? A : 0.0;
                Ab[t] = gl + off < G ? B : 0.0;
                if (gl >= off) A *= Ap;
                if (gl + off < G) B *= Bp;
            }
        }
        for (int b = 0; b < most; ++b) {
            double cur[R];
#pragma unroll
            for (int e = 0; e < R; ++e) cur[e] = (double)raw[e];
            const float* rp = (b < cnt) ? ref_row<TP>(a, q0 + b) : nullptr;
            if (rp) {   // the plane's profile (FP32 planes)
#pragma unroll
                for (int e = 0; e < R; ++e)
                    if (i0 + e < n) cur[e] += (double)__ldg(rp + i0 + e);
            }
            if (b + 1 < most) load(b + 1);
            // forward: run offset, scan, recursion inside the run
            double B = 0.0;
#pragma unroll
            for (int e = 0; e < R; ++e) B = mul_rn(fma_rn(-B, ta[e], cur[e]), id[e]);   // a_0 = 0; beyond the row nothing reads it
#pragma unroll
            for (int t = 0, off = 1; t < kSteps; ++t, off <<= 1) B = fma_rn(Af[t], __shfl_up_sync(kFull, B, off, G), B);
            double d = __shfl_up_sync(kFull, B, 1, G);
            if (gl == 0) d = 0.0;
#pragma unroll
            for (int e = 0; e < R; ++e) {
                if (i0 + e < n) d = mul_rn(fma_rn(-d, ta[e], cur[e]), id[e]);
                cur[e] = i0 + e < n ? d : 0.0;
            }
            // backward: x_{n-1} = d'_{n-1}; c'_{n-1} = 0 and the points beyond are zero
            B = 0.0;
#pragma unroll
            for (int e = R - 1; e >= 0; --e) B = fma_rn(-cp[e], B, cur[e]);
#pragma unroll
            for (int t = 0, off = 1; t < kSteps; ++t, off <<= 1) B = fma_rn(Ab[t], __shfl_down_sync(kFull, B, off, G), B);
            double x = __shfl_down_sync(kFull, B, 1, G);
            if (gl == G - 1) x = 0.0;
            TP* o = g + b * a.pstride;
#pragma unroll
            for (int e = R - 1; e >= 0; --e) {
                x = fma_rn(-cp[e], x, cur[e]);
                cur[e] = rp && i0 + e < n ? sub_rn(x, (double)__ldg(rp + i0 + e)) : x;
                if (!(VW > 1 && vec) && b < cnt && i0 + e < n) o[e] = (TP)cur[e];
            }
            if (VW > 1 && vec) {
#pragma unroll
                for (int e = 0; e < R; e += VW) {
                    Pack v;
#pragma unroll
                    for (int w = 0; w < VW; ++w) v.v[w] = (TP)cur[e + w];
                    if (b < cnt && i0 + e < n) *reinterpret_cast<Pack*>(o + e) = v;
                }
            }
        }
        k += ng;
        settle();
    }
}

// RK4 substeps of Explicit_EC_FP::loop (RungeKutta4_ee::advance,
// def-FokkerPlanck.cpp:518-553) on a thread's points of the cell's f00
template <int PT, int W, int X>
__device__ __forceinline__ void cell_ee(const CollideArgs& a, const StepP& sp, const CellSmem& s, const PointTab<PT>& t,
                                        const int k0, double (&f)[PT]) {
    const double h = sp.hsub;
    for (int sub = 0; sub < sp.nsub; ++sub) {
        double f0[PT], f1[PT], fh[PT];
#pragma unroll
        for (int j = 0; j < PT; ++j) { f0[j] = f[j]; f1[j] = f[j]; }
        // one call site of the slope for the four stages
        for (int st = 0; st < 4; ++st) {
            cell_ee_slope<PT, W, X>(a, s, t, k0, f1, fh);
            const double w = st < 2 ? 0.5 * h : (st == 2 ? h : h / 6.0);
            const double u = st == 1 ? 2.0 / 3.0 : (st == 3 ? 1.0 : 1.0 / 3.0);
#pragma unroll
            for (int j = 0; j < PT; ++j) {
                const double d = mul_rn(fh[j], w);
                f1[j] = add_rn(f0[j], d);
                f[j] = fma_rn(d, u, f[j]);
            }
        }
    }
}

// the logarithms of all its slopes, on a warp of their own
template <int W>
__device__ __forceinline__ void cell_ee_log(const CollideArgs& a, const StepP& sp, const CellSmem& s) {
    for (int i = 0; i < 4 * sp.nsub; ++i) {
        warps_sync<W + 1, 2>();
        double S4 = 0.0, S2 = 0.0;
#pragma unroll
        for (int w = 0; w < W; ++w) { S4 += s.tot[w]; S2 += s.tot[16 + w]; }
        const double norm = a.c_kpre * log_ee(4.0 * M_PI * S2, 4.0 * M_PI * S4, a.density_np);
        if ((threadIdx.x & 31) == 0) s.one[0] = norm;
        warps_sync<W + 1, 3>();
    }
}

// Implicit_FLM_step::reset_coeff (def-FokkerPlanck.cpp:808-939), tridiagonal
// part: the coefficients of the cell in units of the logarithms and moments
struct CoeffP {
    double lnee, zlnei, density, scale, kDt;
};
__device__ __forceinline__ CoeffP coeff_params(const CollideArgs& a, const StepP& sp, const double lnee,
                                               const double zlnei, const double density) {
    return CoeffP{lnee, zlnei, density, (-1.0) * lnee * a.kpre * sp.Dt, a.kpre * sp.Dt};
}
// ... at point k, from its integrals I2, I0, J_{-1}; U3: v^3
__device__ __forceinline__ void point_coeffs(const CollideArgs& a, const CoeffP& c, const TriRows& tri, const int k,
                                             const double f, const double I2, const double I0, const double J1m,
                                             const double U3) {
    const double* vr = a.vr;
    const double v = vr[k];
    double i2 = I2 * (4.0 * M_PI);
    i2 /= v * v;
    const double i0 = I0 * (4.0 * M_PI);
    const double j1m = J1m * (4.0 * M_PI * v);
    const double t1 = add_rn(i0, fma_rn(2.0, j1m, -i2) / 3.0);
    const double t2 = add_rn(i2, j1m) / 3.0;
    double sc = fma_rn(c.zlnei, c.density, (k == 0) ? 0.0 : mul_rn(t1, c.lnee));
    sc /= U3;
    sc *= c.kDt;
    tri.scat[k] = sc;
    double ta = 0.0, tb = 0.0, tc = 0.0;
    if (k == 0) {
        tb = 8.0 * M_PI * f * c.scale;
    } else if (k < a.np - 1) {
        const double vp = vr[k + 1], vm = vr[k - 1];
        const double IvDnDm1 = 1.0 / (v * 0.5 * (vp - vm) * (v - vm));
        const double IvDnDp1 = 1.0 / (v * 0.5 * (vp - vm) * (vp - v));
        const double Ivsq2Dn = 1.0 / (v * v * (vp - vm));
        const double t1s = mul_rn(t1, Ivsq2Dn);
        tb = mul_rn(fma_rn(-t2, add_rn(IvDnDm1, IvDnDp1), mul_rn(8.0 * M_PI, f)), c.scale);
        ta = mul_rn(fma_rn(t2, IvDnDm1, -t1s), c.scale);
        tc = mul_rn(fma_rn(t2, IvDnDp1, t1s), c.scale);
    }
    tri.a[k] = ta; tri.b[k] = tb; tri.c[k] = tc;
}

// W: the warps that hold the row, PT points a thread; CW: the CTA's.  Of the CTA's other warps one takes the slopes'
// logarithms, all join for the coefficients (a point a thread, whose divisions are a chain each) and the solves.
template <typename TP, int G, int R, int PT, int W, int CW>
__device__ __forceinline__ void collide_cell(const CollideArgs& a, const long long cell, double* smem) {
    const int n = a.np;
    constexpr int pts = PT * 32 * W, X = CW > W ? 1 : 0;
    const CellSmem s = carve_cell(smem, n, pts);
    if (X && threadIdx.x >= 32 * W) {
        if (a.do_ee && threadIdx.x < 32 * (W + 1)) cell_ee_log<W>(a, step_params(a), s);
    } else {
        const int k0 = PT * (int)threadIdx.x;
        PointTab<PT> t;
        load_tab<PT>(a, k0, t);
        const StepP sp = step_params(a);
        double f[PT];
#pragma unroll
        for (int j = 0; j < PT; ++j) f[j] = k0 + j < n ? a.f00[cell * n + k0 + j] : 0.0;
        if (threadIdx.x == 0) { s.f[-1] = 0.0; s.f[pts] = 0.0; s.g[-1] = 0.0; s.g[pts] = 0.0; }
        if (a.do_ee) {
            cell_ee<PT, W, X>(a, sp, s, t, k0, f);
#pragma unroll
            for (int j = 0; j < PT; ++j)
                if (k0 + j < n) a.f00[cell * n + k0 + j] = f[j];
        }
        if (a.do_l1 || a.do_lm) {
            double fm[PT], fp[PT], I2[PT], I0[PT], J1m[PT], S4, S2;
            neighbours<PT, W>(s.f, k0, f, fm, fp);
            cell_scans<PT, W>(t, f, fm, fp, s.tot, I2, I0, J1m, S4, S2);
            const double temperature = S4 * (4.0 * M_PI), density = S2 * (4.0 * M_PI);
            if ((int)threadIdx.x >= 32 * (W - 1)) {
                const double l = log_ee(density, temperature, a.density_np);
                if ((threadIdx.x & 31) == 0) s.one[0] = l;
            }
            if (threadIdx.x < 32) {
                const double l = zlog_ei(density, temperature, a.density_np, a.Zeta);
                if (threadIdx.x == 0) { s.one[1] = l; s.one[2] = density; }
            }
            if constexpr (CW > W) {
#pragma unroll
                for (int j = 0; j < PT; ++j)
                    if (k0 + j < n) {
                        s.tri.a[k0 + j] = I2[j]; s.tri.b[k0 + j] = I0[j]; s.tri.c[k0 + j] = J1m[j]; s.tri.scat[k0 + j] = f[j];
                    }
            } else {
                __syncthreads();
                const CoeffP c = coeff_params(a, sp, s.one[0], s.one[1], density);
#pragma unroll
                for (int j = 0; j < PT; ++j)
                    if (k0 + j < n) point_coeffs(a, c, s.tri, k0 + j, f[j], I2[j], I0[j], J1m[j], t.U3[j]);
            }
        }
    }
    if (!a.do_l1 && !a.do_lm) return;
    __syncthreads();
    if constexpr (CW > W) {
        const int k = threadIdx.x;
        const CoeffP c = coeff_params(a, step_params(a), s.one[0], s.one[1], s.one[2]);
        if (k < n) point_coeffs(a, c, s.tri, k, s.tri.scat[k], s.tri.a[k], s.tri.b[k], s.tri.c[k], __ldg(a.U3 + k));
        __syncthreads();
    }
    cell_solves<TP, G, R>(a, s.tri, cell);
}

// The coefficients and the solves of one cell on one warp: virtual warp v of
// the CTA form is this warp's v-th sweep, with the sums in the same order, so
// that the results have its bits.
template <typename TP, int G, int R, int PT, int V>
__device__ __forceinline__ void solve_cell(const CollideArgs& a, const long long cell, double* smem) {
    const int n = a.np;
    const int lane = threadIdx.x & 31;
    TriRows tri;
    tri.a = smem; tri.b = smem + n; tri.c = smem + 2 * n; tri.scat = smem + 3 * n;
    const StepP sp = step_params(a);
    double f[V][PT];
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const int k = PT * (32 * v + lane) + j;
            f[v][j] = k < n ? a.f00[cell * n + k] : 0.0;
        }
    double I2[V][PT], I0[V][PT], J1m[V][PT], r2[V], r0[V], r1[V], T2[V], T0[V], T1[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        double lo = __shfl_up_sync(kFull, f[v][PT - 1], 1), hi = __shfl_down_sync(kFull, f[v][0], 1);
        const double below = v > 0 ? __shfl_sync(kFull, f[v > 0 ? v - 1 : 0][PT - 1], 31) : 0.0;
        const double over = v + 1 < V ? __shfl_sync(kFull, f[v + 1 < V ? v + 1 : 0][0], 0) : 0.0;
        if (lane == 0) lo = below;
        if (lane == 31) hi = over;
        double s2 = 0.0, s0 = 0.0, s1 = 0.0;
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const int k = PT * (32 * v + lane) + j;
            const bool in = k < n, up = k + 1 < n;
            const double fm = j > 0 ? f[v][j > 0 ? j - 1 : 0] : lo, fp = j + 1 < PT ? f[v][j + 1 < PT ? j + 1 : 0] : hi;
            I2[v][j] = fma_rn(in ? __ldg(a.U4 + k) : 0.0, f[v][j], mul_rn(in ? __ldg(a.U4m1 + k) : 0.0, fm));
            I0[v][j] = fma_rn(in ? __ldg(a.U2 + k) : 0.0, f[v][j], mul_rn(in ? __ldg(a.U2m1 + k) : 0.0, fm));
            J1m[v][j] = fma_rn(up ? __ldg(a.U1 + k + 1) : 0.0, fp, mul_rn(up ? __ldg(a.U1m1 + k + 1) : 0.0, f[v][j]));
            s2 += I2[v][j]; s0 += I0[v][j]; s1 += J1m[v][j];
        }
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double u2 = __shfl_up_sync(kFull, s2, off), u0 = __shfl_up_sync(kFull, s0, off);
            const double u1 = __shfl_down_sync(kFull, s1, off);
            if (lane >= off) { s2 += u2; s0 += u0; }
            if (lane + off < 32) s1 += u1;
        }
        T2[v] = __shfl_sync(kFull, s2, 31);
        T0[v] = __shfl_sync(kFull, s0, 31);
        T1[v] = __shfl_sync(kFull, s1, 0);
        r2[v] = __shfl_up_sync(kFull, s2, 1);
        r0[v] = __shfl_up_sync(kFull, s0, 1);
        r1[v] = __shfl_down_sync(kFull, s1, 1);
        if (lane == 0) { r2[v] = 0.0; r0[v] = 0.0; }
        if (lane == 31) r1[v] = 0.0;
    }
    double S2 = 0.0, S0 = 0.0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        double b1 = 0.0;
#pragma unroll
        for (int w = v + 1; w < V; ++w) b1 += T1[w];
        r2[v] += S2; r0[v] += S0; r1[v] += b1;
        S2 += T2[v]; S0 += T0[v];
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            r2[v] += I2[v][j]; I2[v][j] = r2[v];
            r0[v] += I0[v][j]; I0[v][j] = r0[v];
        }
#pragma unroll
        for (int j = PT - 1; j >= 0; --j) { r1[v] += J1m[v][j]; J1m[v][j] = r1[v]; }
    }
    const double temperature = S2 * (4.0 * M_PI), density = S0 * (4.0 * M_PI);
    const CoeffP c = coeff_params(a, sp, log_ee(density, temperature, a.density_np),
                                  zlog_ei(density, temperature, a.density_np, a.Zeta), density);
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const int k = PT * (32 * v + lane) + j;
            if (k < n) point_coeffs(a, c, tri, k, f[v][j], I2[v][j], I0[v][j], J1m[v][j], __ldg(a.U3 + k));
        }
    __syncwarp();
    cell_solves<TP, G, R>(a, tri, cell);
}

// What it measured (B200, the collision launch, one cell a warp before -> now): 256 cells of 128 points, l0 = 1, ten e-e
// substeps 0.21 -> 0.10 ms for the three calls of a step; 384 cells of 432 points, l0 = 31 (the staged-chunk kernel
// before) 0.88 -> 0.2 ms; 512 uneven 1D problems 9.0 -> 7.2 ms a step.  Long e-e runs on few cells wait on the slope's
// three barriers and its logarithm; for many cells see collide_solve_kernel.
template <typename TP, int K, bool MANY>
__global__ void __launch_bounds__(32 * cell_warps(K, MANY), form_blocks(K, MANY)) collide_cell_kernel(const CollideArgs a) {
    extern __shared__ double smem[];
    for (long long cell = blockIdx.x; cell < a.cells; cell += gridDim.x) {
        collide_cell<TP, form_lanes(K), form_run(K), form_points(K), form_warps(K), cell_warps(K, MANY)>(a, cell, smem);
        __syncthreads();
    }
}

// The e-e substeps alone, for more cells than a wave: without the solves' registers 18 to 20 warps an SM of one thread a
// point, 15 or 16 of two (ee_blocks).
// 20000 cells, one substep, in the kernel above -> here: 96 points 169 -> 162 us, 128 228 -> 198, 257 877 -> 372 (two
// CTAs an SM for one); with the joins' counts known to the compiler 154, 189, 282.
template <int K>
__global__ void __launch_bounds__(32 * form_warps(K), ee_blocks(K)) collide_ee_kernel(const CollideArgs a) {
    extern __shared__ double smem[];
    constexpr int PT = form_points(K);
    const int n = a.np, pts = PT * (int)blockDim.x, k0 = PT * (int)threadIdx.x;
    const CellSmem s = carve_cell(smem, n, pts);
    PointTab<PT> t;
    load_tab<PT>(a, k0, t);
    const StepP sp = step_params(a);
    if (threadIdx.x == 0) { s.f[-1] = 0.0; s.f[pts] = 0.0; s.g[-1] = 0.0; s.g[pts] = 0.0; }
    for (long long cell = blockIdx.x; cell < a.cells; cell += gridDim.x) {
        double f[PT];
#pragma unroll
        for (int j = 0; j < PT; ++j) f[j] = k0 + j < n ? a.f00[cell * n + k0 + j] : 0.0;
        cell_ee<PT, form_warps(K), 0>(a, sp, s, t, k0, f);
#pragma unroll
        for (int j = 0; j < PT; ++j)
            if (k0 + j < n) a.f00[cell * n + k0 + j] = f[j];
    }
}

// Coefficients and solves of many cells, one warp a cell: 16 cells an SM under way where CTAs of their own leave 2 to 8,
// most of whose lanes wait for the one that has the plane.  collide_f1 alone, l0 = 1, 20000 cells, a CTA a cell -> here:
// 64 points 150 -> 96 us, 128 289 -> 101, 257 1161 -> 250; a whole collision step of 96 points 289 -> 237.  Weibel (16384
// cells of 96 points, 48 planes), the whole step 3.55 -> 3.47 ms, FP32 split 2.68 -> 2.61.
template <typename TP, int K>
__global__ void __launch_bounds__(32, solve_blocks(K)) collide_solve_kernel(const CollideArgs a) {
    extern __shared__ double smem[];
    for (long long cell = blockIdx.x; cell < a.cells; cell += gridDim.x) {
        solve_cell<TP, form_lanes(K), form_run(K), form_points(K), form_warps(K)>(a, cell, smem);
        __syncwarp();
    }
}

// batched form: work item = (problem, cell); the problems share the form
template <typename TP, int K>
__global__ void __launch_bounds__(32 * form_warps(K), form_blocks(K, true)) collide_cell_batch_kernel(const CollideBatch b) {
    extern __shared__ double smem[];
    __shared__ CollideArgs a;
    static_assert(sizeof(CollideArgs) % 4 == 0, "copied word by word");
    for (long long it = blockIdx.x; it < b.nitems; it += gridDim.x) {
        const int2 w = b.items[it];
        const int* src = reinterpret_cast<const int*>(b.probs + w.x);
        for (int i = threadIdx.x; i < (int)(sizeof(CollideArgs) / 4); i += blockDim.x) reinterpret_cast<int*>(&a)[i] = src[i];
        __syncthreads();
        collide_cell<TP, form_lanes(K), form_run(K), form_points(K), form_warps(K), form_warps(K)>(a, (long long)w.y, smem);
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_ee_implicit(const CollideArgs& a, cudaStream_t st) {
    const size_t smem = ((size_t)kSmemArrays * a.np + kSmemScalars) * sizeof(double);
    {
        const cudaError_t e = ensure_dyn_smem((const void*)ee_implicit_kernel, smem);
        if (e != cudaSuccess) return e;
    }
    const long long blocks = a.cells < (1ll << 30) ? a.cells : (1ll << 30);
    ee_implicit_kernel<<<(unsigned)blocks, 32, smem, st>>>(a);
    return cudaGetLastError();
}

size_t collide_smem_bytes(int np, int chunk, int if_tridiagonal) {
    size_t base = ((size_t)kSmemArrays * np + kSmemScalars) * sizeof(double);
    size_t extra;
    if (if_tridiagonal) extra = (size_t)chunk * 2 * (np + 1) * sizeof(double);
    else extra = ((size_t)np + 2 + (size_t)(kCollideThreads / 32) * 6 * np) * sizeof(double);
    return base + extra;
}

int collide_max_chunk(int np, size_t smem_budget) {
    size_t base = ((size_t)kSmemArrays * np + kSmemScalars) * sizeof(double);
    if (smem_budget <= base) return 0;
    size_t per = (size_t)2 * (np + 1) * sizeof(double);
    return (int)((smem_budget - base) / per);
}

int collide_threads() { return kCollideThreads; }

cudaError_t launch_collide(const CollideArgs& a, cudaStream_t st, size_t smem, int blocks) {
    {
        const cudaError_t e = ensure_dyn_smem((const void*)collide_kernel, smem);
        if (e != cudaSuccess) return e;
    }
    collide_kernel<<<blocks, kCollideThreads, smem, st>>>(a);
    return cudaGetLastError();
}

namespace {
size_t cell_smem(int np) {
    const int K = collide_form(np), pts = 32 * form_warps(K) * form_points(K);
    return cell_smem_doubles(np, pts) * sizeof(double);
}
}  // namespace

int collide_form(int np) {
    const int k = (np + 7) / 8;
    if (k <= 4) return 4;
    if (k <= 16) return (k + 1) / 2 * 2;
    return k <= 32 ? (k + 3) / 4 * 4 : (k + 7) / 8 * 8;
}
// Planes of one l a lane group takes at a time: as many as make the longest
// group's work shortest, a unit's pivots counted as three planes
int collide_unit_planes(int np, int l0, int m0, int mmax_coll, int do_l1, int do_lm, int warps) {
    if (np > 512) return 1;
    const int K = collide_form(np), groups = 32 * (warps ? warps : cell_warps(K, false)) / form_lanes(K);
    int best = 1, cost = 1 << 30;
    const int widest = 1 + 2 * std::min(std::min(l0, m0), mmax_coll);
    for (int C = 1; C <= widest; ++C) {
        int units = 0;
        for (int l = 1; l <= l0; ++l)
            if (l == 1 ? do_l1 : do_lm) units += (1 + 2 * std::min(std::min(l, m0), mmax_coll) + C - 1) / C;
        const int c = (units + groups - 1) / groups * (C + 3);
        if (c < cost) { cost = c; best = C; }
    }
    return best;
}

size_t collide_tri_smem_per_cell(int np, int l0) {
    if (np <= 512) return cell_smem(np);
    return ((size_t)kSmemArrays * np + kSmemScalars + 2 * (size_t)l0 * np + np) * sizeof(double);
}

namespace {
template <typename TP>
cudaError_t launch_cell(const CollideArgs& a0, cudaStream_t st, int blocks) {
    return with_form(collide_form(a0.np), [&](auto form) {
        constexpr int K = decltype(form)::value;
        CollideArgs a = a0;
        int planes = 0;   // that this call solves
        for (int l = 1; l <= a.l0; ++l)
            if (l == 1 ? a.do_l1 : a.do_lm) planes += 1 + 2 * std::min(std::min(l, a.m0), a.mmax_coll);
        const int groups = 32 * cell_warps(K, false) / form_lanes(K);
        // A CTA a cell leaves the lane groups that have no plane idle while the others solve, and only few cells are
        // resident.  A wave of such CTAs is as good as warps of their own (collide_solve_kernel) up to these numbers of
        // cells: one wave where most groups are idle, about one wave of the warps (one and a half with e-e substeps, which
        // then take a launch of their own) where all find a plane at most once, four beyond.  Both sides at 96 points, in
        // us, CTA / warp: one plane and e-e, 2400 cells 47 / 47, 8000 125 / 104; 16 planes 2400 cells 84 / 98, 8000
        // 231 / 219, 16000 455 / 408; 48 planes 2400 cells 168 / 215, 8000 481 / 461, 16000 901 / 811.
        const long long sms = sm_count(), wave = solve_blocks(K) * sms;
        const bool idle = a.do_ee || K > 32 ? 4 * planes <= groups : 5 * planes <= 3 * groups;
        const long long limit = idle ? form_blocks(K, true) * sms : planes > groups ? 4 * wave : a.do_ee ? 3 * wave / 2 : wave;
        const bool split = a.cells > limit, wide = a.cells > form_blocks(K, false) * sms;   // wide: more than a wave
        // (e-e alone on cells that only the many form's wave holds: 1000 cells of 96 points, 15 substeps, 208 -> 191 us)
        const bool in_wave = !planes && a.cells > ee_blocks(K) * sms && a.cells <= form_blocks(K, true) * sms;
        if (a.do_ee && !in_wave && (split || (!planes && wide))) {
            collide_ee_kernel<K><<<blocks, 32 * form_warps(K), cell_smem(a.np), st>>>(a);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess || !planes) return e;
            a.do_ee = 0;
        }
        if (split) {
            a.unit_planes = collide_unit_planes(a.np, a.l0, a.m0, a.mmax_coll, a.do_l1, a.do_lm, 1);
            collide_solve_kernel<TP, K><<<blocks, 32, 4 * sizeof(double) * a.np, st>>>(a);
            return cudaGetLastError();
        }
        if constexpr (form_blocks(K, true) > form_blocks(K, false)) {
            if (wide && (form_points(K) > 1 || planes <= kManyPlanes)) {
                collide_cell_kernel<TP, K, true><<<blocks, 32 * form_warps(K), cell_smem(a.np), st>>>(a);
                return cudaGetLastError();
            }
        }
        collide_cell_kernel<TP, K, false><<<blocks, 32 * cell_warps(K, false), cell_smem(a.np), st>>>(a);
        return cudaGetLastError();
    });
}
template <typename TP>
cudaError_t launch_cell_batch(const CollideBatch& b, int form, cudaStream_t st, size_t smem) {
    const long long blocks = b.nitems < (1ll << 30) ? b.nitems : (1ll << 30);
    if (blocks < 1) return cudaSuccess;
    return with_form(form, [&](auto f) {
        constexpr int K = decltype(f)::value;
        if constexpr (K <= 32) {   // a batch's rows have at most 256 points
            collide_cell_batch_kernel<TP, K><<<(unsigned)blocks, 32 * form_warps(K), smem, st>>>(b);
            return cudaGetLastError();
        }
        return cudaErrorInvalidValue;
    });
}

__global__ void clock_advance_batch_kernel(double* clocks, const double* dt, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) clocks[3 * i] += dt[i];
}
__global__ void clock_commit_batch_kernel(double* clocks, const int* collide, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && (!collide || collide[i])) { clocks[3 * i + 1] = clocks[3 * i]; clocks[3 * i + 2] = clocks[3 * i]; }
}
}  // namespace

cudaError_t launch_collide_batch(const CollideBatch& b, int form, int planes_fp32, size_t smem, cudaStream_t st) {
    return planes_fp32 ? launch_cell_batch<float>(b, form, st, smem) : launch_cell_batch<double>(b, form, st, smem);
}
cudaError_t launch_clock_advance(double* clocks, const double* dt, int n, cudaStream_t st) {
    clock_advance_batch_kernel<<<(n + 127) / 128, 128, 0, st>>>(clocks, dt, n);
    return cudaGetLastError();
}
cudaError_t launch_clock_commit(double* clocks, const int* collide, int n, cudaStream_t st) {
    clock_commit_batch_kernel<<<(n + 127) / 128, 128, 0, st>>>(clocks, collide, n);
    return cudaGetLastError();
}

cudaError_t launch_collide_tri(const CollideArgs& a, cudaStream_t st, int /*cells_per_cta*/, int blocks) {
    if (a.np <= 512) return a.planes_fp32 ? launch_cell<float>(a, st, blocks) : launch_cell<double>(a, st, blocks);
    const size_t smem = collide_tri_smem_per_cell(a.np, a.l0);
    if (a.planes_fp32) {
        const cudaError_t e = ensure_dyn_smem((const void*)collide_warp_kernel<float>, smem);
        if (e != cudaSuccess) return e;
        collide_warp_kernel<float><<<blocks, 32, smem, st>>>(a);
    } else {
        const cudaError_t e = ensure_dyn_smem((const void*)collide_warp_kernel<double>, smem);
        if (e != cudaSuccess) return e;
        collide_warp_kernel<double><<<blocks, 32, smem, st>>>(a);
    }
    return cudaGetLastError();
}

}  // namespace oshun
