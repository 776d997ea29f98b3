// Two-point pipelined RK4-stage kernel: Actions::Adv (OSHUN-1/def-Actions.cpp:73-94),
// or a part of it, on one stage input folded into the stage update of
// Runge_Kutta_4::advance_p1 (OSHUN-1/def-RK.cpp:110-145).  Rows may have any
// number of points up to what a CTA's consumers hold (points() and
// consumer_warps() below): 512 with m0 = 0; 640 (FP32: 896) with m0 = 1, 2; 320
// (640) with m0 = 3 to 6; 192 (384) with m0 = 7, 8.
//
// The launcher of vlasov.cu takes it for m0 = 0, for momentum rows that are
// no multiple of 16 bytes and for partial right-hand sides (the implicit-E
// actions); the one-point kernel of stage_pipe.cu keeps the full right-hand
// side of m0 >= 1.
//
// What it is bound by and what it measured (B200, one small step without
// collisions unless said; before -> now): m0 = 0 waits on memory latency and
// issues one barrier round trip a harmonic -- 8192 cells, l0 = 16, np = 256,
// FP64 1.40 -> 0.96 ms (the one-point kernel); rows of 75 points on 61 x 45
// cells, l0 = 5, m0 = 3, with collisions 1.48 -> 0.94 ms (the global-load
// kernel re-read every neighbour through L1); rows of 75 points, 4000 cells, l0 = 8,
// m0 = 0, two steps, one point a thread -> two: FP64 575 -> 340 us, FP32 577 -> 340
// (the global-load kernel 625 and 478: with one point a tile held 2 cells and
// copied as many neighbours; two points halve the threads of a cell); the RK2 actions on 64 x 48 cells,
// l0 = 8, m0 = 3, np = 96, with collisions 2.46 -> 0.95 ms (global loads).  The
// full right-hand side of m0 >= 3 on 16-byte rows is not taken: its registers
// leave 8 to 12 warps an SM here, and Weibel (128 x 128, l0 = m0 = 6, np = 96)
// took 5.7 to 6.9 ms a step against 3.56.
//
// Persistent CTAs walk tiles of `tx` consecutive cells of one y row.  One
// consumer thread owns two adjacent momentum points of one cell of every
// harmonic; half a warp holds 32 points, so a cell takes ceil(np/32)
// half-warps whatever np is.  Two points a thread share the products of
// coupling coefficients and fields, the coefficient loads and the barrier
// work, read the momentum rows in 16-byte (FP32: 8-byte) pieces and give
// every dependent FP64 chain a second, independent one; FP32 runs both points
// in one paired FMA (__ffma2_rn).
//
// A source row l adds to the target rows l-1, l and l+1, held in registers.
// Sources pass in (l, m) order; target (l-1, m-1) is complete once source
// (l, m) has passed, and is RK-updated and stored there and then, so row l+1
// takes over the registers of row l-1 entry by entry and about two rows are
// live instead of three.
//
// Two producer warps feed shared memory with bulk copies (cp.async.bulk),
// running ahead across tiles: one streams the sources -- the cells, their x
// neighbours and their y-1/y+1 cells, every momentum point, with the tile's
// six fields beside f00 -- into a ring of slots; the other streams the RK
// operands of each target (l, m) into a ring of their own.  Rows that are no
// multiple of 16 bytes come as the aligned spans that hold them (SHIFT), and
// a thread loads its two points of them one by one.  Copies complete on mbarriers, and every wait is bounded.
//
// The consumer warps share no barrier: each half-warp writes its sums of the
// current to shared memory and the last one of a cell to do so adds them in
// order and updates the cell's E and B.
//
// Couplings of source (l, m) at one momentum point, with G/H as in
// MakeGH/G00 (OSHUN-1/def-VlasovMax.cpp:496-535) and the reference's Dp ends
// (OSHUN-1/def-State.cpp:359-380):
//   E (def-VlasovMax.cpp:346-491): Ex G -> (l+1,m), Ex H -> (l-1,m),
//     Em G -> (l+1,m+1), Em H -> (l-1,m+1), Ep H -> (l-1,m-1),
//     Ep G -> (l+1,m-1), real part only into m = 0;
//   B (def-VlasovMax.cpp:597-644): (Bz+iBy)/2 f -> (l,m+1), -i m Bx f -> (l,m),
//     (Bz-iBy) f -> (l,m-1);
//   advection (def-VlasovMax.cpp:834-951): x -> (l+-1,m), y -> (l+-1,m+-1);
//   current (def-VlasovMax.cpp:680-745) from f10, f11; Ampere/Faraday
//   (def-VlasovMax.cpp:979-1035); CLEAN_LOW_PC (def-Actions.cpp:240-253).
#include <cstring>

#include "stage_async.cuh"

namespace oshun {
namespace {

constexpr int kMaxDepth = 12;                 // slots of either ring
constexpr int kMinSrc = 3, kMinTgt = 3;       // fewest slots a plan may have
constexpr int kJBuf = 8;                      // tiles whose current sums can be open at once (see consume_tile)
static_assert(kMaxDepth / 2 + 1 < kJBuf, "sets of current sums");

// a consumer warp's wait: when it runs out the whole warp reports and stops
// (the lanes decide together), so the code behind a wait has no failure path;
// the other warps' and the producers' waits end by their own limits
__device__ __forceinline__ void mbar_wait_or_exit(const uint32_t addr, const uint32_t parity, int* err,
                                                  const unsigned long long limit_ns) {
    if (__all_sync(kFull, mbar_hold(addr, parity))) return;
    const unsigned long long t0 = global_ns();
    while (!__all_sync(kFull, mbar_hold(addr, parity))) {
        if (__any_sync(kFull, global_ns() - t0 > limit_ns)) {
            if ((threadIdx.x & 31) == 0) atomicOr(err, 16);
            asm volatile("exit;");
        }
    }
}
// lane 0 arrives for its warp
__device__ __forceinline__ void warp_arrive(const uint32_t addr, const int lane) {
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "setp.eq.s32 P1, %1, 0;\n\t"
        "@P1 mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(addr),
        "r"(lane)
        : "memory");
}
// ---------------------------------------------------------------------------
// arithmetic on the two points of a thread.  V: a value per point; S: a
// factor common to both (FP32: the pair (s, s), so that products of factors
// stay in the paired form).  Every rounding is spelled out: the kernels of a
// single problem and of a batch give the same bits.
// ---------------------------------------------------------------------------
struct alignas(16) D2 {
    double x, y;
};
template <typename TS, int PT>
struct VecOf;
template <>
struct VecOf<double, 1> { using V = double; };
template <>
struct VecOf<double, 2> { using V = D2; };
template <>
struct VecOf<float, 1> { using V = float; };
template <>
struct VecOf<float, 2> { using V = float2; };
template <typename TS>
struct Arith;
template <>
struct Arith<double> { using S = double; };
template <>
struct Arith<float> { using S = float2; };
__device__ __forceinline__ double v_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double v_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double v_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double v_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ D2 v_mul(D2 a, D2 b) { return {__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)}; }
__device__ __forceinline__ D2 v_mul(double a, D2 b) { return {__dmul_rn(a, b.x), __dmul_rn(a, b.y)}; }
__device__ __forceinline__ D2 v_fma(D2 a, D2 b, D2 c) { return {__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y)}; }
__device__ __forceinline__ D2 v_fma(double a, D2 b, D2 c) { return {__fma_rn(a, b.x, c.x), __fma_rn(a, b.y, c.y)}; }
__device__ __forceinline__ D2 v_sub(D2 a, D2 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)}; }
__device__ __forceinline__ D2 v_add(D2 a, D2 b) { return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)}; }
__device__ __forceinline__ float v_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float v_mul(float2 a, float b) { return __fmul_rn(a.x, b); }
__device__ __forceinline__ float v_fma(float2 a, float b, float c) { return __fmaf_rn(a.x, b, c); }
__device__ __forceinline__ float v_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float v_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float v_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double s_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double s_neg(double a) { return -a; }
__device__ __forceinline__ float2 v_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 v_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 v_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 v_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 s_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 s_neg(float2 a) { return __fmul2_rn(a, make_float2(-1.f, -1.f)); }
__device__ __forceinline__ double bcast(double v) { return v; }
__device__ __forceinline__ float2 bcast(float v) { return make_float2(v, v); }
template <typename V>
constexpr bool kOne = std::is_same_v<V, double> || std::is_same_v<V, float>;   // one point a thread
// a thread's points from its first and second value (one point: the first)
template <typename V, typename T>
__device__ __forceinline__ V make_v(T a, T b) {
    if constexpr (kOne<V>) return a;
    else return V{a, b};
}
template <typename V>
__device__ __forceinline__ auto& first(V& v) {
    if constexpr (kOne<std::remove_const_t<V>>) return v;
    else return v.x;
}
template <typename V>
__device__ __forceinline__ auto second(const V& v) {
    if constexpr (kOne<V>) return V(0);
    else return v.y;
}
// a thread's points from shared memory; o2: from the first to the second.  A
// pair's address is aligned, except in rows that are no multiple of 16 bytes
// (SHIFT).
template <bool SHIFT, typename V, typename T>
__device__ __forceinline__ V ld_v(const T* p, const int o2) {
    if constexpr (kOne<V>) return *p;
    else if constexpr (SHIFT) return V{p[0], p[o2]};
    else return *reinterpret_cast<const V*>(p);
}
// sums of three and two products added to an accumulator.  FP64: the products
// summed first, so that the accumulators' chains stay one addition a source
// long; FP32: paired FMAs onto the accumulator.
template <typename V, typename S>
__device__ __forceinline__ V v_acc3(S a, V x, S b, V y, S c, V z, V acc) {
    if constexpr (std::is_same_v<S, double>) return v_add(acc, v_fma(a, x, v_fma(b, y, v_mul(c, z))));
    else return v_fma(a, x, v_fma(b, y, v_fma(c, z, acc)));
}
template <typename V, typename S>
__device__ __forceinline__ V v_acc2(S a, V x, S b, V y, V acc) {
    if constexpr (std::is_same_v<S, double>) return v_add(acc, v_fma(a, x, v_mul(b, y)));
    else return v_fma(a, x, v_fma(b, y, acc));
}

// coupling coefficients of one source, in pairs used together (16-byte loads)
enum : int { kExG = 0, kAxP, kExH, kAxM, kEmG, kAyPP, kEmH, kAyMP, kEpH, kAyMM, kEpG, kAyPM, kBm2, kGfac, kInvpax, kHp0 };
template <typename TS>
struct alignas(16) CoefS {
    typename Arith<TS>::S v[16];
};
constexpr uint32_t kCoefBytes = 128;
static_assert(sizeof(CoefS<double>) == kCoefBytes && sizeof(CoefS<float>) == kCoefBytes, "CoefS layout");
// entry i of a source's coefficients (b_m doubled: it multiplies half fields)
__host__ __device__ inline double coef_entry(const CoefLM& c, int i) {
    switch (i) {
        case kExG: return c.ex_g;
        case kAxP: return c.ax_p;
        case kExH: return c.ex_h;
        case kAxM: return c.ax_m;
        case kEmG: return c.em_g;
        case kAyPP: return c.ay_pp;
        case kEmH: return c.em_h;
        case kAyMP: return c.ay_mp;
        case kEpH: return c.ep_h;
        case kAyMM: return c.ay_mm;
        case kEpG: return c.ep_g;
        case kAyPM: return c.ay_pm;
        case kBm2: return 2.0 * c.b_m;
        case kGfac: return c.gfac;
        case kInvpax: return c.invpax;
        default: return c.hp0;
    }
}
template <typename S>
struct S2 {
    S a, b;
};
// the pair of coefficients i, i + 1 (i even)
__device__ __forceinline__ S2<double> coef2(const CoefS<double>* c, int i) {
    const double2 v = *reinterpret_cast<const double2*>(c->v + i);
    return {v.x, v.y};
}
__device__ __forceinline__ S2<float2> coef2(const CoefS<float>* c, int i) {
    const float4 v = *reinterpret_cast<const float4*>(c->v + i);
    return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}

// The stencil operands of one component in a slot: the thread's points, the
// cells beside, below and above them; pp: from c to the point above them (edge
// rule applied).
template <typename TS>
struct Ops {
    const TS *c, *xm, *xp, *ym, *yp;
};
// Where a thread finds them.  Rows of 16-byte multiples lie back to back
// (x-1, the tile's cells, x+1, then the cells of y-1 and y+1) and every
// thread's neighbours are the same distances away.  Other rows (SHIFT) are
// copied as the 16-byte aligned spans that hold them, each of the five pieces
// in a region of its own: the first element of a piece lies (A + q B) mod
// (16 bytes) behind its region's start, A and B the piece's first element and
// the planes' distance in elements, q the plane.
struct Nb {
    int ctr, pp;
    int o2;                   // from the first point to the second (SHIFT: 0 where the row ends between them)
    int x, ym, yp;            // from ctr: x-1 is -x, x+1 is +x (SHIFT: ym and yp are offsets in the slot)
    int xm, xp;               // SHIFT: offsets in the slot
    int ac, axm, axp, aym, ayp, b, bxm, bxp;   // SHIFT: A of each piece, B of the planes and of the x neighbours
    int p, p_1, p_m, p_p;     // momentum index of the points and of their outer neighbours (FP32 profile)
};
template <bool SHIFT, typename TS>
__device__ __forceinline__ Ops<TS> operands(const TS* sb, const Nb& nb, const int q) {
    if constexpr (!SHIFT) {
        const TS* c = sb + nb.ctr;
        return {c, c - nb.x, c + nb.x, c + nb.ym, c + nb.yp};
    } else {
        constexpr int kMask = 16 / (int)sizeof(TS) - 1;
        return {sb + nb.ctr + ((nb.ac + q * nb.b) & kMask), sb + nb.xm + ((nb.axm + q * nb.bxm) & kMask),
                sb + nb.xp + ((nb.axp + q * nb.bxp) & kMask), sb + nb.ym + ((nb.aym + q * nb.b) & kMask),
                sb + nb.yp + ((nb.ayp + q * nb.b) & kMask)};
    }
}

// per-thread constants of the coupling arithmetic
template <typename TS, typename V>
struct Th {
    typename Arith<TS>::S ex, ey, ez, bx, hby, hbz;   // fields of the cell (half By, Bz)
    V invp, vr;
    bool is0;               // the first point is p = 0: G = 0, H = f[1] hp0
};

// slope accumulators of one target row (I[0] is never used: m = 0 is real)
template <typename V, int MC>
struct Acc {
    V R[MC + 1], I[MC + 1];
};
template <typename TS, typename V, int MC>
__device__ __forceinline__ void acc_zero(Acc<V, MC>& a) {
#pragma unroll
    for (int m = 0; m <= MC; ++m) { a.R[m] = make_v<V>(TS(0), TS(0)); a.I[m] = make_v<V>(TS(0), TS(0)); }
}

// f[p-1] - f[p+1] of a thread's points: f the values, fm and fp the outer neighbours
template <typename V, typename T>
__device__ __forceinline__ V p_diff(const V f, const T fm, const T fp) {
    if constexpr (kOne<V>) return sub_rn(fm, fp);
    else return make_v<V>(sub_rn(fm, f.y), sub_rn(f.x, fp));
}
// the value one point above the first
template <typename V, typename T>
__device__ __forceinline__ T above(const V f, const T fp) {
    if constexpr (kOne<V>) return fp;
    else return f.y;
}

// stencils of one component of a source: value, G, H, x and y differences (times v)
template <typename TS, typename V, bool Y, bool SHIFT>
__device__ __forceinline__ void stencils(const Ops<TS> op, const Nb& nb, const Th<TS, V>& th, const V ipx,
                                         const typename Arith<TS>::S gfac, const typename Arith<TS>::S hp0,
                                         const TS* __restrict__ ref, V& f, V& G, V& H, V& dx, V& dy) {
    auto ld = [&](const TS* q) { return ld_v<SHIFT, V>(q, nb.o2); };
    f = ld(op.c);
    // below p = 0 lies another point of the slot: G and H there do not use it
    TS fm = op.c[-1], fp = op.c[nb.pp];
    dx = v_mul(v_sub(ld(op.xm), ld(op.xp)), th.vr);
    if constexpr (Y) dy = v_mul(v_sub(ld(op.ym), ld(op.yp)), th.vr);
    if constexpr (sizeof(TS) == 4) {
        // FP32 planes hold f - ref (the plane's momentum profile, if it keeps
        // one): the differences above act on the stored deviation alone, the
        // momentum stencil and the value on f
        if (ref) {
            f = v_add(f, make_v<V>(__ldg(ref + nb.p), __ldg(ref + nb.p_1)));
            fm = __fadd_rn(fm, __ldg(ref + nb.p_m));
            fp = __fadd_rn(fp, __ldg(ref + nb.p_p));
        }
    }
    const V d = p_diff(f, fm, fp);
    H = v_fma(f, ipx, d);
    G = v_fma(gfac, d, H);
    TS h0;
    if constexpr (sizeof(TS) == 8) h0 = mul_rn(above(f, fp), hp0);
    else h0 = mul_rn(above(f, fp), hp0.x);
    first(H) = th.is0 ? h0 : first(H);
    first(G) = th.is0 ? TS(0) : first(G);
}

// couplings of source (s, M), s >= 1, into target rows s-1 (A0), s (A1), s+1
// (A2).  Row s+1 first meets entry M+1 here (and entry 0 at M = 0), so those
// start from the product.
template <int MC, int M, bool SHIFT, typename TS, typename V>
__device__ __forceinline__ void couple_src(Acc<V, MC>& A0, Acc<V, MC>& A1, Acc<V, MC>& A2,
                                           const CoefS<TS>* __restrict__ c, const TS* __restrict__ sb, const int seg,
                                           const Nb& nb, const Th<TS, V>& th, const TS* __restrict__ ref,
                                           const int np, const int q) {
    using S = typename Arith<TS>::S;
    constexpr bool UP = M + 1 <= MC;
    constexpr bool DN = M >= 1;
    const S2<S> cg = coef2(c, kBm2), ch = coef2(c, kInvpax);   // (2 b_m, gfac), (invpax, hp0)
    const V ipx = v_mul(ch.a, th.invp);
    V fr, Gr, Hr, dxr, dyr, fi, Gi, Hi, dxi, dyi;
    stencils<TS, V, MC >= 1, SHIFT>(operands<SHIFT>(sb, nb, q), nb, th, ipx, cg.b, ch.b, ref, fr, Gr, Hr, dxr, dyr);
    if constexpr (DN)
        stencils<TS, V, true, SHIFT>(operands<SHIFT>(sb + seg, nb, q + 1), nb, th, ipx, cg.b, ch.b, ref ? ref + np : ref, fi, Gi,
                              Hi, dxi, dyi);
    // Ex and x advection: (s+1, M), (s-1, M)
    {
        const S2<S> g = coef2(c, kExG), h = coef2(c, kExH);
        const S eg = s_mul(g.a, th.ex), eh = s_mul(h.a, th.ex);
        if constexpr (DN) {
            A2.R[M] = v_acc2(eg, Gr, g.b, dxr, A2.R[M]);
            A2.I[M] = v_acc2(eg, Gi, g.b, dxi, A2.I[M]);
            A0.I[M] = v_acc2(eh, Hi, h.b, dxi, A0.I[M]);
        } else {
            A2.R[M] = v_fma(eg, Gr, v_mul(g.b, dxr));
        }
        A0.R[M] = v_acc2(eh, Hr, h.b, dxr, A0.R[M]);
    }
    if constexpr (UP) {
        // Em G -> (s+1, M+1), Em H -> (s-1, M+1), y advection, (Bz + iBy)/2 f -> (s, M+1)
        const S2<S> g = coef2(c, kEmG), h = coef2(c, kEmH);
        const S gy = s_mul(g.a, th.ey), gz = s_mul(g.a, th.ez);
        const S hy = s_mul(h.a, th.ey), hz = s_mul(h.a, th.ez);
        const S ngz = s_neg(gz), nhz = s_neg(hz);
        if constexpr (DN) {
            A2.R[M + 1] = v_fma(gy, Gr, v_fma(gz, Gi, v_mul(g.b, dyr)));
            A2.I[M + 1] = v_fma(gy, Gi, v_fma(ngz, Gr, v_mul(g.b, dyi)));
            A0.R[M + 1] = v_acc3(hy, Hr, hz, Hi, h.b, dyr, A0.R[M + 1]);
            A0.I[M + 1] = v_acc3(hy, Hi, nhz, Hr, h.b, dyi, A0.I[M + 1]);
            A1.R[M + 1] = v_acc2(th.hbz, fr, s_neg(th.hby), fi, A1.R[M + 1]);
            A1.I[M + 1] = v_acc2(th.hbz, fi, th.hby, fr, A1.I[M + 1]);
        } else {
            // an m = 0 source is real: its imaginary terms are zero
            A2.R[M + 1] = v_fma(gy, Gr, v_mul(g.b, dyr));
            A2.I[M + 1] = v_mul(ngz, Gr);
            A0.R[M + 1] = v_acc2(hy, Hr, h.b, dyr, A0.R[M + 1]);
            A0.I[M + 1] = v_fma(nhz, Hr, A0.I[M + 1]);
            A1.R[M + 1] = v_fma(th.hbz, fr, A1.R[M + 1]);
            A1.I[M + 1] = v_fma(th.hby, fr, A1.I[M + 1]);
        }
    }
    if constexpr (DN) {
        // Ep H -> (s-1, M-1), Ep G -> (s+1, M-1), y advection, -i M Bx f -> (s, M),
        // (Bz - iBy) f -> (s, M-1); only real parts into m = 0
        const S2<S> h = coef2(c, kEpH), g = coef2(c, kEpG);
        const S py = s_mul(h.a, th.ey), pz = s_mul(h.a, th.ez);
        const S qy = s_mul(g.a, th.ey), qz = s_mul(g.a, th.ez);
        const S cz = s_mul(cg.a, th.hbz), cy = s_mul(cg.a, th.hby);
        const S mb = s_mul(bcast(TS(M)), th.bx);
        A0.R[M - 1] = v_acc3(py, Hr, s_neg(pz), Hi, h.b, dyr, A0.R[M - 1]);
        A2.R[M - 1] = v_acc3(qy, Gr, s_neg(qz), Gi, g.b, dyr, A2.R[M - 1]);
        A1.R[M - 1] = v_acc2(cz, fr, cy, fi, A1.R[M - 1]);
        A1.R[M] = v_fma(mb, fi, A1.R[M]);
        A1.I[M] = v_fma(s_neg(mb), fr, A1.I[M]);
        if constexpr (M >= 2) {
            A0.I[M - 1] = v_acc3(py, Hi, pz, Hr, h.b, dyi, A0.I[M - 1]);
            A2.I[M - 1] = v_acc3(qy, Gi, qz, Gr, g.b, dyi, A2.I[M - 1]);
            A1.I[M - 1] = v_acc2(cz, fi, s_neg(cy), fr, A1.I[M - 1]);
        }
    }
}

// couplings of the f00 source into row 1 (A, from zero); G00 at p = 0 from
// the extrapolated f00(p=0) (OSHUN-1/def-VlasovMax.cpp:520-535)
template <int MC, bool SHIFT, typename TS, typename V>
__device__ __forceinline__ void couple_f00(Acc<V, MC>& A, const CoefS<TS>* __restrict__ c,
                                           const Ops<double> op, const Nb& nb, const Th<TS, V>& th,
                                           const double g00_s, const double g00_inv, const double g00_gr) {
    using S = typename Arith<TS>::S;
    using VD = std::conditional_t<kOne<V>, double, D2>;
    auto round = [](const VD v) -> V {
        if constexpr (sizeof(TS) == 8) return v;
        else return make_v<V>((float)first(v), (float)second(v));
    };
    auto ld = [&](const double* q) { return ld_v<SHIFT, VD>(q, nb.o2); };
    const V f = round(ld(op.c));
    const TS fm = (TS)op.c[-1], fp = (TS)op.c[nb.pp];
    const V dx = v_mul(round(v_sub(ld(op.xm), ld(op.xp))), th.vr);
    V G = p_diff(f, fm, fp);
    if (th.is0) {
        const TS f1 = above(f, fp);
        const TS f0 = fma_rn(-f1, (TS)g00_s, first(f));   // f00(p=0) (1 - s)
        first(G) = mul_rn(fma_rn(-f0, (TS)g00_inv, f1), (TS)g00_gr);
    }
    const S2<S> e = coef2(c, kExG);
    A.R[0] = v_fma(s_mul(e.a, th.ex), G, v_mul(e.b, dx));
    if constexpr (MC >= 1) {
        const V dy = v_mul(round(v_sub(ld(op.ym), ld(op.yp))), th.vr);
        const S2<S> g2 = coef2(c, kEmG);
        A.R[1] = v_fma(s_mul(g2.a, th.ey), G, v_mul(g2.b, dy));
        A.I[1] = v_mul(s_neg(s_mul(g2.a, th.ez)), G);
    }
}

// ---------------------------------------------------------------------------
// geometry and shared-memory plan
// ---------------------------------------------------------------------------
struct Geo {
    int np, nx, ny, tx, tiles_x, nseg;
    bool has_y;
};
__host__ __device__ inline Geo make_geo(int np, int nx, int ny, int tx) {
    Geo g;
    g.np = np; g.nx = nx; g.ny = ny; g.tx = tx;
    g.tiles_x = (nx + tx - 1) / tx;
    g.has_y = ny > 1;
    g.nseg = (np + 31) >> 5;
    return g;
}
// Bytes of `cells` cells' rows in shared memory: back to back, or (SHIFT) the
// aligned span that holds them.
template <bool SHIFT>
__host__ __device__ inline size_t piece_bytes(const Geo& g, int cells, int elem_bytes) {
    const size_t b = (size_t)cells * g.np * elem_bytes;
    return SHIFT ? align_up(b, 16) + 16 : b;
}
// one component of a source: the x-1 cell, the tile's cells, the x+1 cell, and
// in 2D the cells of y-1 and of y+1 (a piece each)
template <bool SHIFT>
__host__ __device__ inline size_t comp_bytes(const Geo& g, int elem_bytes) {
    return 2 * piece_bytes<SHIFT>(g, 1, elem_bytes) + (g.has_y ? 3 : 1) * piece_bytes<SHIFT>(g, g.tx, elem_bytes);
}
// a source slot: one harmonic's Re and Im cells (Re alone when m0 = 0), or
// the FP64 f00 cells with the tile's six fields behind them
__host__ __device__ inline size_t fld_stride(int tx, int elem_bytes) { return align_up((size_t)tx * elem_bytes, 16) + 16; }
template <bool SHIFT>
__host__ __device__ inline size_t src_slot_bytes(const Geo& g, int elem_bytes, int m0) {
    const size_t pl = (m0 > 0 ? 2 : 1) * comp_bytes<SHIFT>(g, elem_bytes);
    const size_t f0 = comp_bytes<SHIFT>(g, 8) + 6 * fld_stride(g.tx, elem_bytes);
    return align_up(pl > f0 ? pl : f0, 128);
}
// one operand array of a target slot: Re and Im of the tile's cells, or f00's
template <bool SHIFT>
__host__ __device__ inline size_t tgt_array_bytes(const Geo& g, int elem_bytes, int m0) {
    const size_t pl = (m0 > 0 ? 2 : 1) * piece_bytes<SHIFT>(g, g.tx, elem_bytes);
    const size_t f0 = piece_bytes<SHIFT>(g, g.tx, 8);
    return align_up(pl > f0 ? pl : f0, 16);
}
struct Plan {
    int D, RD;                       // slots of the source and target rings
    uint32_t src_stride, tgt_arr, tgt_stride;
    uint32_t off_cnt, off_j, off_coef, off_plane, off_src, off_tgt, total;
    int hw;                          // half-warps of the consumers
};
// barriers at offset 0: source full/empty, target full/empty
static_assert(4 * kMaxDepth * sizeof(uint64_t) <= 384, "barrier area");
__host__ __device__ inline Plan make_plan(int D, int RD, size_t src_bytes, size_t tgt_arr, int narr, int hw, int ncoef) {
    Plan P;
    P.D = D; P.RD = RD; P.hw = hw;
    P.off_cnt = 384;
    P.off_j = (uint32_t)align_up(P.off_cnt + sizeof(int) * kJBuf * hw, 16);
    P.off_coef = (uint32_t)align_up(P.off_j + sizeof(double) * 3 * kJBuf * hw, 16);
    P.off_plane = P.off_coef + 128u * ncoef;
    P.off_src = (uint32_t)align_up(P.off_plane + sizeof(int) * ncoef, 128);
    P.src_stride = (uint32_t)align_up(src_bytes, 128);
    P.off_tgt = P.off_src + D * P.src_stride;
    P.tgt_arr = (uint32_t)tgt_arr;
    P.tgt_stride = (uint32_t)align_up(tgt_arr * narr, 128);
    P.total = P.off_tgt + RD * P.tgt_stride;
    return P;
}
// the deepest rings within `cap`: both look about equally far ahead, the
// sources first; false when the smallest rings do not fit
inline bool deepest_plan(size_t cap, size_t src_bytes, size_t tgt_arr, int narr, int hw, int ncoef, Plan& P) {
    int D = kMinSrc, RD = narr ? kMinTgt : 0;
    auto fits = [&](int d, int r) {
        return make_plan(d, r, src_bytes, tgt_arr, narr, hw, ncoef).total <= cap;
    };
    if (!fits(D, RD)) return false;
    for (bool more = true; more;) {
        more = false;
        if (D < kMaxDepth && (D <= RD + 1 || !narr || RD == kMaxDepth) && fits(D + 1, RD)) { ++D; more = true; }
        if (narr && RD < kMaxDepth && RD < D && fits(D, RD + 1)) { ++RD; more = true; }
    }
    while (D < kMaxDepth && fits(D + 1, RD)) ++D;
    while (narr && RD < kMaxDepth && fits(D, RD + 1)) ++RD;
    P = make_plan(D, RD, src_bytes, tgt_arr, narr, hw, ncoef);
    return true;
}

// a ring position: slot index and the parity of its current use
struct RingPos {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int depth) {
        if (++slot == depth) { slot = 0; phase ^= 1u; }
    }
};

// a consumer's ring position: byte offset of the slot, address of its full
// barrier (the empty barrier is kMaxDepth further) and the parity
struct RingAddr {
    uint32_t off, bar, phase;
    __device__ __forceinline__ void start(uint32_t off0, uint32_t bar0) { off = off0; bar = bar0; phase = 0; }
    __device__ __forceinline__ void next(uint32_t stride, uint32_t end, uint32_t off0, uint32_t bar0) {
        off += stride; bar += 8;
        if (off == end) { off = off0; bar = bar0; phase ^= 1u; }
    }
};

// ---------------------------------------------------------------------------
// producers: one thread each, walking the stream in the consumers' order; they
// stop (returning false) when a wait for a free slot runs out
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool slot_free(uint64_t* empty, const RingPos& r, int issued, int depth,
                                          unsigned long long wlim) {
    return issued < depth || mbar_wait_hold(empty + r.slot, r.phase ^ 1u, wlim);
}
// the 16-byte aligned span around [src, src + bytes): it never leaves the
// allocation's pages; bytes itself where rows are 16-byte multiples
template <bool SHIFT>
__device__ __forceinline__ uint32_t span_bytes(const void* src, size_t bytes) {
    if constexpr (!SHIFT) return (uint32_t)bytes;
    const uintptr_t lo = reinterpret_cast<uintptr_t>(src), hi = lo + bytes;
    return (uint32_t)(((hi + 15) & ~(uintptr_t)15) - (lo & ~(uintptr_t)15));
}
template <bool SHIFT>
__device__ __forceinline__ void copy_span(void* dst, const void* src, size_t bytes, uint64_t* bar) {
    if constexpr (!SHIFT) bulk_g2s(dst, src, (uint32_t)bytes, bar);
    else bulk_g2s(dst, reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15),
                  span_bytes<true>(src, bytes), bar);
}

// the sources of one tile.  BATCH: its problem's descriptor comes along with
// f00 (to desc_dst), and every source's coefficients at the end of its slot.
template <typename TS, bool SHIFT, bool BATCH = false>
__device__ __forceinline__ bool produce_sources(const StageArgs<TS>& a, const Geo& g, const Plan& P, const int tile,
                                                unsigned char* smem, RingPos& r, int& issued,
                                                const unsigned long long wlim, const int withhold,
                                                const unsigned char* desc = nullptr, const uint32_t desc_bytes = 0,
                                                unsigned char* desc_dst = nullptr) {
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + kMaxDepth;
    const int np = g.np, nx = g.nx, tx = g.tx;
    const int y = tile / g.tiles_x;
    const int x0 = (tile - y * g.tiles_x) * tx;
    const int txv = min(tx, nx - x0);
    const long long row = (long long)y * nx;
    const long long rym = (long long)(y == 0 ? g.ny - 1 : y - 1) * nx;
    const long long ryp = (long long)(y == g.ny - 1 ? 0 : y + 1) * nx;
    const long long xm_cell = row + (x0 == 0 ? nx - 1 : x0 - 1);
    const long long xp_cell = row + (x0 + txv == nx ? 0 : x0 + txv);
    // the x-stencil cells are one contiguous run unless it wraps
    const bool x_contig = !SHIFT && x0 > 0 && x0 + txv < nx;
    long long q = 0;   // planes are stored in (l, m) order, Re then Im
    for (int s = 0; s <= a.l0; ++s) {
        for (int m = 0; m <= min(s, a.m0); ++m) {
            if (issued == withhold) return false;   // fault injection (tests): this copy and all later ones stay out
            if (!slot_free(empty, r, issued, P.D, wlim)) return false;
            unsigned char* dst = smem + P.off_src + (size_t)r.slot * P.src_stride;
            uint64_t* bar = full + r.slot;
            const int esz = s == 0 ? 8 : (int)sizeof(TS);
            const int ncomp = m > 0 ? 2 : 1;
            const unsigned char* src = s == 0 ? reinterpret_cast<const unsigned char*>(a.f00_in)
                                              : reinterpret_cast<const unsigned char*>(a.pl_in + q * a.pstride);
            const size_t bpc = (size_t)np * esz;            // bytes per cell
            const size_t one = piece_bytes<SHIFT>(g, 1, esz), many = piece_bytes<SHIFT>(g, tx, esz);
            // the five pieces of component `comp`: x-1, the cells, x+1, y-1, y+1.  The edge
            // neighbours come from the x halo columns when the grid has them (an x slab, or
            // mirrored x boundaries).
            auto piece = [&](int comp, int i) -> const unsigned char* {
                const unsigned char* pb = src + (size_t)comp * a.pstride * esz;
                if (a.hx && ((i == 0 && x0 == 0) || (i == 2 && x0 + txv == nx))) {
                    const int side = i == 0 ? 0 : 1;
                    if (s == 0) return reinterpret_cast<const unsigned char*>(hx_f00(a, side, y));
                    return reinterpret_cast<const unsigned char*>(hx_plane(a, side, q + comp, y));
                }
                const long long cell = i == 0 ? xm_cell : i == 1 ? row + x0 : i == 2 ? xp_cell : (i == 3 ? rym : ryp) + x0;
                return pb + (size_t)cell * bpc;
            };
            const int npieces = g.has_y ? 5 : 3;
            uint32_t bytes = 0;
            if constexpr (SHIFT) {
                for (int comp = 0; comp < ncomp; ++comp)
                    for (int i = 0; i < npieces; ++i) bytes += span_bytes<true>(piece(comp, i), (i == 0 || i == 2 ? 1 : txv) * bpc);
            } else {
                bytes = (uint32_t)(ncomp * (txv + 2 + (g.has_y ? 2 * txv : 0)) * bpc);
            }
            if (s == 0)   // the tile's fields: per field the aligned span holding its txv values
                for (int f = 0; f < 6; ++f) bytes += span_bytes<true>(a.fld_in + f * a.cells + row + x0, txv * sizeof(TS));
            if constexpr (BATCH) bytes += kCoefBytes + (s == 0 ? desc_bytes : 0u);
            mbar_expect_tx(bar, bytes);
            if constexpr (BATCH) {
                if (s == 0) bulk_g2s(desc_dst, desc, desc_bytes, bar);
                bulk_g2s(dst + P.src_stride - kCoefBytes,
                         reinterpret_cast<const unsigned char*>(a.coef_ts) + (size_t)(s * (a.m0 + 1) + m) * kCoefBytes,
                         kCoefBytes, bar);
            }
            for (int comp = 0; comp < ncomp; ++comp) {
                unsigned char* cb = dst + comp * comp_bytes<SHIFT>(g, esz);
                if (x_contig) {
                    copy_span<false>(cb, piece(comp, 0), (txv + 2) * bpc, bar);
                } else {
                    copy_span<SHIFT>(cb, piece(comp, 0), bpc, bar);
                    copy_span<SHIFT>(cb + one, piece(comp, 1), txv * bpc, bar);
                    copy_span<SHIFT>(cb + one + (SHIFT ? many : txv * bpc), piece(comp, 2), bpc, bar);
                }
                if (g.has_y) {
                    copy_span<SHIFT>(cb + 2 * one + many, piece(comp, 3), txv * bpc, bar);
                    copy_span<SHIFT>(cb + 2 * one + 2 * many, piece(comp, 4), txv * bpc, bar);
                }
            }
            if (s == 0) {
                unsigned char* fd = dst + comp_bytes<SHIFT>(g, 8);
                for (int f = 0; f < 6; ++f)
                    copy_span<true>(fd + f * fld_stride(tx, (int)sizeof(TS)), a.fld_in + f * a.cells + row + x0,
                                    txv * sizeof(TS), bar);
            } else {
                q += ncomp;
            }
            r.next(P.D);
            ++issued;
        }
    }
    return true;
}

// the RK operands of one tile's targets, (l, m) order
template <typename TS, bool SHIFT>
__device__ __forceinline__ bool produce_targets(const StageArgs<TS>& a, const Geo& g, const Plan& P, const int tile,
                                                unsigned char* smem, RingPos& r, int& issued,
                                                const unsigned long long wlim) {
    uint64_t* full = reinterpret_cast<uint64_t*>(smem) + 2 * kMaxDepth;
    uint64_t* empty = full + kMaxDepth;
    const int y = tile / g.tiles_x;
    const int x0 = (tile - y * g.tiles_x) * g.tx;
    const int txv = min(g.tx, g.nx - x0);
    const long long base = ((long long)y * g.nx + x0) * g.np;
    const int kind = a.kind;
    const int narr = stage_arrays(kind);
    long long q = 0;
    for (int t = 0; t <= a.l0; ++t) {
        for (int m = 0; m <= min(t, a.m0); ++m) {
            if (!slot_free(empty, r, issued, P.RD, wlim)) return false;
            unsigned char* dst = smem + P.off_tgt + (size_t)r.slot * P.tgt_stride;
            uint64_t* bar = full + r.slot;
            const int esz = t == 0 ? 8 : (int)sizeof(TS);
            const int ncomp = m > 0 ? 2 : 1;
            const size_t b = (size_t)txv * g.np * esz;
            // Y0, then Y (the last stage reads Y alone)
            auto operand = [&](int i, int comp) -> const unsigned char* {
                const bool acc = i == 1 || kind == kStageLast;
                if (t == 0) return reinterpret_cast<const unsigned char*>((acc ? a.f00_A : a.f00_B) + base);
                return reinterpret_cast<const unsigned char*>((acc ? a.pl_A : a.pl_B) + (q + comp) * a.pstride + base);
            };
            uint32_t bytes = 0;
            for (int i = 0; i < narr; ++i)
                for (int comp = 0; comp < ncomp; ++comp) bytes += span_bytes<SHIFT>(operand(i, comp), b);
            mbar_expect_tx(bar, bytes);
            for (int i = 0; i < narr; ++i)
                for (int comp = 0; comp < ncomp; ++comp)
                    copy_span<SHIFT>(dst + (size_t)i * P.tgt_arr + comp * piece_bytes<SHIFT>(g, g.tx, esz),
                                     operand(i, comp), b, bar);
            if (t > 0) q += ncomp;
            r.next(P.RD);
            ++issued;
        }
    }
    return true;
}

// waits (bounded) for the copies a stopped producer may still have in flight
__device__ __forceinline__ void drain(uint64_t* full, RingPos r, int issued, int depth, unsigned long long wlim) {
    for (int k = min(issued, depth); k > 0; --k) {
        if (--r.slot < 0) { r.slot = depth - 1; r.phase ^= 1u; }
        mbar_wait_hold(full + r.slot, r.phase, wlim);
    }
}

// ---------------------------------------------------------------------------
// consumers
// ---------------------------------------------------------------------------
struct Consumer {
    RingAddr src, tgt;
    int tile_iter;
    __device__ __forceinline__ void start(const Plan& P, const unsigned char* smem) {
        src.start(P.off_src, smem_u32(smem));
        tgt.start(P.off_tgt, smem_u32(smem) + 2 * kMaxDepth * 8);
        tile_iter = 0;
    }
};
// barrier offset from a slot's full to its empty barrier
constexpr uint32_t kEmptyOff = kMaxDepth * 8;

// MC: the problem's m0; PT: momentum points of a thread; BATCH: the source
// slots end with the source's coefficients (coef and plane_of are not read;
// m0 = 0, whose plane of row l is l - 1)
template <int MC, typename TS, int PT, bool SHIFT, bool BATCH = false>
__device__ __forceinline__ void consume_tile(const StageArgs<TS>& a, const CoefS<TS>* __restrict__ coef,
                                             const int* __restrict__ plane_of, const Geo& g, const Plan& P,
                                             const int tile, unsigned char* smem, Consumer& cs, int* err,
                                             const unsigned long long wlim) {
    using V = typename VecOf<TS, PT>::V;
    constexpr int kSeg = 32 / PT;   // lanes of 32 points
    constexpr int m0 = MC;
    const uint32_t bar0 = smem_u32(smem), tbar0 = bar0 + 2 * kMaxDepth * 8;
    const int tid = threadIdx.x, lane = tid & 31, lseg = lane & (kSeg - 1);
    const int np = g.np, nx = g.nx, tx = g.tx;
    const int mstride = m0 + 1;
    const int y = tile / g.tiles_x;
    const int x0 = (tile - y * g.tiles_x) * tx;
    const int txv = min(tx, nx - x0);
    const int hw = tid / kSeg;
    const int c = hw / g.nseg, hseg = hw - c * g.nseg;
    const int p0 = hseg * 32 + PT * lseg;
    const bool cv = c < txv;
    const bool pv = cv && p0 < np, pv1 = PT > 1 && cv && p0 + 1 < np;
    // invalid threads read a valid point (finite data) and store nothing
    const int cc = cv ? c : 0, pc = p0 < np ? p0 : 0;
    const int pc1 = min(pc + 1, np - 1);
    const int xc = x0 + cc;
    const long long cell = (long long)y * nx + xc;
    const long long o = cell * np + pc;

    Nb nb;
    nb.pp = PT == 1 ? (pc + 1 < np ? 1 : 0) : (pc + 2 < np ? 2 : 1);
    nb.o2 = pc1 - pc;
    nb.p = pc;
    nb.p_1 = pc1;
    nb.p_m = pc - (pc > 0 ? 1 : 0);
    nb.p_p = min(pc + PT, np - 1);
    constexpr int kElems = 16 / (int)sizeof(TS);
    // offsets in elements of this size (FP32: f00 lies in a slot of its own layout, set below)
    auto place = [&](Nb& n, const int esz) {
        const int one = (int)(piece_bytes<SHIFT>(g, 1, esz) / esz), many = (int)(piece_bytes<SHIFT>(g, tx, esz) / esz);
        n.ctr = one + cc * np + pc;
        if constexpr (!SHIFT) {
            n.x = np;
            n.ym = g.has_y ? (tx + 1) * np : 0;
            n.yp = g.has_y ? (2 * tx + 1) * np : 0;
        } else {
            const bool left = cc == 0, right = cc == txv - 1;
            n.xm = left ? pc : n.ctr - np;
            n.xp = right ? one + many + pc : n.ctr + np;
            n.ym = g.has_y ? 2 * one + many + cc * np + pc : n.ctr;
            n.yp = g.has_y ? 2 * one + 2 * many + cc * np + pc : n.ctr;
            const long long row = (long long)y * nx;
            const long long rym = (long long)(y == 0 ? g.ny - 1 : y - 1) * nx, ryp = (long long)(y == g.ny - 1 ? 0 : y + 1) * nx;
            auto el = [&](long long cell) { return (int)(cell * np % kElems); };
            const bool hl = a.hx && x0 == 0, hr = a.hx && x0 + txv == nx;
            n.ac = el(row + x0);
            n.axm = left ? el(hl ? y : row + (x0 == 0 ? nx - 1 : x0 - 1)) : n.ac;
            n.axp = right ? el(hr ? y : row + (x0 + txv == nx ? 0 : x0 + txv)) : n.ac;
            n.aym = g.has_y ? el(rym + x0) : n.ac;
            n.ayp = g.has_y ? el(ryp + x0) : n.ac;
            n.b = (int)(a.pstride % kElems);
            n.bxm = left && hl ? el(g.ny) : n.b;
            n.bxp = right && hr ? el(g.ny) : n.b;
        }
    };
    place(nb, (int)sizeof(TS));
    const int seg = (int)(comp_bytes<SHIFT>(g, (int)sizeof(TS)) / sizeof(TS));
    const int toff = cc * np + pc;               // this thread's points inside a target array
    const int tcomp = (int)(piece_bytes<SHIFT>(g, tx, (int)sizeof(TS)) / sizeof(TS));   // Re to Im there
    const int tel = SHIFT ? (int)(((long long)y * nx + x0) * np % kElems) : 0;           // SHIFT: the tile's first element

    auto acquire = [&]() { mbar_wait_or_exit(cs.src.bar, cs.src.phase, err, wlim); };
    auto release = [&]() {
        warp_arrive(cs.src.bar + kEmptyOff, lane);
        cs.src.next(P.src_stride, P.off_tgt, P.off_src, bar0);
    };

    auto slot_coef = [&]() {
        return reinterpret_cast<const CoefS<TS>*>(smem + cs.src.off + P.src_stride - kCoefBytes);
    };

    acquire();
    Th<TS, V> th;
    {
        // field f of this cell: its span's start is the aligned-down address
        const unsigned char* fb = smem + cs.src.off + comp_bytes<SHIFT>(g, 8);
        const size_t fst = fld_stride(tx, (int)sizeof(TS));
        auto fval = [&](int f) -> TS {
            const uintptr_t sh = reinterpret_cast<uintptr_t>(a.fld_in + f * a.cells + (long long)y * nx + x0) & 15;
            return reinterpret_cast<const TS*>(fb + f * fst + sh)[cc];
        };
        const int parts = a.parts;
        // the couplings of the parts not evaluated see a zero field
        th.ex = bcast((parts & kPartEx) ? fval(0) : TS(0));
        th.ey = bcast((parts & kPartEy) ? fval(1) : TS(0));
        th.ez = bcast((parts & kPartEz) ? fval(2) : TS(0));
        const bool b = (parts & kPartB) != 0;
        th.bx = bcast(b ? fval(3) : TS(0));
        th.hby = bcast(b ? mul_rn(TS(0.5), fval(4)) : TS(0));
        th.hbz = bcast(b ? mul_rn(TS(0.5), fval(5)) : TS(0));
        th.is0 = pc == 0;
        th.invp = make_v<V>((TS)ldg(a.inv_pr + pc), (TS)ldg(a.inv_pr + pc1));
        const bool adv = (parts & kPartAdv) != 0;
        th.vr = adv ? make_v<V>((TS)ldg(a.vr + pc), (TS)ldg(a.vr + pc1)) : make_v<V>(TS(0), TS(0));
    }

    // RK update of the targets: t = k c1, out = Y0 + t, Y = (Y0 or Y) + t c2
    const int kind = a.kind;
    const bool staged = kind != kStageSlope, has_out = kind != kStageLast;
    const uint32_t yoff = kind == kStageMid ? P.tgt_arr : 0u;   // Y behind Y0, or the only operand
    const int nclean = (a.parts & kPartClean) ? 80 : 0;
    // outputs at this thread's pair, moved plane by plane ((l, m) order, Re then Im)
    TS* out = has_out ? a.pl_out + o : nullptr;
    TS* acc = a.pl_A + o;
    auto put = [&](TS* d, const V v) {
        if constexpr (SHIFT && PT > 1) {
            if (pv) d[0] = first(v);
            if (pv1) d[1] = second(v);
        } else {
            if (pv) *reinterpret_cast<V*>(d) = v;
        }
    };
    auto ld = [&](const TS* q) { return ld_v<SHIFT, V>(q, nb.o2); };
    auto tgt_acquire = [&]() { if (staged) mbar_wait_or_exit(cs.tgt.bar, cs.tgt.phase, err, wlim); };
    auto tgt_release = [&]() {
        if (staged) {
            warp_arrive(cs.tgt.bar + kEmptyOff, lane);
            cs.tgt.next(P.tgt_stride, P.total, P.off_tgt, tbar0);
        }
    };
    auto component = [&](V k, const TS* B, const int nz) {
        if (p0 < nz) {
            if constexpr (PT == 1) k = TS(0);
            else k = make_v<V>(TS(0), p0 + 1 < nz ? TS(0) : second(k));
        }
        if (staged) {
            const V tt = v_mul(k, make_v<V>((TS)a.c1, (TS)a.c1));
            if (has_out) put(out, v_add(ld(B), tt));
            const TS* Y = reinterpret_cast<const TS*>(reinterpret_cast<const unsigned char*>(B) + yoff);
            put(acc, v_fma(tt, make_v<V>((TS)a.c2, (TS)a.c2), ld(Y)));
        } else {
            put(out, k);
        }
        out += a.pstride;
        acc += a.pstride;
    };
    // target (t, m), t >= 1
    int tq = 0;   // its plane
    auto finish = [&](const int t, auto mcst, const V kr, const V ki) {
        tgt_acquire();
        const TS* B = reinterpret_cast<const TS*>(smem + cs.tgt.off) + toff;
        auto sh = [&](int q) { return SHIFT ? (tel + q * nb.b) & (kElems - 1) : 0; };
        const int nz = t >= 2 ? min(t - 1, nclean) : 0;
        component(kr, B + sh(tq), nz);
        ++tq;
        if constexpr (decltype(mcst)::value > 0) {
            component(ki, B + tcomp + sh(tq), nz);
            ++tq;
        }
        tgt_release();
    };
    // target (0, 0): the FP64 f00 plane
    auto finish_f00 = [&](const V kr) {
        tgt_acquire();
        const double* B = reinterpret_cast<const double*>(smem + cs.tgt.off) + toff + (tel & 1);
        const double* Y = reinterpret_cast<const double*>(reinterpret_cast<const unsigned char*>(B) + yoff);
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const double k = (double)(j == 0 ? first(kr) : second(kr));
            if (j == 0 ? pv : pv1) {
                if (staged) {
                    const double tt = mul_rn(k, a.c1);
                    if (has_out) a.f00_out[o + j] = add_rn(B[j], tt);
                    a.f00_A[o + j] = fma_rn(tt, a.c2, Y[j]);
                } else {
                    a.f00_out[o + j] = k;
                }
            }
        }
        tgt_release();
    };

    Acc<V, MC> A0, A1;
    acc_zero<TS, V, MC>(A0);
    acc_zero<TS, V, MC>(A1);
    // the current, a thread's points apart until the last addition: the order of
    // a sum over 32 lanes of one point each
    double jx[PT] = {}, jyr[PT] = {}, jyi[PT] = {};

    // source row 0: f00 into row 1
    {
        Nb n0 = nb;
        if constexpr (sizeof(TS) == 4) place(n0, 8);
        couple_f00<MC, SHIFT, TS, V>(A1, BATCH ? slot_coef() : coef, operands<SHIFT>(reinterpret_cast<const double*>(smem + cs.src.off), n0, 0), n0, th,
                              a.g00_s, a.g00_inv, a.g00_gr);
    }
    release();

    // A0, A1, A2 hold target rows s-1, s, s+1 while source row s is added.
    // Target (s-1, m-1) is complete after source (s, m), and (s-1, m0) after
    // the row.
    const int l0 = a.l0;
    for (int s = 1; s <= l0; ++s) {
        const CoefS<TS>* crow = BATCH ? nullptr : coef + s * mstride;
        Acc<V, MC> A2;
        // the sources of the row, one inside the other: a row that ends early
        // leaves them all at once, and no accumulator passes a join per source
        auto sources = [&](auto self, auto mcst) -> void {
            constexpr int m = decltype(mcst)::value;
            acquire();
            const TS* sb = reinterpret_cast<const TS*>(smem + cs.src.off);
            const TS* ref = nullptr;
            const int qs = BATCH ? s - 1 : (sizeof(TS) == 4 || SHIFT) ? plane_of[s * mstride + m] : 0;
            if constexpr (sizeof(TS) == 4) ref = (a.pl_ref && __ldg(a.pl_keep + qs)) ? a.pl_ref + (long long)qs * np : nullptr;
            couple_src<MC, m, SHIFT, TS, V>(A0, A1, A2, BATCH ? slot_coef() : crow + m, sb, seg, nb, th, ref, np, qs);
            if constexpr (m <= 1) {
                if (s == 1) {
                    // the current of f = ref + stored deviation
                    auto quad = [&](double (&j)[PT], const TS* v, const TS* rf) {
#pragma unroll
                        for (int k = 0; k < PT; ++k) {
                            double f = (double)v[k == 0 ? 0 : SHIFT ? nb.o2 : 1];
                            if (rf) f = add_rn(f, (double)rf[k == 0 ? pc : pc1]);
                            if (k == 0 ? pv : pv1) j[k] = mul_rn(ldg(a.wj + (k == 0 ? pc : pc1)), f);
                        }
                    };
                    if constexpr (m == 0) {
                        quad(jx, operands<SHIFT>(sb, nb, qs).c, ref);
                    } else {
                        quad(jyr, operands<SHIFT>(sb, nb, qs).c, ref);
                        quad(jyi, operands<SHIFT>(sb + seg, nb, qs + 1).c, ref ? ref + np : nullptr);
                    }
                }
            }
            release();
            if constexpr (m >= 1) {
                if (m == 1 && s == 1) finish_f00(A0.R[0]);
                else finish(s - 1, std::integral_constant<int, m - 1>{}, A0.R[m - 1], A0.I[m - 1]);
            }
            if constexpr (m < MC) {
                if (m < s && m < m0) {
                    self(self, std::integral_constant<int, m + 1>{});
                    return;
                }
            }
            if (m == m0 && s > m0) {
                if (m == 0 && s == 1) finish_f00(A0.R[0]);
                else finish(s - 1, mcst, A0.R[m], A0.I[m]);
            }
        };
        sources(sources, std::integral_constant<int, 0>{});
        // the rows move down one accumulator: one copy of the source-row code
        // keeps the loop within the instruction cache
        A0 = A1;
        A1 = A2;
    }
    static_for<MC + 1>([&](auto mcst) {
        constexpr int m = decltype(mcst)::value;
        if (m <= min(l0, m0)) finish(l0, mcst, A0.R[m], A0.I[m]);
    });

    // the cell's current: sums over 32 points to shared memory; the last
    // half-warp of the cell adds them in order and updates E and B.  No
    // barrier joins the consumer warps: a warp whose wait ran out stops on its
    // own.  A source slot is filled again only when every warp has released it,
    // also in slope launches (no operand ring): a warp can be at most kMaxDepth
    // slots, two or more of them a tile, ahead of one that is still adding, so
    // kJBuf sets of sums are enough.
    auto total = [&](double (&j)[PT]) -> double {
#pragma unroll
        for (int off = kSeg / 2; off > 0; off >>= 1)
#pragma unroll
            for (int k = 0; k < PT; ++k) j[k] += __shfl_xor_sync(kFull, j[k], off);
        return PT > 1 ? add_rn(j[0], j[PT - 1]) : j[0];
    };
    const double Sx = total(jx), Syr = total(jyr), Syi = total(jyi);
    double* sj = reinterpret_cast<double*>(smem + P.off_j) + (size_t)(cs.tile_iter % kJBuf) * 3 * P.hw;
    int* cnt = reinterpret_cast<int*>(smem + P.off_cnt) + (cs.tile_iter % kJBuf) * P.hw;
    int old = -1;
    if (lseg == 0 && cv) {
        sj[3 * hw] = Sx;
        sj[3 * hw + 1] = Syr;
        sj[3 * hw + 2] = Syi;
        __threadfence_block();
        old = atomicAdd(cnt + c, 1);
    }
    old = __shfl_sync(kFull, old, lane & ~(kSeg - 1));
    if (old == g.nseg - 1) {
        __threadfence_block();
        double Jx = 0.0, Jyr = 0.0, Jyi = 0.0;
        const double* j = sj + 3 * (size_t)c * g.nseg;
        for (int w = 0; w < g.nseg; ++w) { Jx += j[3 * w]; Jyr += j[3 * w + 1]; Jyi += j[3 * w + 2]; }
        if (lseg < 6) field_update(a, lseg, cell, y, xc, Jx, Jyr, Jyi);
        if (lseg == 0) cnt[c] = 0;
    }
    __syncwarp();
    ++cs.tile_iter;
}

// cells of a tile: as many as the consumers' 32-point segments hold (rows of up
// to 32 points fill them with 16: 62500 such cells, l0 = 1, a step without
// collisions 0.43 ms with 8 cells, 0.29 with 16)
constexpr int kMaxCells = 16;
inline int tile_cells(int np, int nx, int segments) { return batch_cells(np, nx, 32 * segments, kMaxCells); }

// Warps of a CTA.  Registers are granted per SM sub-partition, so a CTA costs
// multiples of 4 warps: 8 warps leave 255 registers a thread, 12 warps 168, 16
// warps 128; each form takes the most warps whose registers hold its
// accumulators without spilling (the rings leave the L1 too small to hold
// spilled registers).  Two points a thread where that fits, else one (FP64, m0
// >= 3).  FP32 rows of 51 points on 64 x 64 cells, l0 = m0 = 6, two steps 2.18
// -> 1.60 ms with two, in spite of 376 bytes spilled; FP64 rows of 129 points
// on 30 x 31 cells, l0 = 4, m0 = 2, 646 -> 407 us (128 bytes spilled).
template <int MC, typename TS>
constexpr int points() { return sizeof(TS) == 4 || MC <= 2 ? 2 : 1; }
template <int MC, typename TS>
constexpr int consumer_warps() {
    if (MC == 0) return 8;
    if (sizeof(TS) == 8) return MC <= 6 ? 10 : 6;
    return MC <= 2 ? 14 : MC <= 6 ? 10 : 6;
}
// CTAs per SM: two for m0 = 0, so that one CTA's tile starts and ends overlap
// the other's work
template <int MC>
constexpr int tile_min_blocks() { return MC == 0 ? 2 : 1; }

// MC: the problem's m0; PT: points of a thread
template <int MC, typename TS, bool SHIFT, int PT>
__global__ void __launch_bounds__((consumer_warps<MC, TS>() + 2) * 32, tile_min_blocks<MC>())
    rk_stage_pair_kernel(const __grid_constant__ StageArgs<TS> a, const __grid_constant__ Plan P, const int tx) {
    extern __shared__ __align__(128) unsigned char smem[];
    const Geo g = make_geo(a.np, a.nx, a.ny, tx);
    const int tid = threadIdx.x;
    const int nct = (int)blockDim.x - 64;              // consumer threads
    const int ncw = nct >> 5;
    const int ncoef = (a.l0 + 1) * (a.m0 + 1);
    const int ntiles = g.tiles_x * g.ny;
    const unsigned long long wlim = a.wait_ns;   // every pipeline wait gives up after this
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    CoefS<TS>* scoef = reinterpret_cast<CoefS<TS>*>(smem + P.off_coef);
    int* splane = reinterpret_cast<int*>(smem + P.off_plane);

    // tables to shared memory (coefficients in the arithmetic type), barriers
    for (int i = tid; i < ncoef * 16; i += blockDim.x) scoef[i >> 4].v[i & 15] = bcast((TS)coef_entry(a.coef[i >> 4], i & 15));
    for (int i = tid; i < ncoef; i += blockDim.x) splane[i] = a.plane_of[i];
    for (int i = tid; i < kJBuf * P.hw; i += blockDim.x) reinterpret_cast<int*>(smem + P.off_cnt)[i] = 0;
    if (tid == 0) {
        for (int k = 0; k < kMaxDepth; ++k) {
            mbar_init(bars + k, 1);
            mbar_init(bars + kMaxDepth + k, ncw);
            mbar_init(bars + 2 * kMaxDepth + k, 1);
            mbar_init(bars + 3 * kMaxDepth + k, ncw);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (tid >= nct) {
        if ((tid & 31) != 0) return;
        const bool sources = tid == nct;
        if (!sources && a.kind == kStageSlope) return;   // the slope form reads no operands
        RingPos r;
        int issued = 0;
        bool ok = true, injected = false;
        const int withhold = (sources && blockIdx.x == 0) ? a.withhold : -1;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
            ok = sources ? produce_sources<TS, SHIFT>(a, g, P, tile, smem, r, issued, wlim, withhold)
                         : produce_targets<TS, SHIFT>(a, g, P, tile, smem, r, issued, wlim);
            if (!ok && issued == withhold) injected = true;
        }
        if (!ok) {
            if (!injected) atomicOr(a.err, 16);
            // bounded drain of every copy that may still be in flight
            drain(bars + (sources ? 0 : 2 * kMaxDepth), r, issued, sources ? P.D : P.RD, wlim);
        }
        return;
    }

    Consumer cs;
    cs.start(P, smem);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
        consume_tile<MC, TS, PT, SHIFT>(a, scoef, splane, g, P, tile, smem, cs, a.err, wlim);
}

template <int MC, typename TS, bool SHIFT, int PT>
cudaError_t pair_form(const StageArgs<TS>& a, cudaStream_t s) {
    constexpr int per_warp = PT;                             // 32-point segments of a warp
    constexpr int max_hw = per_warp * consumer_warps<MC, TS>();
    constexpr int elem = (int)sizeof(TS);
    if ((a.np + 31) / 32 > max_hw) return cudaErrorNotSupported;
    int tx = tile_cells(a.np, a.nx, max_hw);
    const int widest = tx;
    auto tiles_of = [&](int t) { return (long long)a.ny * ((a.nx + t - 1) / t); };
    // at least one tile per SM where the grid has the cells for it
    const long long per_sm = (long long)a.nx * a.ny / sm_count();
    if (tx > per_sm) tx = per_sm > 1 ? (int)per_sm : 1;
    // one CTA an SM: the fewest cells that leave no CTA a second tile, since a
    // tile's time is mostly latency (FP32, 16 x 17 cells of 201 points, l0 = 6,
    // m0 = 4, two steps: tiles of one cell 699 us, of two 401; the global-load
    // kernel 584)
    if (MC > 0)
        for (int t = tx; t <= widest; ++t)
            if (tiles_of(t) <= sm_count()) { tx = t; break; }
    const int ncoef = (a.l0 + 1) * (a.m0 + 1);
    Plan P;
    auto plan = [&](size_t cap, int t) {
        const Geo g = make_geo(a.np, a.nx, a.ny, t);
        const int hw = (t * g.nseg + per_warp - 1) / per_warp * per_warp;
        return deepest_plan(cap, src_slot_bytes<SHIFT>(g, elem, a.m0), tgt_array_bytes<SHIFT>(g, elem, a.m0), stage_arrays(a.kind),
                            hw, ncoef, P);
    };
    // m0 = 0: half an SM's shared memory, so that two CTAs share it, where the
    // rings fit; otherwise the whole of it, with fewer cells a tile if need be
    if (!(MC == 0 && plan(kSmemHalf, tx))) {
        while (!plan(kSmemMax, tx)) {
            if (tx == 1) return cudaErrorNotSupported;
            --tx;
        }
    }
    const auto kernel = rk_stage_pair_kernel<MC, TS, SHIFT, PT>;
    cudaError_t e = ensure_dyn_smem((const void*)kernel, P.total);
    if (e != cudaSuccess) return e;
    const int threads = P.hw * (32 / per_warp) + 64;
    const long long tiles = tiles_of(tx);
    int per_sm_ctas = 1;
    if (tile_min_blocks<MC>() > 1) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_ctas, kernel, threads, P.total);
        if (e != cudaSuccess || per_sm_ctas < 1) { (void)cudaGetLastError(); per_sm_ctas = 1; }
        if (per_sm_ctas > tile_min_blocks<MC>()) per_sm_ctas = tile_min_blocks<MC>();
    }
    const long long resident = (long long)sm_count() * per_sm_ctas;
    const long long blocks = tiles < resident ? tiles : resident;
    kernel<<<dim3((unsigned)blocks), dim3(threads), P.total, s>>>(a, P, tx);
    return cudaGetLastError();
}

template <typename TS, int MC>
cudaError_t pair_mc(const StageArgs<TS>& a, cudaStream_t s) {
    constexpr int PT = points<MC, TS>();
    if ((a.np * (int)sizeof(TS)) % 16 == 0) return pair_form<MC, TS, false, PT>(a, s);
    // odd rows of at most a cell an SM: the chain of one tile is the launch, and
    // twice the warps of one point a thread are the faster ones (8 x 8 cells, l0 = 6,
    // m0 = 2, a step, one point / two: 33 points 123 / 130 us, 189 points 129 / 132)
    if constexpr (sizeof(TS) == 8 && (MC == 1 || MC == 2)) {
        if (a.cells <= sm_count() && (a.np + 31) / 32 <= consumer_warps<MC, TS>()) return pair_form<MC, TS, true, 1>(a, s);
    }
    return pair_form<MC, TS, true, PT>(a, s);
}

// ---------------------------------------------------------------------------
// a batch of problems with m0 = 0: persistent CTAs walk the (problem, tile)
// list.  Every problem's rows are 16-byte multiples (oshun_batch_create).
//
// An item is one tile of a few harmonics, so what counts is how many items an
// SM has under way: three small CTAs (80 registers a thread) instead of two,
// two points a thread, nothing read from global memory between the ring's
// copies (the descriptor comes with f00, a source's coefficients with its
// slot), E and B updated in the launch.  512 uneven problems, FP32, two steps:
// 15.2 -> 11.6 ms against the one-point kernel (its consumers took 12.9
// thousand cycles an item, 1.9 of them waiting for copies).
// ---------------------------------------------------------------------------
// Descriptors kept in shared memory: the producer is at most kMaxDepth slots,
// two or more of them a tile, ahead of a warp that still reads its tile's.
constexpr int kDescs = 8;
static_assert(kMaxDepth / 2 + 1 < kDescs, "descriptor ring");
constexpr int kBatchWarps = 5;   // consumer warps: 320 points, two a thread

template <typename TS>
__global__ void __launch_bounds__((kBatchWarps + 2) * 32, 3)
    rk_stage_pair_batch_kernel(const __grid_constant__ BatchWork bw, const __grid_constant__ Plan P, const int nc, int* err) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x;
    const int nct = (int)blockDim.x - 64;              // consumer threads
    const int ncw = nct >> 5;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
    auto desc_at = [&](int iter) { return smem + P.off_coef + (size_t)(iter % kDescs) * bw.desc_bytes; };

    for (int i = tid; i < kJBuf * P.hw; i += blockDim.x) reinterpret_cast<int*>(smem + P.off_cnt)[i] = 0;
    if (tid == 0) {
        for (int k = 0; k < kMaxDepth; ++k) {
            mbar_init(bars + k, 1);
            mbar_init(bars + kMaxDepth + k, ncw);
            mbar_init(bars + 2 * kMaxDepth + k, 1);
            mbar_init(bars + 3 * kMaxDepth + k, ncw);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto geo = [&](const StageArgs<TS>& a) { return make_geo(a.np, a.nx, a.ny, batch_cells(a.np, a.nx, nc, bw.tx_cap)); };

    if (tid >= nct) {
        if ((tid & 31) != 0) return;
        const bool sources = tid == nct;
        RingPos r;
        int issued = 0, iter = 0;
        bool ok = true;
        auto desc = [&](int it) { return bw.probs + (size_t)bw.items[it].x * bw.desc_bytes; };
        for (int it = blockIdx.x; it < bw.nitems && ok; it += gridDim.x, ++iter) {
            StageArgs<TS> a = *reinterpret_cast<const StageArgs<TS>*>(desc(it));
            a.hx = nullptr;   // batched problems have no halo columns
            a.m0 = 0;
            const Geo g = geo(a);
            const int tile = bw.items[it].y;
            ok = sources ? produce_sources<TS, false, true>(a, g, P, tile, smem, r, issued, kWaitNs, -1, desc(it),
                                                            (uint32_t)bw.desc_bytes, desc_at(iter))
                         : produce_targets<TS, false>(a, g, P, tile, smem, r, issued, kWaitNs);
        }
        if (!ok) {
            atomicOr(err, 16);
            drain(bars + (sources ? 0 : 2 * kMaxDepth), r, issued, sources ? P.D : P.RD, kWaitNs);
        }
        return;
    }

    Consumer cs;
    cs.start(P, smem);
    for (int it = blockIdx.x; it < bw.nitems; it += gridDim.x) {
        const int tile = bw.items[it].y;
        mbar_wait_or_exit(cs.src.bar, cs.src.phase, err, kWaitNs);   // the descriptor comes with f00
        const StageArgs<TS>& a = *reinterpret_cast<const StageArgs<TS>*>(desc_at(cs.tile_iter));
        consume_tile<0, TS, 2, false, true>(a, nullptr, nullptr, geo(a), P, tile, smem, cs, err, kWaitNs);
    }
}

}  // namespace

void stage_pair_batch_sizes(int np, int nx, int ny, int tx, int elem_bytes, size_t* src_bytes, size_t* tgt_bytes) {
    const Geo g = make_geo(np, nx, ny, tx);
    *src_bytes = align_up(src_slot_bytes<false>(g, elem_bytes, 0), 128) + kCoefBytes;
    *tgt_bytes = tgt_array_bytes<false>(g, elem_bytes, 0);
}

// entry of a batch's coupling table: the factors of one source as the kernel reads them
int stage_pair_coef(const CoefLM& c, int elem_bytes, unsigned char* dst) {
    for (int i = 0; i < 16; ++i) {
        const double v = coef_entry(c, i);
        const float f[2] = {(float)v, (float)v};
        if (elem_bytes == 4) std::memcpy(dst + 8 * i, f, 8);
        else std::memcpy(dst + 8 * i, &v, 8);
    }
    return (int)kCoefBytes;
}

// nc: momentum points (rows rounded up to 32) of a tile
template <typename TS>
cudaError_t launch_stage_pair_batch(const StageArgs<TS>& a1, const BatchWork& bw, int nc, cudaStream_t s) {
    if (nc < 32 || nc > 64 * kBatchWarps || nc % 32) return cudaErrorInvalidValue;
    if (bw.nitems < 1) return cudaSuccess;
    const int hw = (nc / 32 + 1) / 2 * 2, threads = hw * 16 + 64;
    const auto kernel = rk_stage_pair_batch_kernel<TS>;
    // as many CTAs an SM as its registers hold, each with at least five source
    // slots (about a tile of few harmonics): what one CTA waits for, the others hide
    const int desc_units = (int)((kDescs * (size_t)bw.desc_bytes + kCoefBytes - 1) / kCoefBytes);
    Plan P;
    int n = 1;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0);
    if (e != cudaSuccess || n < 1) { (void)cudaGetLastError(); n = 1; }
    for (;; --n) {
        const size_t cap = n > 1 ? (size_t)(228 * 1024) / n - 1024 : kSmemMax;
        if (deepest_plan(cap, bw.pair_src, bw.pair_tgt, stage_arrays(a1.kind), hw, desc_units, P) && (n == 1 || P.D >= 5)) break;
        if (n == 1) return cudaErrorNotSupported;
    }
    e = ensure_dyn_smem((const void*)kernel, P.total);
    if (e != cudaSuccess) return e;
    const long long resident = (long long)sm_count() * n;
    const long long blocks = bw.nitems < resident ? bw.nitems : resident;
    kernel<<<dim3((unsigned)blocks), dim3(threads), P.total, s>>>(bw, P, nc, a1.err);
    return cudaGetLastError();
}
template cudaError_t launch_stage_pair_batch<double>(const StageArgs<double>&, const BatchWork&, int, cudaStream_t);
template cudaError_t launch_stage_pair_batch<float>(const StageArgs<float>&, const BatchWork&, int, cudaStream_t);

// cudaErrorNotSupported when a momentum row does not fit the CTA or its rings
template <typename TS>
cudaError_t launch_stage_pair(const StageArgs<TS>& a, cudaStream_t s) {
    switch (a.m0) {
        case 0: return pair_mc<TS, 0>(a, s);
        case 1: return pair_mc<TS, 1>(a, s);
        case 2: return pair_mc<TS, 2>(a, s);
        case 3: return pair_mc<TS, 3>(a, s);
        case 4: return pair_mc<TS, 4>(a, s);
        case 5: return pair_mc<TS, 5>(a, s);
        case 6: return pair_mc<TS, 6>(a, s);
        case 7: return pair_mc<TS, 7>(a, s);
        case 8: return pair_mc<TS, 8>(a, s);
        default: return cudaErrorNotSupported;
    }
}
template cudaError_t launch_stage_pair<double>(const StageArgs<double>&, cudaStream_t);
template cudaError_t launch_stage_pair<float>(const StageArgs<float>&, cudaStream_t);

}  // namespace oshun
