// Asynchronous-copy and barrier helpers of the pipelined stage kernels
// (stage_pipe.cuh, stage_pair.cu).
#pragma once

#include <type_traits>
#include <utility>

#include "stage_common.cuh"

namespace oshun {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned long long kWaitNs = 1000000000ull;   // a pipeline wait gives up after 1 s
constexpr int kMaxTx = 8;
constexpr size_t kSmemMax = 227 * 1024;          // dynamic shared memory of one CTA
constexpr size_t kSmemHalf = (228 * 1024 - 2 * 1024) / 2;   // each of two CTAs on one SM (1 KB reserved each)

// cells of a batch's tile: nc points of momentum rows rounded up to 32, tx_cap cells at most
__host__ __device__ inline int batch_cells(int np, int nx, int nc, int tx_cap) {
    const int np_pad = (np + 31) & ~31;
    int tx = nc / np_pad;
    if (tx > tx_cap) tx = tx_cap;
    if (tx > nx) tx = nx;
    return tx < 1 ? 1 : tx;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
    uint32_t done;
    // a non-blocking test of the phase (the caller polls with a time bound);
    // it timed 0.7 % faster per stage than a try_wait that may suspend the thread
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P1;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    return done != 0;
}
// bounded wait for the phase with this parity; false after limit_ns
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          const unsigned long long limit_ns = kWaitNs) {
    const uint32_t addr = smem_u32(bar);
    if (mbar_try(addr, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (mbar_try(addr, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}
// one try of the phase's wait that may hold the thread for a short, bounded
// time, which leaves the issue slots to the other warps
__device__ __forceinline__ bool mbar_hold(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P1;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    return done != 0;
}
// bounded wait by holding tries; false after limit_ns
__device__ __forceinline__ bool mbar_wait_hold(uint64_t* bar, uint32_t parity, const unsigned long long limit_ns) {
    const uint32_t addr = smem_u32(bar);
    if (mbar_hold(addr, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (mbar_hold(addr, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}
// global -> shared bulk copy completing on `bar`; 16-byte aligned, size % 16 == 0
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__host__ __device__ inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

template <int N, typename F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant<int, 0>) ... f(integral_constant<int, N-1>)
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_impl<N>(f, std::make_integer_sequence<int, N>{});
}

}  // namespace
}  // namespace oshun
