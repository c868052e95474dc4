// Inline-PTX helpers for sm_100a kernels: shared-memory addresses, the global
// timer, mbarriers with bounded waits, and TMA tensor loads (no multicast).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace oflow {

// Longest a kernel waits on an mbarrier before it reports an error.
constexpr unsigned long long kWaitNs = 1000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Asynchronous copies to shared memory (waited for by cp.async.wait_*); !ok: zero
// fill, src is not read.  _l1: through L1, for lines that other blocks of the SM or
// later copies read again.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool ok) {
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async16_l1(uint32_t dst, const void *src, bool ok) {
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void *src, bool ok) {
    const int n = ok ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}

// Two neighbouring float2 at q, past L1 (vec: 16-byte aligned); in0, in1: which are
// inside the level.
__device__ __forceinline__ float4 ld_two(const float2 *p, size_t q, int vec, bool in0, bool in1) {
    if (vec) return in0 ? __ldcg(reinterpret_cast<const float4 *>(p + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 z = make_float2(0.f, 0.f);
    const float2 a = in0 ? __ldcg(p + q) : z, b = in1 ? __ldcg(p + q + 1) : z;
    return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

// Makes mbarrier initialisation visible to the async proxy (TMA, tcgen05).
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity to complete; false after kWaitNs.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer();
    while (!mbar_try_wait(bar, parity))
        if (globaltimer() - t0 > kWaitNs) return false;
    return true;
}

// One arrival that also expects `bytes` of asynchronous transactions.
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
}

// All threads of the cluster meet; what they wrote to shared memory before is
// visible to each other after.
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// A load from the shared memory of block `rank` of the cluster, and a store to it, at
// the address a has in this block.
__device__ __forceinline__ float4 cluster_ld4(uint32_t a, int rank) {
    float4 v;
    asm volatile(
        "{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %4, %5;\n\t"
        "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [r];\n\t}\n"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "r"(a), "r"(rank)
        : "memory");
    return v;
}
__device__ __forceinline__ void cluster_st1(uint32_t a, int rank, int v) {
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\tst.shared::cluster.s32 [r], %2;\n\t}\n" ::"r"(a),
                 "r"(rank), "r"(v)
                 : "memory");
}

__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}

// Untiled copy of `bytes` (a multiple of 16; both addresses 16-byte aligned)
// into shared memory, completing on `bar`.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Tiled TMA loads of one box into shared memory, completing on `bar`.  The
// innermost coordinate times the element size must be a multiple of 16 bytes;
// other coordinates may be negative or past the end (zero fill).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

}  // namespace oflow
