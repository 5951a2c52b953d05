// Bulk (1D TMA) copies global -> shared with mbarrier completion.
//
// Rules followed by the callers: source and destination 16-byte aligned, size a
// multiple of 16 bytes (block strides are padded to 4 floats); every wait is
// bounded -- on timeout the caller records an error status, waits (bounded
// again) for its own copy in flight and leaves the kernel.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vk {

constexpr int kMbarSpin = 1 << 22;      // try_wait polls before giving up: 16 s (one that fails takes 7 760 cycles)

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One thread: announce `bytes` of transaction and start the copy.
__device__ __forceinline__ void tma_load_1d(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

// At most `polls` looks at phase `parity` of the barrier, none of which suspends.
__device__ __forceinline__ bool mbar_poll(uint64_t *bar, uint32_t parity, int polls) {
    for (int i = 0; i < polls; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}

// Bounded wait for phase `parity` of the barrier; false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    for (int i = 0; i < kMbarSpin; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Copies of 8 bytes that only the issuing thread waits for and reads.
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A double and a tag in two 64-bit words, each of them single-copy atomic: a
// reader of its shared memory that finds the tag in both has the value, and
// the writer in another CTA of the cluster needs no fence.
__device__ __forceinline__ ulonglong2 tagged(double v, unsigned tag) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
    return make_ulonglong2((u & 0xffffffffull) | t, (u >> 32) | t);
}
__device__ __forceinline__ void put_tagged(uint32_t cluster_smem, double v, unsigned tag) {
    const ulonglong2 w = tagged(v, tag);
    asm volatile("st.volatile.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(cluster_smem), "l"(w.x), "l"(w.y) : "memory");
}
__device__ __forceinline__ bool get_tagged(uint32_t smem, double &v, unsigned tag) {
    unsigned long long a, b;
    asm volatile("ld.volatile.shared::cta.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(smem) : "memory");
    v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
    return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

// Padded stride (floats) of an n x n FP32 block so every block starts on 16 bytes.
__host__ __device__ __forceinline__ int block_stride32(int n) { return (n * n + 3) & ~3; }

}  // namespace vk
