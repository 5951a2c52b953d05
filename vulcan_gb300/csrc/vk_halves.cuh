// Work queue over half-columns: the two-sided solves eliminate every column
// from its bottom (layers 0 .. m-1) and its top (layers nz-1 .. m+1) towards
// the middle layer m = nz / 2, and whoever finishes a column's second half does
// its middle.  Unit u is half u & 1 of the column order[u >> 1] (longest first).
// DevBatch::queue holds the next unit and, per column, how many halves are done.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "vk_internal.cuh"
#include "vk_tma.cuh"

namespace vk {

__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// (not the .aligned forms: a warp may arrive diverged)
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// The next of `units` from a counter, -1 when there is none left.  All threads
// call it; in a cluster (CL) every CTA gets rank 0's, -1 too once a CTA that gave
// up a wait has set `lost` (NULL: none) in rank 0's shared memory: its word is
// read between two cluster barriers, so all CTAs leave together.
template <bool CL>
__device__ __forceinline__ int next_unit(unsigned *queue, int units, int *s_unit, int rank, int csize,
                                         const int *lost) {
    if (CL) {
        cluster_sync_all();
        if (rank == 0 && threadIdx.x == 0) {
            const int u = lost && *(const volatile int *)lost ? units : (int)atomicAdd(queue, 1u);
            const uint32_t la = smem_u32(s_unit);
            for (int d = 0; d < csize; ++d)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(la, (uint32_t)d)), "r"(u) : "memory");
        }
        cluster_sync_all();
    } else {
        __syncthreads();
        if (threadIdx.x == 0) *s_unit = (int)atomicAdd(queue, 1u);
        __syncthreads();
    }
    const int u = *s_unit;
    return u < units ? u : -1;
}
template <bool CL>
__device__ __forceinline__ int next_half(const DevBatch &b, int *s_unit, int rank, int csize,
                                         const int *lost = nullptr) {
    return next_unit<CL>(b.queue, 2 * b.ncols, s_unit, rank, csize, lost);
}

// True for the second of a column's halves to get here; what the first wrote
// before is then visible.  All threads call it (in a cluster: of every CTA); a
// cluster that lost a message (`lost` as in next_unit) does not count as there.
template <bool CL>
__device__ __forceinline__ bool second_half(const DevBatch &b, int c, int *s_unit, int rank, int csize,
                                            const int *lost = nullptr) {
    __threadfence();
    if (CL) {
        cluster_sync_all();
        if (rank == 0 && threadIdx.x == 0) {
            const int a = lost && *(const volatile int *)lost ? -1 : (int)atomicAdd(b.queue + 1 + c, 1u);
            __threadfence();
            const uint32_t la = smem_u32(s_unit);
            for (int d = 0; d < csize; ++d)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(la, (uint32_t)d)), "r"(a) : "memory");
        }
        cluster_sync_all();
    } else {
        __syncthreads();
        if (threadIdx.x == 0) {
            *s_unit = (int)atomicAdd(b.queue + 1 + c, 1u);
            __threadfence();
        }
        __syncthreads();
    }
    return *s_unit == 1;
}

// Grid of a half-column kernel: CTAs per SM from vk_set_launch, else the
// batch's override, else the kernel's default; never more than the units.
inline int half_grid(const DevBatch &b, int kernel, int cps_default) {
    const int cps = b.cps_k[kernel] > 0 ? b.cps_k[kernel] : b.cps > 0 ? b.cps : cps_default;
    const long long g = (long long)cps * b.nsm;
    return (g > 0 && g < 2ll * b.ncols) ? (int)g : 2 * b.ncols;
}

// Zero the queue position, the columns' arrival counts and the second position.
inline void reset_queue(const DevBatch &b, cudaStream_t s) {
    cudaMemsetAsync(b.queue, 0, (size_t)(2 + b.ncols) * sizeof(unsigned), s);
}

}  // namespace vk
