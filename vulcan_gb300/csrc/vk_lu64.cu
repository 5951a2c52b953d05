// FP64 block-tridiagonal solve of the Ros2 system, two-sided ("twisted")
// block-Thomas: every column is eliminated from its bottom and from its top at
// once and the halves meet in the middle layer m = nz / 2.  A half-column is
// the unit of work, so a column's chain of dependent layers is half as long
// and the queue balances twice as many, half as long units.
//
//   k_lu64    G_j = D'_j^-1 of every layer.  Bottom half (j = 0 .. m-1):
//               D'_j = D_j - diag(dC_j) G_{j-1} diag(dB_{j-1}),
//             top half (j = nz-1 .. m+1):
//               D'_j = D_j - diag(dB_j) G_{j+1} diag(dC_{j+1});
//             whoever finishes a column's second half inverts its middle
//             layer, which has both terms.  D_j = c0 I - J_j - diag(dA_j).
//   k_sweep64<true>   z_j = G_j (b_j + coupling o z_prev) along both halves; the second
//             half to finish does the middle: x_m = z_m.
//   k_sweep64<false>  x_j = z_j + G_j (coupling o x_next) from the middle outwards.
//
// k_lu64 is bound by the FP64 unit when the columns fill the chip (one
// warp-wide FP64 instruction per 19 cycles and SM, measured) and by the chain
// of dependent pivots (vk_lu64.cuh) when they do not: then the CTAs of a
// cluster share each block.  Measured against the one-sided factorisation,
// one CTA per column, that it replaced (ms, GB300): one CHO column of 100
// layers 6.1 -> 1.4, one NCHO column of 150 layers 21.4 -> 3.7, 64 uneven NCHO
// columns 28.0 -> 10.2, 512 50.6 -> 46.0.  The sweeps are bound by the FP64
// products of a layer and the latency between dependent layers.
//
// Reference: the banded LU of the Ros2 LHS, op.py:2913-2929.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <functional>

#include "vk_internal.cuh"
#include "vk_halves.cuh"
#include "vk_lu64.cuh"
#include "vk_tma.cuh"

namespace vk {

namespace {

constexpr size_t kMaxSmem = 232448;    // dynamic shared memory of a CTA
constexpr int kLongMax = 256;          // most half-columns lu64_long looks at

__host__ __device__ inline size_t lu64_smem(int n, int csize) {
    const int w = lu64_slice_max(n, csize);
    const size_t d = (((size_t)n * w + 1) & ~(size_t)1) + (size_t)(csize > 1 ? n : 2) * lu64_msg(n) + 4 * (size_t)n + 12;
    return d * 8 + (size_t)n * 8 + 4 * (size_t)n * 4 + 64;
}

}  // namespace

namespace {

// This CTA's part of the shared memory at sm and of the blocks (rank of csize).
template <bool CL>
__device__ __forceinline__ Lu64Mem lu64_mem(double *sm, int n, int csize, int rank, int *s_sing, int *s_dead, int *s_lost,
                                            int spin) {
    Lu64Mem m;
    m.n = n;
    m.csize = CL ? csize : 1;
    m.rank = CL ? rank : 0;
    m.pw = lu64_prep_warps(n);
    m.c0 = lu64_slice(n, m.csize, m.rank);
    m.w = lu64_slice(n, m.csize, m.rank + 1) - m.c0;
    m.S = sm;
    m.msg = m.S + ((n * lu64_slice_max(n, m.csize) + 1) & ~1);
    m.srow = m.msg + (CL ? n : 2) * lu64_msg(n);
    m.rowf = m.srow + n;
    m.colf = m.rowf + n;
    m.diag = m.colf + n;
    m.xval = m.diag + n;
    m.xkey = reinterpret_cast<unsigned *>(m.xval + 8);
    m.bar = reinterpret_cast<uint64_t *>(m.xkey + 8);
    m.rowid = reinterpret_cast<int *>(m.bar + n);
    m.colid = m.rowid + n;
    m.perm = m.colid + n;
    m.kinv = m.perm + n;
    m.sing = s_sing;
    m.dead = s_dead;
    m.lost = s_lost;
    m.spin = spin;
    return m;
}

// The half-column u (and the column's middle, if it is the second half).
// DENSE: the blocks are given, jv = D [layer][n][n], and so are the couplings
// (their sign cancels in the Schur terms); the inverses are packed (stride n n).
// mid1: the middle layer, nz / 2 if negative.  phase: inversions so far.
template <bool CL, bool DENSE>
__device__ __forceinline__ void lu64_half(const DevNet &net, const DevBatch &b, const Lu64Mem &m,
                                          const double *__restrict__ jv, const double *__restrict__ dA,
                                          const double *__restrict__ dB, const double *__restrict__ dC,
                                          const double *__restrict__ dt, double *G, int *status, int mid1, int u,
                                          int *s_unit, unsigned &phase) {
    const int n = net.ni, gst = DENSE ? n * n : block_stride64(n);
    const int tid = threadIdx.x, nth = blockDim.x;
    const int w = m.w, c0s = m.c0, ne = n * w;
    int *rowpos = m.perm, *colpos = m.kinv;            // free between inversions
    const int c = b.order[u >> 1], half = u & 1;
    if (b.active && !b.active[c]) return;
    const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = mid1 >= 0 ? mid1 : nz / 2;
    const int cnt = half ? nz - 1 - mid : mid;
    const double cdt = DENSE ? 0.0 : 1.0 / (R_ROS * dt[c]);
    if (tid == 0) *m.sing = 0;
    for (int t = tid; t < n; t += nth) { m.rowid[t] = t; m.colid[t] = t; }
    __syncthreads();
    bool middle = false;
    // t < cnt: the half's layers; t == cnt: the last inverse is stored and,
    // for the second half to get there, the middle layer follows
    for (int t = 0; t <= cnt || middle; ++t) {
        const int j = middle ? mid : (half ? nz - 1 - t : t);
        const size_t l = (size_t)l0 + j;
        const bool build = t < cnt || middle;
        const double *Dl = DENSE ? jv + l * gst : nullptr;
        if (build) {
            const double *rf = half ? dB + l * n : dC + l * n;
            const double *cf = half ? dC + (l + 1) * n : dB + (l - 1) * n;
            for (int q = tid; q < n; q += nth) {
                if (!DENSE) m.diag[q] = cdt - dA[l * n + q];
                if (t > 0 && !middle) {
                    m.rowf[q] = -rf[m.rowid[q]] * m.srow[q];
                    m.colf[q] = cf[m.colid[q]];
                }
            }
        }
        __syncthreads();
        if (middle) {
            // natural order; both neighbours' inverses from global memory
            const double *Gd = G + (l - 1) * gst, *Gu = G + (l + 1) * gst;
            const bool down = mid > 0, up = mid + 1 < nz;
            for (int e = tid; e < ne; e += nth) {
                const int r = e / w, q = c0s + e - r * w;
                double v = down ? -dC[l * n + r] * __ldcg(Gd + r * n + q) * dB[(l - 1) * n + q] : 0.0;
                if (up) v -= dB[l * n + r] * __ldcg(Gu + r * n + q) * dC[(l + 1) * n + q];
                if (DENSE) v += Dl[r * n + q];
                else if (r == q) v += m.diag[r];
                m.S[e] = v;
            }
        } else if (t == 0) {
            if (build) for (int e = tid; e < ne; e += nth) {
                const int r = e / w, q = c0s + e - r * w;
                m.S[e] = DENSE ? Dl[r * n + q] : r == q ? m.diag[r] : 0.0;
            }
        } else {
            // store the previous layer's inverse and replace it by this layer's Schur term
            double *Gp = G + (l + (half ? 1 : -1)) * (long long)gst;
            for (int e = tid; e < ne; e += nth) {
                const int r = e / w, q = c0s + e - r * w;
                const int ri = m.rowid[r], ci = m.colid[q];
                const double s = m.S[e];
                Gp[ri * n + ci] = s * m.srow[r];
                if (build) {
                    double v = s * m.rowf[r] * m.colf[q];
                    if (DENSE) v += Dl[ri * n + ci];
                    else if (ri == ci) v += m.diag[ri];
                    m.S[e] = v;
                }
            }
        }
        if (build) {
            if (!DENSE) {
                for (int q = tid; q < n; q += nth) {
                    rowpos[m.rowid[q]] = q;
                    colpos[m.colid[q]] = q - c0s;
                }
                __syncthreads();
                const double *jl = jv + l * net.nnz;
                for (int e = tid; e < net.nnz; e += nth) {
                    const int q = colpos[net.jcol[e]];
                    if (!CL || (unsigned)q < (unsigned)w) m.S[rowpos[net.jrow[e]] * w + q] += jl[e];
                }
            }
            __syncthreads();
            if (!lu64_invert<CL>(m, phase)) {
                // nothing of this block is stored; the cluster meets where it would have
                if (!middle) second_half<CL>(b, c, s_unit, m.rank, m.csize, m.lost);
                break;
            }
            ++phase;
        }
        if (middle) {
            double *Gl = G + l * gst;
            for (int e = tid; e < ne; e += nth) {
                const int r = e / w, q = c0s + e - r * w;
                Gl[m.rowid[r] * n + m.colid[q]] = m.S[e] * m.srow[r];
            }
            break;
        }
        if (t == cnt) {
            middle = second_half<CL>(b, c, s_unit, m.rank, m.csize, CL ? m.lost : nullptr);
            if (!middle) break;
            for (int q = tid; q < n; q += nth) { m.rowid[q] = q; m.colid[q] = q; }
            __syncthreads();
        }
    }
    if (CL && tid == 0 && *m.dead) atomicExch(&status[c], VK_ETIMEOUT);
    else if (tid == 0 && m.rank == 0 && *m.sing)
        atomicCAS(&status[c], 0, *m.sing == 2 ? VK_ENAN : VK_ESINGULAR);
}

// The message barriers of a cluster.
__device__ __forceinline__ void lu64_open(const Lu64Mem &m) {
    for (int k = threadIdx.x; k < m.n; k += blockDim.x) mbar_init(&m.bar[k], 1);
    mbar_fence_init();
    cluster_sync_all();
}

// The cluster leaves: no message is on its way to a CTA that has left, or whose
// memory has another use from here on.  A CTA that gave up waits, bounded, for
// what was sent to it all the same: messages of the inversion it gave up in,
// and of the next one from a CTA that had all of this one's.
__device__ __forceinline__ void lu64_close(const Lu64Mem &m, unsigned phase) {
    constexpr int kDrainPolls = 1 << 16;   // milliseconds; a message takes microseconds
    if (*m.dead)
        for (int k = threadIdx.x; k < m.n; k += blockDim.x) {
            if (k >= m.c0 && k < m.c0 + m.w) continue;
            if (!mbar_poll(&m.bar[k], phase & 1, kDrainPolls)) continue;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         ::"r"(smem_u32(&m.bar[k])), "r"((uint32_t)lu64_msg(m.n) * 8) : "memory");
            mbar_poll(&m.bar[k], (phase + 1) & 1, kDrainPolls);
        }
    cluster_sync_all();
}

}  // namespace

template <bool CL, bool DENSE>
__global__ void __launch_bounds__(CL ? 384 : 544, CL ? 1 : 2)
k_lu64(DevNet net, DevBatch b, const double *__restrict__ jv, const double *__restrict__ dA,
       const double *__restrict__ dB, const double *__restrict__ dC,
       const double *__restrict__ dt, double *G, int *status, int csize, int mid1) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_unit, s_sing, s_dead, s_lost;
    const Lu64Mem m = lu64_mem<CL>(sm, net.ni, csize, CL ? (int)cluster_rank() : 0, &s_sing, &s_dead, &s_lost, b.spin);
    if (threadIdx.x == 0) s_dead = s_lost = 0;
    if (CL) lu64_open(m);
    unsigned phase = 0;
    for (int u; (u = next_half<CL>(b, &s_unit, m.rank, m.csize, CL ? &s_lost : nullptr)) >= 0;)
        lu64_half<CL, DENSE>(net, b, m, jv, dA, dB, dC, dt, G, status, mid1, u, &s_unit, phase);
    if (CL) lu64_close(m, phase);
}

// Clusters of two: the longest nlong half-columns are each shared by a
// cluster, then every CTA goes on alone (lu64_long).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(544, 1)
k_lu64_long(DevNet net, DevBatch b, const double *__restrict__ jv, const double *__restrict__ dA,
            const double *__restrict__ dB, const double *__restrict__ dC,
            const double *__restrict__ dt, double *G, int *status) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_unit, s_sing, s_dead, s_lost;
    unsigned phase = 0;
    if (threadIdx.x == 0) s_dead = s_lost = 0;
    {
        const Lu64Mem m = lu64_mem<true>(sm, net.ni, 2, (int)cluster_rank(), &s_sing, &s_dead, &s_lost, b.spin);
        lu64_open(m);
        for (int u; (u = next_unit<true>(b.queue, b.nlong, &s_unit, m.rank, 2, &s_lost)) >= 0;)
            lu64_half<true, false>(net, b, m, jv, dA, dB, dC, dt, G, status, -1, u, &s_unit, phase);
        lu64_close(m, phase);
        if (s_lost) return;                // the same in both CTAs: no wait follows next_unit
        // the barriers' memory holds data from here on
        for (int k = threadIdx.x; k < m.n; k += blockDim.x)
            asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(&m.bar[k])) : "memory");
        __syncthreads();
    }
    const Lu64Mem m = lu64_mem<false>(sm, net.ni, 1, 0, &s_sing, &s_dead, &s_lost, 0);
    for (int u; (u = next_unit<false>(b.queue + 1 + b.ncols, 2 * b.ncols - b.nlong, &s_unit, 0, 1, nullptr)) >= 0;)
        lu64_half<false, false>(net, b, m, jv, dA, dB, dC, dt, G, status, -1, b.nlong + u, &s_unit, phase);
}

// One FP64 sweep over half-columns.  FWD: towards the middle,
//   z_j = G_j (rhs_j + coupling o z_prev), the second half to finish adding
//   z_m = G_m (rhs_m + dC_m o z_{m-1} + dB_m o z_{m+1});
// else from the middle outwards, starting at out_m = z_m,
//   out_j = z_j + G_j (coupling o out_prev), optional yk2 = y + out / r.
// A row's product is the same sums in the same order in both kernels below:
// eight parts, part p over the columns p, p + 8, .., combined
// ((p0 + p4) + (p1 + p5)) + ((p2 + p6) + (p3 + p7)).
// The lane that ends up with row r of a result also computes row r of the next
// visit's input, so a visit has one barrier; y + out / r (a division each) is
// formed in a parallel pass after the half.

// y + out / r of the layers [j0, j1) of a half
__device__ __forceinline__ void yk2_pass(size_t e0, int ne, int first, int step, const double *__restrict__ y,
                                         const double *out, double *__restrict__ yk2) {
#pragma unroll 2
    for (int e = first; e < ne; e += step) yk2[e0 + e] = y[e0 + e] + out[e0 + e] / R_ROS;
}

// --- one CTA per half-column, four lanes a row (two parts each).  The
// inverses come by bulk copies in visit order, nbuf in flight, the row vectors
// by cp.async two visits ahead.  Bound by the FP64 unit with many columns
// (two solves of 512 NCHO columns 5.4 -> 5.1 ms against three barriers a visit
// and a division by r in it, 64 columns 1.49 -> 1.12) and by the chain of visits with few.
constexpr int kSweepBars = 8;
__host__ __device__ inline int sweep64_threads(int n) { return (4 * n + 31) / 32 * 32; }
__host__ __device__ inline size_t sweep64_smem(int n, int nbuf) {
    return kSweepBars * 8 + (size_t)(nbuf * block_stride64(n) + 8 * n) * sizeof(double);
}
// Blocks in flight: as many as the CTA's share of the SM holds; one above ~115 species.
inline int sweep64_nbuf(int n, int ctas) {
    int nb = 4;
    while (nb > 1 && ctas * (sweep64_smem(n, nb) + 1100) > 233472) --nb;
    return nb;
}

// Copy k of a CTA's block stream lands in buffer k % nbuf and completes
// phase (k / nbuf) & 1 of that buffer's mbarrier.
__device__ __forceinline__ bool wait_copy(uint64_t *bar, unsigned k, unsigned nbuf) {
    return mbar_wait(&bar[k % nbuf], (k / nbuf) & 1u);
}

// After a bulk copy that never landed: wait (bounded) for the copies still in
// flight, visits [v, last), so none lands in a CTA that has left; the caller
// then records VK_ETIMEOUT and leaves.
__device__ __forceinline__ void drain_copies(uint64_t *bar, unsigned cnt, int v, int last, int nbuf) {
    for (int u = v; u < last; ++u) wait_copy(bar, cnt + (unsigned)u, nbuf);
}

template <bool FWD>
__global__ void __launch_bounds__(640)
k_sweep64(DevNet net, DevBatch b, const double *G, const double *__restrict__ dB,
          const double *__restrict__ dC, const double *__restrict__ rhs, double *z, double *out,
          const double *__restrict__ y, double *__restrict__ yk2, int *__restrict__ status, int nbuf) {
    extern __shared__ __align__(16) unsigned char smb[];
    const int n = net.ni, gst = block_stride64(n);
    const int tid = threadIdx.x, nth = blockDim.x;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smb);      // [nbuf]
    double *Gbuf = reinterpret_cast<double *>(smb + kSweepBars * 8);    // [nbuf][gst]
    double *xs = Gbuf + nbuf * gst;                         // [2][n] inputs of two visits
    double *vec = xs + 2 * n;                               // [3][2][n] (coupling, rhs or z) of three visits
    __shared__ int s_unit;
    const uint32_t bytes = (uint32_t)gst * sizeof(double);
    const int row = tid >> 2, part = tid & 3;
    const bool rowt = row < n, lead = rowt && part == 0;
    if (tid == 0) {
        for (int i = 0; i < nbuf; ++i) mbar_init(&bar[i], 1);
        mbar_fence_init();
    }
    unsigned cnt = 0;              // copies this CTA consumed before the current unit
    for (int u; (u = next_half<false>(b, &s_unit, 0, 1)) >= 0;) {
        const int c = b.order[u >> 1], half = u & 1;
        if (b.active && !b.active[c]) continue;
        const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = nz / 2;
        const int nvis = half ? nz - 1 - mid : mid;
        const int first = FWD ? (half ? nz - 1 : 0) : (half ? mid + 1 : mid - 1);
        const int step = FWD == (half != 0) ? -1 : 1;
        const double *cpl = FWD == (half != 0) ? dB : dC;
        const size_t e1 = ((size_t)l0 + first) * n;         // first layer visited
        const ptrdiff_t es = (ptrdiff_t)step * n;
        auto issue = [&](int v) {                           // thread 0
            const unsigned k = cnt + (unsigned)v, bi = k % (unsigned)nbuf;
            tma_load_1d(Gbuf + bi * gst, G + ((size_t)l0 + first + step * v) * gst, bytes, &bar[bi]);
        };
        // the lead's own vectors: of visit v's result (z) and of the input that follows it
        auto fetch = [&](int v) {
            if (lead && v < nvis) {
                double *s = vec + (v % 3) * 2 * n + row;
                const size_t e = e1 + es * v + row;
                if (v + 1 < nvis) cp_async8(s, cpl + e + es);
                if (!FWD) cp_async8(s + n, z + e);
                else if (v + 1 < nvis) cp_async8(s + n, rhs + e + es);
            }
            cp_async_commit();
        };
        if (tid == 0)
            for (int v = 0; v < nbuf && v < nvis; ++v) issue(v);
        fetch(0);
        fetch(1);
        int p = 0, v = 0, timed_out = 0;
        if (FWD) {
            if (lead && nvis > 0) xs[row] = rhs[e1 + row];
        } else {
            const size_t em = ((size_t)l0 + mid) * n;
            if (lead) {
                const double xv = z[em + row];
                if (half == 0) out[em + row] = xv;
                if (nvis > 0) xs[row] = cpl[e1 + row] * xv;
            }
        }
        // rows of the product of block k with the current input
        auto product = [&](unsigned k) {
            const double *g = Gbuf + (k % (unsigned)nbuf) * gst + row * n, *xin = xs + p * n;
            double a = 0.0, d = 0.0;
            if (rowt) {
                int q = part;
                for (; q + 12 < n; q += 16) {
                    const double g0 = g[q], g1 = g[q + 4], g2 = g[q + 8], g3 = g[q + 12];
                    const double x0 = xin[q], x1 = xin[q + 4], x2 = xin[q + 8], x3 = xin[q + 12];
                    a = __fma_rn(g0, x0, a);
                    d = __fma_rn(g1, x1, d);
                    a = __fma_rn(g2, x2, a);
                    d = __fma_rn(g3, x3, d);
                }
                for (; q < n; q += 8) {
                    a = __fma_rn(g[q], xin[q], a);
                    if (q + 4 < n) d = __fma_rn(g[q + 4], xin[q + 4], d);
                }
            }
            a += d;
            __syncwarp();
            a += __shfl_xor_sync(0xffffffffu, a, 1);
            return a + __shfl_xor_sync(0xffffffffu, a, 2);
        };
        for (; v < nvis; ++v) {
            if (nbuf == 1 && v > 0) {                       // the one buffer, when all have read it
                __syncthreads();
                if (tid == 0) issue(v);
            }
            const bool ok = wait_copy(bar, cnt + (unsigned)v, nbuf);
            if (__syncthreads_or(!ok)) { timed_out = 1; break; }
            if (tid == 0 && nbuf > 1 && v > 0 && v - 1 + nbuf < nvis) issue(v - 1 + nbuf);      // its buffer is free
            cp_async_wait<1>();
            double r = product(cnt + (unsigned)v);
            if (lead) {
                const double *s = vec + (v % 3) * 2 * n + row;
                if (!FWD) r += s[n];
                (FWD ? z : out)[e1 + es * v + row] = r;
                if (v + 1 < nvis) xs[(p ^ 1) * n + row] = FWD ? __fma_rn(s[0], r, s[n]) : s[0] * r;
            }
            p ^= 1;
            fetch(v + 2);
        }
        cp_async_wait<0>();
        if (timed_out) {
            // issued so far: up to visit v - 2 + nbuf, v at least
            const int last = v == 0 || nbuf == 1 ? v + nbuf : v - 1 + nbuf;
            drain_copies(bar, cnt, v, nvis < last ? nvis : last, nbuf);
            if (tid == 0) status[c] = VK_ETIMEOUT;
            return;
        }
        cnt += (unsigned)nvis;
        if (FWD && second_half<false>(b, c, &s_unit, 0, 1)) {
            const size_t e = ((size_t)l0 + mid) * n + row;
            if (tid == 0) tma_load_1d(Gbuf + (cnt % (unsigned)nbuf) * gst, G + ((size_t)l0 + mid) * gst, bytes,
                                      &bar[cnt % (unsigned)nbuf]);
            if (lead) {
                double s = rhs[e];
                if (mid > 0) s = __fma_rn(dC[e], __ldcg(z + e - n), s);
                if (mid + 1 < nz) s = __fma_rn(dB[e], __ldcg(z + e + n), s);
                xs[p * n + row] = s;
            }
            const bool ok = wait_copy(bar, cnt, nbuf);
            if (__syncthreads_or(!ok)) {
                drain_copies(bar, cnt, 0, 1, nbuf);
                if (tid == 0) status[c] = VK_ETIMEOUT;
                return;
            }
            const double r = product(cnt);
            if (lead) z[e] = r;
            cnt += 1;
        }
        if (!FWD && yk2) {
            __syncthreads();
            const int j0 = half ? mid + 1 : 0, j1 = half ? nz : mid + 1;
            yk2_pass(((size_t)l0 + j0) * n, (j1 - j0) * n, tid, nth, y, out, yk2);
        }
    }
}

// --- a cluster per half-column: CTA c has the rows [c n / cs, (c + 1) n / cs),
// eight lanes each (one part), whose blocks a lane copies itself, kSweepAhead
// visits ahead (its own copies need no barrier).  The eight lanes
// send the row of the next input to one CTA each, tagged with the visit: a lane
// waits for the entries it reads, and no barrier is needed.  (Two input buffers
// are enough: a row is sent when all entries of the visit before have been
// read by its warp, and every CTA needs all rows to go on.)
// Results are kept in shared memory for kSweepHist visits: waiting stores to
// global memory would hold up the ones to the cluster.
// Bound by the chain of a visit: n / 8 dependent FMAs, three exchanges and the
// way to the other CTAs.
// Two solves of one NCHO column of 150 layers: 0.89 ms with one CTA per half,
// 0.53 with a cluster barrier a visit, 0.49.
constexpr int kSweepAhead = 4;
constexpr int kSweepHist = 32;          // visits whose results wait in shared memory
__host__ __device__ inline int sweep64c_threads(int n, int cs) { return (8 * lu64_slice_max(n, cs) + 31) / 32 * 32; }
__host__ __device__ inline size_t sweep64c_smem(int n, int cs) {
    return (size_t)(kSweepAhead * ((n + 7) / 8 + 2) * sweep64c_threads(n, cs) + 4 * n +
                    kSweepHist * lu64_slice_max(n, cs)) * sizeof(double);
}

// sgn: sign of the couplings (+1: the solver's, A = D - dC - dB; -1: A = D + lower +
// upper); gst: stride of the blocks; mid1: the middle layer, nz / 2 if negative;
// a column whose blocks were not inverted (status not 0) is left alone if skip -- all
// but VK_ETIMEOUT, which another cluster may be writing here while this one's CTAs
// read it, one before and one after.
template <bool FWD>
__global__ void __launch_bounds__(640)
k_sweep64c(int n, int gst, DevBatch b, const double *G, const double *__restrict__ dB,
           const double *__restrict__ dC, double sgn, const double *__restrict__ rhs, double *z, double *out,
           const double *__restrict__ y, double *__restrict__ yk2, int *status, int csize, int mid1, int skip) {
    extern __shared__ __align__(16) double smc[];
    __shared__ int s_unit, s_dead;
    const int tid = threadIdx.x, nth = blockDim.x, K = (n + 7) / 8;
    double *ring = smc;                                     // [ahead][K][nth] each lane's part of its row
    double *vec = ring + kSweepAhead * K * nth;             // [ahead][2][nth] coupling, rhs or z
    ulonglong2 *xs = reinterpret_cast<ulonglong2 *>(vec + kSweepAhead * 2 * nth);   // [2][n] tagged inputs of two visits
    double *hist = reinterpret_cast<double *>(xs + 2 * n);  // [kSweepHist][rows] results
    const int rank = (int)cluster_rank(), u = (int)blockIdx.x / csize;
    const int r0 = lu64_slice(n, csize, rank), r1 = lu64_slice(n, csize, rank + 1);
    const int row = r0 + (tid >> 3), part = tid & 7;
    const bool rowt = row < r1, lead = rowt && part == 0;
    const int c = b.order[u >> 1], half = u & 1;
    // (the same for every CTA of the cluster)
    const int st = skip ? *(volatile int *)&status[c] : 0;
    if ((b.active && !b.active[c]) || (st != 0 && st != VK_ETIMEOUT)) return;
    const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = mid1 >= 0 ? mid1 : nz / 2;
    const int nvis = half ? nz - 1 - mid : mid;
    const int first = FWD ? (half ? nz - 1 : 0) : (half ? mid + 1 : mid - 1);
    const int step = FWD == (half != 0) ? -1 : 1;
    const double *cpl = FWD == (half != 0) ? dB : dC;
    const size_t e1 = ((size_t)l0 + first) * n;
    const ptrdiff_t es = (ptrdiff_t)step * n;
    const int nfetch = FWD ? nvis + 1 : nvis;               // FWD: the middle's block too
    auto fetch = [&](int v) {
        if (rowt && v < nfetch) {
            const int s = v % kSweepAhead;
            const double *g = G + ((size_t)l0 + first + step * v) * gst + (size_t)row * n + part;
            for (int i = 0; part + 8 * i < n; ++i) cp_async8(ring + (s * K + i) * nth + tid, g + 8 * i);
            if (v < nvis) {
                const size_t e = e1 + es * v + row;
                if (v + 1 < nvis) cp_async8(vec + (s * 2) * nth + tid, cpl + e + es);
                if (!FWD) cp_async8(vec + (s * 2 + 1) * nth + tid, z + e);
                else if (v + 1 < nvis) cp_async8(vec + (s * 2 + 1) * nth + tid, rhs + e + es);
            }
        }
        cp_async_commit();
    };
    for (int v = 0; v < kSweepAhead - 1; ++v) fetch(v);
    if (tid == 0) s_dead = 0;
    for (int t = tid; t < n; t += nth) xs[n + t] = make_ulonglong2(0, 0);
    if (FWD) {
        if (nvis > 0)
            for (int t = tid; t < n; t += nth) xs[t] = tagged(rhs[e1 + t], 1);
    } else {
        const size_t em = ((size_t)l0 + mid) * n;
        if (nvis > 0)
            for (int t = tid; t < n; t += nth) xs[t] = tagged((sgn * cpl[e1 + t]) * z[em + t], 1);
        if (half == 0 && lead) out[em + row] = z[em + row];
    }
    const uint32_t xs0 = smem_u32(xs);
    auto product = [&](int v) {
        const double *g = ring + (v % kSweepAhead) * K * nth + tid;
        const uint32_t xin = xs0 + (uint32_t)((v & 1) * n) * 16u;
        const unsigned tag = (unsigned)v + 1;
        double a = 0.0;
        if (rowt)
            for (int i = 0, q = part; q < n; q += 96, i += 12) {    // twelve entries at a time
                double x[12];
#pragma unroll
                for (int u = 0; u < 12; ++u) x[u] = 0.0;
                for (int tries = b.spin;; --tries) {
                    bool ok = true;
#pragma unroll
                    for (int u = 0; u < 12; ++u)
                        if (q + 8 * u < n) ok &= get_tagged(xin + (uint32_t)(q + 8 * u) * 16u, x[u], tag);
                    if (ok) break;
                    if ((tries & 255) == 0 && (tries <= 0 || *(volatile int *)&s_dead)) {
                        *(volatile int *)&s_dead = 1;
                        break;
                    }
                }
#pragma unroll
                for (int u = 0; u < 12; ++u)
                    if (q + 8 * u < n) a = __fma_rn(g[(i + u) * nth], x[u], a);
            }
        __syncwarp();
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        return a + __shfl_xor_sync(0xffffffffu, a, 2);
    };
    const uint32_t peer = part < csize ? cluster_addr(xs0, (uint32_t)part) : 0u;
    cluster_sync_all();                                     // every CTA of the cluster runs
    for (int v = 0; v < nvis; ++v) {
        cp_async_wait<kSweepAhead - 2>();
        double r = product(v);
        if (rowt) {
            const double *s = vec + (v % kSweepAhead) * 2 * nth + tid;
            if (!FWD) r += s[nth];
            if (v + 1 < nvis && part < csize) {
                const double f = sgn * s[0], xn = FWD ? __fma_rn(f, r, s[nth]) : f * r;
                put_tagged(peer + (uint32_t)(((v + 1) & 1) * n + row) * 16u, xn, (unsigned)v + 2);
            }
            if (part == 0) hist[(v % kSweepHist) * (r1 - r0) + row - r0] = r;
        }
        fetch(v + kSweepAhead - 1);
        if (v + 1 == nvis || (v + 1) % kSweepHist == 0) {
            __syncwarp();
            const int v0 = v - v % kSweepHist;
            if (rowt)
                for (int t = v0 + part; t <= v; t += 8)
                    (FWD ? z : out)[e1 + es * t + row] = hist[(t - v0) * (r1 - r0) + row - r0];
            __syncwarp();
        }
    }
    cp_async_wait<0>();
    if (FWD) {
        if (second_half<true>(b, c, &s_unit, rank, csize)) {
            const size_t em = ((size_t)l0 + mid) * n;
            for (int t = tid; t < n; t += nth) {
                double s = rhs[em + t];
                if (mid > 0) s = __fma_rn(sgn * dC[em + t], __ldcg(z + em - n + t), s);
                if (mid + 1 < nz) s = __fma_rn(sgn * dB[em + t], __ldcg(z + em + n + t), s);
                xs[(nvis & 1) * n + t] = tagged(s, (unsigned)nvis + 1);
            }
            __syncthreads();
            const double r = product(nvis);
            if (lead) z[em + row] = r;
        }
    } else if (yk2) {
        __threadfence();
        cluster_sync_all();
        const int j0 = half ? mid + 1 : 0, j1 = half ? nz : mid + 1;
        const size_t e0 = ((size_t)l0 + j0) * n;
        const int ne = (j1 - j0) * n;
        for (int e = rank * nth + tid; e < ne; e += csize * nth)
            yk2[e0 + e] = y[e0 + e] + __ldcg(out + e0 + e) / R_ROS;
    }
    cluster_sync_all();                                     // no store to a CTA that has left
    if (tid == 0 && s_dead) atomicExch(&status[c], VK_ETIMEOUT);
}

// ---------------------------------------------------------------------------
namespace {
// Launch configuration with clusters of cs CTAs.
struct ClusterLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    ClusterLaunch(int grid, int threads, size_t smem, int cs, cudaStream_t s) {
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cs;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = cs > 1 ? 1 : 0;
    }
};
}  // namespace

// CTAs per half-column.  While the half-columns do not fill the chip, sharing
// each block between the CTAs of a cluster shortens the chain of its pivots
// (one NCHO column: 9.5, 6.7, 4.5 and 3.7 ms with 1, 2, 4 and 8); the line
// lies where every CTA still has an SM of its own, because beyond it the
// shared FP64 units gain nothing (64 columns: 12.2, 12.4, 18.1 and 36.5 ms),
// and where the device holds all the clusters at once: an SM count that a
// GPC does not divide into clusters leaves SMs over (nine columns: 18 clusters of eight
// take two turns, 8.3 ms, 18 of four 4.7).
static int cluster_size(const DevBatch &b, const int *limit, bool (*fits)(int, int), int n) {
    for (int i = 2; i >= 0; --i)
        if (2 * b.ncols <= limit[i] && 2ll * b.ncols * (2 << i) <= b.nsm && fits(n, 2 << i)) return 2 << i;
    return 1;
}
static bool lu64_fits(int n, int cs) { return n >= kLu64MinCluster && lu64_smem(n, cs) <= kMaxSmem; }
// (the sweeps, one NCHO column, two solves: 0.89 ms with one CTA per half, 0.49 with eight)
static bool sweep64_fits(int n, int cs) { return sweep64c_smem(n, cs) <= kMaxSmem; }

template <class K>
static int active_clusters(K *kernel, int threads, size_t smem, int cs) {
    const ClusterLaunch L(cs, threads, smem, cs, nullptr);
    int k = 0;
    if (cudaOccupancyMaxActiveClusters(&k, kernel, &L.cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return k;
}

// Clusters of 2, 4 and 8 CTAs that the current device holds at once (after init_lu64).
void cluster_limits(int n, int lu[3], int sweep[3]) {
    for (int i = 0; i < 3; ++i) {
        const int cs = 2 << i;
        lu[i] = lu64_fits(n, cs) ? active_clusters(k_lu64<true, false>, lu64_threads(n, cs), lu64_smem(n, cs), cs) : 0;
        sweep[i] = sweep64_fits(n, cs)
                       ? active_clusters(k_sweep64c<true>, sweep64c_threads(n, cs), sweep64c_smem(n, cs), cs) : 0;
    }
}

cudaError_t init_lu64(int n) {
    size_t scl = 0, ssc = 0;
    for (int cs = 2; cs <= 8; cs *= 2) {
        if (lu64_fits(n, cs) && lu64_smem(n, cs) > scl) scl = lu64_smem(n, cs);
        if (sweep64_fits(n, cs) && sweep64c_smem(n, cs) > ssc) ssc = sweep64c_smem(n, cs);
    }
    cudaError_t e = raise_smem_limit(k_lu64<false, false>, lu64_smem(n, 1));
    if (e == cudaSuccess && scl) e = raise_smem_limit(k_lu64<true, false>, scl);
    if (e == cudaSuccess && lu64_fits(n, 2)) e = raise_smem_limit(k_lu64_long, std::max(lu64_smem(n, 1), lu64_smem(n, 2)));
    const size_t ssw = sweep64_smem(n, sweep64_nbuf(n, 1));
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64<true>, ssw);
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64<false>, ssw);
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64c<true>, ssc);
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64c<false>, ssc);
    return e;
}

// How many of the half-columns (lengths by decreasing nz, two to a column) a
// cluster should share while every CTA has an SM of its own but not a cluster: the
// number that makes the last CTA finish first, by the steps' costs in cycles (the
// FP64 unit's 19 per warp-wide instruction, and what a step waits for).  NCHO
// columns of 60 to 200 layers, without and with it: 40 columns 12.3 and 8.4 ms, 64
// columns 12.2 and 10.2, 76 columns 12.7 and 10.8.
int lu64_long(int n, int nsm, int clusters2, int ncols, const int *nz) {
    const int units = 2 * ncols, ncl = std::min(clusters2, nsm / 2), lim = kLongMax;
    if (!lu64_fits(n, 2) || units > 2 * ncl || 2 * units <= nsm || units > lim) return 0;
    const int pw = lu64_prep_warps(n);
    const double one = 19. * (n * n / 32. + 3 * pw) + 560, two = 19. * (n * n / 64. + 5 * pw) + 900;
    int best = 0;
    double tbest = 0;
    double cl[kLongMax], cta[2 * kLongMax];
    // to whoever is free first (v a heap, the earliest on top)
    auto assign = [](double *v, int k, double cost) {
        std::pop_heap(v, v + k, std::greater<double>());
        v[k - 1] += cost;
        std::push_heap(v, v + k, std::greater<double>());
    };
    for (int a = 0; a <= units; a += 4) {
        std::fill(cl, cl + ncl, 0.);
        for (int u = 0; u < a; ++u) assign(cl, ncl, two * (nz[u / 2] / 2));
        for (int i = 0; i < 2 * ncl; ++i) cta[i] = cl[i / 2];
        std::make_heap(cta, cta + 2 * ncl, std::greater<double>());
        for (int u = a; u < units; ++u) assign(cta, 2 * ncl, one * (nz[u / 2] / 2));
        const double t = *std::max_element(cta, cta + 2 * ncl);
        if (a == 0 || t < 0.97 * tbest) { tbest = t; best = a; }
    }
    return best;
}

void launch_lu64(const DevNet &net, const DevBatch &b, const Work &w, cudaStream_t s) {
    const int n = net.ni, cs = cluster_size(b, b.ncl_lu, lu64_fits, n);
    reset_queue(b, s);
    // (whatever CTAs per SM are set: lu64_long shares halves only where each has an SM to itself)
    if (b.nlong > 0 && cs == 1) {
        const ClusterLaunch L(std::min(b.ncl_lu[0], b.nsm / 2) * 2, lu64_threads(n, 1),
                              std::max(lu64_smem(n, 1), lu64_smem(n, 2)), 1, s);
        cudaLaunchKernelEx(&L.cfg, k_lu64_long, net, b, (const double *)w.jv, (const double *)w.dA,
                           (const double *)w.dB, (const double *)w.dC, (const double *)w.dt, w.G, w.status);
        return;
    }
    const ClusterLaunch L(cs == 1 ? half_grid(b, VK_TUNE_LU64, 2) : 2 * b.ncols * cs, lu64_threads(n, cs),
                          lu64_smem(n, cs), cs, s);
    cudaLaunchKernelEx(&L.cfg, cs == 1 ? k_lu64<false, false> : k_lu64<true, false>, net, b, (const double *)w.jv,
                       (const double *)w.dA, (const double *)w.dB, (const double *)w.dC, (const double *)w.dt, w.G,
                       w.status, cs, -1);
}

template <bool FWD>
static void launch_sweep64(const DevNet &net, const DevBatch &b, const double *G, const double *dB, const double *dC,
                           const double *rhs, double *z, double *x, const double *y, double *yk2, int *status,
                           cudaStream_t s) {
    const int n = net.ni, cs = cluster_size(b, b.ncl_sweep, sweep64_fits, n);
    reset_queue(b, s);
    if (cs > 1) {
        const ClusterLaunch L(2 * b.ncols * cs, sweep64c_threads(n, cs), sweep64c_smem(n, cs), cs, s);
        cudaLaunchKernelEx(&L.cfg, k_sweep64c<FWD>, n, block_stride64(n), b, G, dB, dC, 1.0, rhs, z, x, y, yk2,
                           status, cs, -1, 0);
        return;
    }
    const int nbuf = sweep64_nbuf(n, 2 * b.ncols <= b.nsm ? 1 : 2);
    k_sweep64<FWD><<<half_grid(b, VK_TUNE_SWEEP64, 2), sweep64_threads(n), sweep64_smem(n, nbuf), s>>>(
        net, b, G, dB, dC, rhs, z, x, y, yk2, status, nbuf);
}

void launch_fwd64(const DevNet &net, const DevBatch &b, const double *G, const double *dB,
                  const double *dC, const double *rhs, double *z, int *status, cudaStream_t s) {
    launch_sweep64<true>(net, b, G, dB, dC, rhs, z, nullptr, nullptr, nullptr, status, s);
}

void launch_back64(const DevNet &net, const DevBatch &b, const double *G, const double *dB,
                   const double *dC, double *z, double *x, const double *y, double *yk2, int *status,
                   cudaStream_t s) {
    launch_sweep64<false>(net, b, G, dB, dC, nullptr, z, x, y, yk2, status, s);
}

// ---------------------------------------------------------------------------
// One column whose blocks and couplings are given (vk_block_solve_noalloc).

__global__ void k_solve64_words(int nz, int *words) {
    words[0] = 0;                          // order
    words[1] = 0;                          // col_off
    words[2] = nz;                         // col_end
    words[3] = 0;                          // status
    for (int i = 4; i < kSolve64Words; ++i) words[i] = 0;       // queues of the two launches
}

// Such a system may be one that only the elimination from the bottom solves
// well: where a Schur term from the top, up_j G_{j+1} lo_{j+1}, exceeds 4 times the
// largest |D_j| of its row, its rounding errors drown the block's digits, and the
// status becomes kSolve64Grew.  (A step's own blocks have no such growth: the terms
// stay below the rows' largest entries, from 1e-28 of them at dt = 1e-10 s to 0.87 at
// 1e9 s.)  A warp per row of the layers that have such a term; one pass over half
// of D and G: 0.014 of 3.72 ms for 150 layers of 69 species.
__global__ void __launch_bounds__(256)
k_solve64_growth(int nz, int n, const double *__restrict__ D, const double *__restrict__ lo,
                 const double *__restrict__ up, const double *__restrict__ G, int *status) {
    const int j0 = nz / 2, rows = (nz - 1 - j0) * n, lane = threadIdx.x & 31, step = gridDim.x * 8;
    for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < rows; i += step) {
        const int j = j0 + i / n, r = i % n;
        const double *Dr = D + ((size_t)j * n + r) * n, *Gr = G + ((size_t)(j + 1) * n + r) * n;
        const double *l1 = lo + (size_t)(j + 1) * n;
        const double u = up[(size_t)j * n + r];
        double d = 0.0, g = 0.0;
        for (int q = lane; q < n; q += 32) {
            d = fmax(d, fabs(Dr[q]));
            g = fmax(g, fabs(u * Gr[q] * l1[q]));
        }
        for (int o = 16; o; o >>= 1) {
            d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
            g = fmax(g, __shfl_xor_sync(0xffffffffu, g, o));
        }
        if (lane == 0 && g > 4.0 * d) atomicCAS(status, 0, kSolve64Grew);
    }
}

// A small system in one launch: one CTA factorises from the bottom (words and G
// stay its own) and does both sweeps, a warp per row.
__global__ void __launch_bounds__(544)
k_solve64_small(int nz, int n, const double *__restrict__ D, const double *__restrict__ lo,
                const double *__restrict__ up, const double *rhs, double *x, double *G, double *z, int *words) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_unit, s_sing, s_dead, s_lost;
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31;
    if (tid < kSolve64Words) words[tid] = tid == 2 ? nz : 0;    // order, col_off, col_end, status, queue
    __syncthreads();
    DevNet net = {};
    net.ni = n;
    DevBatch b = {};
    b.ncols = 1;
    b.order = words;
    b.col_off = words + 1;
    b.col_end = words + 2;
    b.queue = reinterpret_cast<unsigned *>(words + 4);
    const Lu64Mem m = lu64_mem<false>(sm, n, 1, 0, &s_sing, &s_dead, &s_lost, 0);
    unsigned phase = 0;
    for (int u = 0; u < 2; ++u) {          // the layers below the last one, the last one
        lu64_half<false, true>(net, b, m, D, nullptr, up, lo, nullptr, G, words + 3, nz - 1, u, &s_unit, phase);
        __syncthreads();
    }
    double *v = sm;                        // [n] the product's input
    auto product = [&](int j, int r) {
        const double *g = G + ((size_t)j * n + r) * n;
        double s = 0.0;
        for (int q = lane; q < n; q += 32) s = __fma_rn(g[q], v[q], s);
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    const int warp = tid >> 5, nwarp = nth >> 5;
    for (int j = 0; j < nz; ++j) {
        const size_t e = (size_t)j * n;
        for (int t = tid; t < n; t += nth) v[t] = j ? __fma_rn(-lo[e + t], z[e - n + t], rhs[e + t]) : rhs[t];
        __syncthreads();
        for (int r = warp; r < n; r += nwarp) {
            const double s = product(j, r);
            if (lane == 0) z[e + r] = s;
        }
        __syncthreads();
    }
    for (int j = nz - 1; j >= 0; --j) {
        const size_t e = (size_t)j * n;
        for (int t = tid; t < n && j + 1 < nz; t += nth) v[t] = -up[e + t] * x[e + n + t];
        __syncthreads();
        for (int r = warp; r < n; r += nwarp) {
            const double s = j + 1 < nz ? product(j, r) : 0.0;
            if (lane == 0) x[e + r] = z[e + r] + s;
        }
        __syncthreads();
    }
}
// Where the four or five launches of the general form take longer than the layers
// (us a call, this kernel and the general one: 1 layer of 1 species 26 and 37, 8 of 4 65
// and 70, 3 of 16 65 and 70, 2 of 24 63 and 81; 12 of 4 88 and 82, 6 of 16 112 and 96, 3 of 24
// 88 and 81).
bool solve64_small(int nz, int n) { return n <= 32 && nz <= 8 && nz * n <= 48; }

cudaError_t init_solve64(int nmax) {
    size_t scl = 0, ssc = 0;
    for (int n = 1; n <= nmax; ++n) {
        if (lu64_fits(n, 8) && lu64_smem(n, 8) > scl) scl = lu64_smem(n, 8);
        if (sweep64c_smem(n, 8) > ssc) ssc = sweep64c_smem(n, 8);
    }
    cudaError_t e = raise_smem_limit(k_lu64<false, true>, lu64_smem(nmax, 1));
    if (e == cudaSuccess) e = raise_smem_limit(k_lu64<true, true>, scl);
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64c<true>, ssc);
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64c<false>, ssc);
    if (e == cudaSuccess) e = raise_smem_limit(k_solve64_small, lu64_smem(nmax, 1));
    return e;
}

// G: nz n n doubles, z: nz n, words: kSolve64Words ints, words[3] the status.
cudaError_t launch_solve64(int nz, int n, const double *D, const double *lo, const double *up, const double *rhs,
                           double *x, double *G, double *z, int *words, int mid, cudaStream_t s) {
    if (mid == nz - 1 && solve64_small(nz, n)) {
        k_solve64_small<<<1, lu64_threads(n, 1), lu64_smem(n, 1), s>>>(nz, n, D, lo, up, rhs, x, G, z, words);
        return cudaGetLastError();
    }
    DevNet net = {};
    net.ni = n;
    DevBatch b = {};
    b.ncols = 1;
    b.L = nz;
    b.order = words;
    b.col_off = words + 1;
    b.col_end = words + 2;
    b.queue = reinterpret_cast<unsigned *>(words + 4);
    b.spin = kMbarSpin;
    int *status = words + 3;
    k_solve64_words<<<1, 1, 0, s>>>(nz, words);
    const int cl = lu64_fits(n, 8) ? 8 : 1;
    const ClusterLaunch A(2 * cl, lu64_threads(n, cl), lu64_smem(n, cl), cl, s);
    cudaError_t e = cudaLaunchKernelEx(&A.cfg, cl > 1 ? k_lu64<true, true> : k_lu64<false, true>, net, b, D,
                                       (const double *)nullptr, up, lo, (const double *)nullptr, G, status, cl, mid);
    if (e != cudaSuccess) return e;
    if (mid < 0) {
        const int rows = (nz - 1 - nz / 2) * n;
        k_solve64_growth<<<std::min((rows + 7) / 8, 1024), 256, 0, s>>>(nz, n, D, lo, up, G, status);
    }
    const ClusterLaunch S(16, sweep64c_threads(n, 8), sweep64c_smem(n, 8), 8, s);
    b.queue += 2;
    e = cudaLaunchKernelEx(&S.cfg, k_sweep64c<true>, n, n * n, b, (const double *)G, up, lo, -1.0, rhs, z,
                           (double *)nullptr, (const double *)nullptr, (double *)nullptr, status, 8, mid, 1);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernelEx(&S.cfg, k_sweep64c<false>, n, n * n, b, (const double *)G, up, lo, -1.0,
                              (const double *)nullptr, z, x, (const double *)nullptr, (double *)nullptr,
                              status, 8, mid, 1);
}

}  // namespace vk
