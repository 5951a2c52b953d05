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
//   k_fwd64   z_j = G_j (b_j + coupling o z_prev) along both halves; the second
//             half to finish does the middle: x_m = z_m.
//   k_back64  x_j = z_j + G_j (coupling o x_next) from the middle outwards.
//
// k_lu64 is bound by the FP64 unit when the columns fill the chip (one
// warp-wide FP64 instruction per 19 cycles and SM, measured) and by the chain
// of dependent pivots (vk_lu64.cuh) when they do not: then the CTAs of a
// cluster share each block.  Measured against the one-sided factorisation,
// one CTA per column, that it replaced (ms, GB300): one CHO column of 100
// layers 6.1 -> 1.6, one NCHO column of 150 layers 21.4 -> 4.4, 64 uneven NCHO
// columns 28.0 -> 12.5, 512 50.6 -> 49.4.  The sweeps are bound by the FP64
// products of a layer and the latency between dependent layers.
//
// Reference: the banded LU of the Ros2 LHS, op.py:2913-2929.
#include <cuda_runtime.h>
#include <math.h>

#include "vk_internal.cuh"
#include "vk_gj.cuh"
#include "vk_halves.cuh"
#include "vk_lu64.cuh"
#include "vk_tma.cuh"

namespace vk {

namespace {

__host__ __device__ inline size_t lu64_smem(int n, int csize) {
    const int w = lu64_slice_max(n, csize);
    const size_t d = (((size_t)n * w + 1) & ~(size_t)1) + (size_t)(csize > 1 ? n : 2) * lu64_msg(n) + 4 * (size_t)n + 12;
    return d * 8 + (size_t)n * 8 + 4 * (size_t)n * 4 + 64;
}

}  // namespace

template <bool CL>
__global__ void __launch_bounds__(352, CL ? 1 : 2)
k_lu64(DevNet net, DevBatch b, const double *__restrict__ jv, const double *__restrict__ dA,
       const double *__restrict__ dB, const double *__restrict__ dC,
       const double *__restrict__ dt, double *G, int *status, int csize) {
    extern __shared__ __align__(16) double sm[];
    __shared__ int s_unit, s_sing, s_dead;
    const int n = net.ni, gst = block_stride64(n);
    const int tid = threadIdx.x, nth = blockDim.x;
    Lu64Mem m;
    m.n = n;
    m.csize = CL ? csize : 1;
    m.rank = CL ? (int)cluster_rank() : 0;
    m.pw = lu64_prep_warps(n);
    m.c0 = lu64_slice(n, m.csize, m.rank);
    m.w = lu64_slice(n, m.csize, m.rank + 1) - m.c0;
    m.S = sm;
    m.msg = m.S + ((n * lu64_slice_max(n, m.csize) + 1) & ~1);
    m.srow = m.msg + (CL ? n : 2) * lu64_msg(n);
    double *rowf = m.srow + n;             // [n] row factors of the Schur term, by stored row
    double *colf = rowf + n;               // [n] column factors, by stored column
    double *diag = colf + n;               // [n] c0 - dA, by species
    m.xval = diag + n;
    m.xkey = reinterpret_cast<unsigned *>(m.xval + 8);
    m.bar = reinterpret_cast<uint64_t *>(m.xkey + 8);
    m.rowid = reinterpret_cast<int *>(m.bar + n);
    m.colid = m.rowid + n;
    m.perm = m.colid + n;
    m.kinv = m.perm + n;
    m.sing = &s_sing;
    m.dead = &s_dead;
    const int w = m.w, c0s = m.c0, ne = n * w;
    int *rowpos = m.perm, *colpos = m.kinv;            // free between inversions
    if (tid == 0) s_dead = 0;
    if (CL) {
        for (int k = tid; k < n; k += nth) mbar_init(&m.bar[k], 1);
        mbar_fence_init();
        cluster_sync_all();
    }
    unsigned phase = 0;
    for (int u; (u = next_half<CL>(b, &s_unit, m.rank, m.csize)) >= 0;) {
        const int c = b.order[u >> 1], half = u & 1;
        if (b.active && !b.active[c]) continue;
        const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = nz / 2;
        const int cnt = half ? nz - 1 - mid : mid;
        const double cdt = 1.0 / (R_ROS * dt[c]);
        if (tid == 0) s_sing = 0;
        for (int t = tid; t < n; t += nth) { m.rowid[t] = t; m.colid[t] = t; }
        __syncthreads();
        bool middle = false;
        // t < cnt: the half's layers; t == cnt: the last inverse is stored and,
        // for the second half to get there, the middle layer follows
        for (int t = 0; t <= cnt || middle; ++t) {
            const int j = middle ? mid : (half ? nz - 1 - t : t);
            const size_t l = (size_t)l0 + j;
            const bool build = t < cnt || middle;
            if (build) {
                const double *rf = half ? dB + l * n : dC + l * n;
                const double *cf = half ? dC + (l + 1) * n : dB + (l - 1) * n;
                for (int q = tid; q < n; q += nth) {
                    diag[q] = cdt - dA[l * n + q];
                    if (t > 0 && !middle) {
                        rowf[q] = -rf[m.rowid[q]] * m.srow[q];
                        colf[q] = cf[m.colid[q]];
                    }
                }
            }
            __syncthreads();
            if (middle) {
                // natural order; both neighbours' inverses from global memory
                const double *Gd = G + (l - 1) * gst, *Gu = G + (l + 1) * gst;
                const bool up = mid + 1 < nz;
                for (int e = tid; e < ne; e += nth) {
                    const int r = e / w, q = c0s + e - r * w;
                    double v = -dC[l * n + r] * __ldcg(Gd + r * n + q) * dB[(l - 1) * n + q];
                    if (up) v -= dB[l * n + r] * __ldcg(Gu + r * n + q) * dC[(l + 1) * n + q];
                    if (r == q) v += diag[r];
                    m.S[e] = v;
                }
            } else if (t == 0) {
                if (build) for (int e = tid; e < ne; e += nth) {
                    const int r = e / w, q = c0s + e - r * w;
                    m.S[e] = r == q ? diag[r] : 0.0;
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
                        double v = s * rowf[r] * colf[q];
                        if (ri == ci) v += diag[ri];
                        m.S[e] = v;
                    }
                }
            }
            if (build) {
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
                __syncthreads();
                lu64_invert<CL>(m, phase);
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
                middle = second_half<CL>(b, c, &s_unit, m.rank, m.csize);
                if (!middle) break;
                for (int q = tid; q < n; q += nth) { m.rowid[q] = q; m.colid[q] = q; }
                __syncthreads();
            }
        }
        if (tid == 0 && s_dead) atomicExch(&status[c], VK_ETIMEOUT);
        else if (tid == 0 && m.rank == 0 && s_sing)
            atomicCAS(&status[c], 0, s_sing == 2 ? VK_ENAN : VK_ESINGULAR);
    }
    if (CL) cluster_sync_all();            // no message is still on its way to a CTA that has left
}

// Shared memory of the FP64 sweeps: the mbarriers, nbuf blocks of the padded
// stride, two vectors and the product's partial sums.
constexpr int kSweepBars = 12;
static __host__ __device__ inline size_t sweep64_smem(int n, int nth, int nbuf) {
    return kSweepBars * 8 + (size_t)(nbuf * block_stride64(n) + 2 * n + (nth > n ? nth : n)) * sizeof(double);
}
// Blocks in flight: as many as the CTA's share of the SM holds (a bulk copy of a
// block takes longer than the product that uses it); one above ~115 species.
static inline int sweep64_nbuf(int n, int ctas) {
    int nb = kSweepBars;
    while (nb > 1 && ctas * (sweep64_smem(n, 256, nb) + 1024) > 233472) --nb;
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

// One sweep over half-columns.  FWD: towards the middle,
//   z_j = G_j (rhs_j + coupling o z_prev), the second half to finish adding
//   z_m = G_m (rhs_m + dC_m o z_{m-1} + dB_m o z_{m+1});
// else from the middle outwards, starting at out_m = z_m,
//   out_j = z_j + G_j (coupling o out_prev), optional yk2 = y + out / r.
// The inverses stream into shared memory by bulk copies in visit order, nbuf
// in flight.
template <bool FWD>
__global__ void __launch_bounds__(256)
k_sweep64(DevNet net, DevBatch b, const double *G, const double *__restrict__ dB,
          const double *__restrict__ dC, const double *__restrict__ rhs, double *z, double *out,
          const double *__restrict__ y, double *__restrict__ yk2, int *__restrict__ status, int nbuf) {
    extern __shared__ __align__(16) unsigned char smb[];
    const int n = net.ni, gst = block_stride64(n);
    const int tid = threadIdx.x, nth = blockDim.x;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smb);      // [nbuf]
    double *Gbuf = reinterpret_cast<double *>(smb + kSweepBars * 8);    // [nbuf][gst]
    double *xs = Gbuf + nbuf * gst;                         // [n] input of the visit
    double *xn = xs + n;                                    // [n] its result
    double *part = xn + n;                                  // [max(nth, n)]
    __shared__ int s_unit;
    const uint32_t bytes = (uint32_t)gst * sizeof(double);
    if (tid == 0) {
        for (int i = 0; i < nbuf; ++i) mbar_init(&bar[i], 1);
        mbar_fence_init();
    }
    unsigned cnt = 0;              // copies this CTA consumed before the current unit
    for (int u; (u = next_half<false>(b, &s_unit, 0, 1)) >= 0;) {
        const int c = b.order[u >> 1], half = u & 1;
        if (b.active && !b.active[c]) continue;
        const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = nz / 2;
        int nvis = half ? nz - 1 - mid : mid;
        auto layer_of = [&](int v) {
            if (FWD) return half ? nz - 1 - v : v;
            return half ? mid + 1 + v : mid - 1 - v;
        };
        auto issue = [&](int v, int j) {                    // thread 0
            const unsigned k = cnt + (unsigned)v, bi = k % (unsigned)nbuf;
            tma_load_1d(Gbuf + bi * gst, G + ((size_t)l0 + j) * gst, bytes, &bar[bi]);
        };
        if (tid == 0)
            for (int v = 0; v < nbuf && v < nvis; ++v) issue(v, layer_of(v));
        if (!FWD) {
            const size_t l = (size_t)l0 + mid;
            for (int t = tid; t < n; t += nth) {
                const double xv = z[l * n + t];
                xn[t] = xv;
                if (half == 0) {
                    out[l * n + t] = xv;
                    if (yk2) yk2[l * n + t] = y[l * n + t] + xv / R_ROS;
                }
            }
            __syncthreads();
        }
        int v = 0, timed_out = 0;
        for (; v < nvis; ++v) {
            const int j = layer_of(v);
            const size_t l = (size_t)l0 + j;
            // the input: this thread's xn entry is the one it wrote itself (FWD:
            // it reads the previous result, visible since the product's barrier)
            for (int t = tid; t < n; t += nth) {
                if (FWD) {
                    const double cpl = v == 0 ? 0.0 : (half ? dB[l * n + t] : dC[l * n + t]) * xn[t];
                    xs[t] = rhs[l * n + t] + cpl;
                } else {
                    xs[t] = (half ? dC[l * n + t] : dB[l * n + t]) * xn[t];
                }
            }
            const unsigned k = cnt + (unsigned)v;
            const bool ok = wait_copy(bar, k, nbuf);
            if (__syncthreads_or(!ok)) { timed_out = 1; break; }
            matvec_f64(Gbuf + (k % (unsigned)nbuf) * gst, n, xs, part, xn, FWD ? nullptr : z + l * n);
            if (tid == 0 && v + nbuf < nvis) issue(v + nbuf, layer_of(v + nbuf));   // the buffer just read is free
            for (int t = tid; t < n; t += nth) {
                const double xv = xn[t];
                if (FWD) {
                    z[l * n + t] = xv;
                } else {
                    out[l * n + t] = xv;
                    if (yk2) yk2[l * n + t] = y[l * n + t] + xv / R_ROS;
                }
            }
        }
        if (timed_out) {
            drain_copies(bar, cnt, v, nvis < v + nbuf ? nvis : v + nbuf, nbuf);
            if (tid == 0) status[c] = VK_ETIMEOUT;
            return;
        }
        cnt += (unsigned)nvis;
        if (FWD && second_half<false>(b, c, &s_unit, 0, 1)) {
            const size_t l = (size_t)l0 + mid;
            if (tid == 0) issue(0, mid);
            for (int t = tid; t < n; t += nth) {
                double s = rhs[l * n + t] + dC[l * n + t] * __ldcg(z + (l - 1) * n + t);
                if (mid + 1 < nz) s += dB[l * n + t] * __ldcg(z + (l + 1) * n + t);
                xs[t] = s;
            }
            const bool ok = wait_copy(bar, cnt, nbuf);
            if (__syncthreads_or(!ok)) {
                drain_copies(bar, cnt, 0, 1, nbuf);
                if (tid == 0) status[c] = VK_ETIMEOUT;
                return;
            }
            matvec_f64(Gbuf + (cnt % (unsigned)nbuf) * gst, n, xs, part, xn, nullptr);
            for (int t = tid; t < n; t += nth) z[l * n + t] = xn[t];
            cnt += 1;
        }
    }
}

// ---------------------------------------------------------------------------
// CTAs per half-column.  While the half-columns do not fill the chip, sharing
// each block between the CTAs of a cluster shortens the chain of its pivots
// (one NCHO column: 9.8, 6.5, 5.0 and 4.4 ms with 1, 2, 4 and 8); the line
// lies where every CTA still has an SM of its own, because beyond it the
// shared FP64 units gain nothing (64 columns: 12.5, 12.4, 18.1 and 36.5 ms).
static int lu64_cluster(const DevBatch &b, int n) {
    if (n < kLu64MinCluster) return 1;
    for (int cs = 8; cs > 1; cs /= 2)
        if (2ll * b.ncols * cs <= b.nsm && lu64_smem(n, cs) <= 232448) return cs;
    return 1;
}

cudaError_t init_lu64(int n) {
    size_t scl = 0;
    for (int cs = 2; cs <= 8; cs *= 2)
        if (n >= kLu64MinCluster && lu64_smem(n, cs) <= 232448 && lu64_smem(n, cs) > scl) scl = lu64_smem(n, cs);
    cudaError_t e = raise_smem_limit(k_lu64<false>, lu64_smem(n, 1));
    if (e == cudaSuccess && scl) e = raise_smem_limit(k_lu64<true>, scl);
    const size_t ssw = sweep64_smem(n, 256, sweep64_nbuf(n, 1));
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64<true>, ssw);
    if (e == cudaSuccess) e = raise_smem_limit(k_sweep64<false>, ssw);
    return e;
}

void launch_lu64(const DevNet &net, const DevBatch &b, const Work &w, cudaStream_t s) {
    const int n = net.ni, cs = lu64_cluster(b, n);
    reset_queue(b, s);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3((unsigned)lu64_threads(n));
    cfg.dynamicSmemBytes = lu64_smem(n, cs);
    cfg.stream = s;
    if (cs == 1) {
        cfg.gridDim = dim3((unsigned)half_grid(b, VK_TUNE_LU64, 2));
        cudaLaunchKernelEx(&cfg, k_lu64<false>, net, b, (const double *)w.jv, (const double *)w.dA,
                           (const double *)w.dB, (const double *)w.dC, (const double *)w.dt, w.G,
                           w.status, 1);
        return;
    }
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)(2 * b.ncols * cs));
    cudaLaunchKernelEx(&cfg, k_lu64<true>, net, b, (const double *)w.jv, (const double *)w.dA,
                       (const double *)w.dB, (const double *)w.dC, (const double *)w.dt, w.G, w.status,
                       cs);
}

// CTAs of a sweep an SM should hold
static int sweep64_ctas(const DevBatch &b) { return 2 * b.ncols <= b.nsm ? 1 : 2; }

void launch_fwd64(const DevNet &net, const DevBatch &b, const double *G, const double *dB,
                  const double *dC, const double *rhs, double *z, int *status, cudaStream_t s) {
    reset_queue(b, s);
    const int nbuf = sweep64_nbuf(net.ni, sweep64_ctas(b));
    k_sweep64<true><<<half_grid(b, VK_TUNE_SWEEP64, 2), 256, sweep64_smem(net.ni, 256, nbuf), s>>>(
        net, b, G, dB, dC, rhs, z, nullptr, nullptr, nullptr, status, nbuf);
}

void launch_back64(const DevNet &net, const DevBatch &b, const double *G, const double *dB,
                   const double *dC, double *z, double *x, const double *y, double *yk2, int *status,
                   cudaStream_t s) {
    reset_queue(b, s);
    const int nbuf = sweep64_nbuf(net.ni, sweep64_ctas(b));
    k_sweep64<false><<<half_grid(b, VK_TUNE_SWEEP64, 2), 256, sweep64_smem(net.ni, 256, nbuf), s>>>(
        net, b, G, dB, dC, nullptr, z, x, y, yk2, status, nbuf);
}

}  // namespace vk
