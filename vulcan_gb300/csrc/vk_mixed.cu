// Mixed-precision block-tridiagonal solve: FP32 factorisation on scaled
// blocks, FP64 residual and iterative refinement.
//
// The system is the Ros2 LHS  A = c0 I - J_chem - J_diff  (op.py:1973-2042):
// dense diagonal blocks D_j = c0 I + (-J_j) - diag(dA_j) and diagonal couplings
// L_j = -diag(dC_j) (to layer j-1), U_j = -diag(dB_j) (to layer j+1).
//
// The factorisation (k_prep32, k_lu32) works on the scaled
// system R A S, with per-layer power-of-two row scales R_j (row maxima of D_j)
// and column scales S_j (column maxima of R_j D_j), so the scaling itself is
// exact; each Schur-complemented scaled block
//     D~'_j = R_j D_j S_j - L~_j G~_{j-1} U~_{j-1}
// is inverted in FP32 and G~_j is stored in FP32 (half the bytes of FP64).
//
// k_refine (one column at a time per CTA) solves A x = b: x = 0, r = b; repeat
// { d = S M~^-1 R r  (FP32 forward/back sweeps with G~);  x += d (FP64);
//   r = b - A x  (FP64, matrix-free from the sparse -J and dA/dB/dC) }
// until max |d| / (|x| + |yscale| + 1e-10 n_0) <= tol or max sweeps; a
// column that does not converge is flagged for the FP64 path.
//
// Routing.  At large dt the scaled diagonal blocks of a near-steady column
// reach condition numbers of 1e10..1e16 (c0 -> 0 exposes the conserved and
// slow chemical modes), beyond what FP32 factors can precondition: refinement
// diverges.  A column whose refinement failed at step size dt therefore sends
// every later attempt with a step >= dt/4 straight to the FP64 path (thr64),
// and tries the mixed path again only after its step has dropped below that:
// the margin keeps a rejected attempt (dt halved) and the step-size rule's
// 0.5x..2x changes from retrying a factorisation that has just failed.
#include <cuda_runtime.h>
#include <math.h>

#include "vk_halves.cuh"
#include "vk_internal.cuh"
#include "vk_tma.cuh"

namespace vk {

constexpr double kRouteMargin = 0.25;   // FP64 from dt >= kRouteMargin x the failed step


// Iterative refinement of A x = b with the FP32 factors, a cluster of two CTAs
// per column (columns from the work queue): CTA h takes half h of the layers
// (0 .. m, m + 1 .. nz - 1) in the order the two-sided factorisation eliminated
// them.  A sweep runs both halves towards the middle at once, the middle layer
// in CTA 0, and both halves back; the halves exchange one vector each way.
// A visit is FP32 only -- the product with G~_j, whose row r also yields row r
// of the next visit's input (one fma with the precomputed scaled coupling) --
// and costs one block barrier.  The last warp has no rows: it issues the bulk
// copies of the inverse blocks (visit order, NB - 1 ahead), loads the rows'
// couplings and residuals two visits ahead, and waits for both while the
// other warps work on the visit before.  Everything in FP64 (the couplings,
// the scaled residual, x += S x~ and the correction size of the convergence
// test, the residual b - A x) runs in parallel passes over the half between
// the sweeps.
// What bounds it: at a full chip reading the inverses twice a sweep and the
// FP64 passes, of which the residual's rows are cut into pieces of similar
// length (164 -> 75 warp-wide FP64 steps a layer on the 69-species network);
// for few columns the chain of dependent visits, which two CTAs halve.
// Two solves of an attempt, 69 species: 512 columns 9.4 -> 6.8 ms, 64 columns
// 6.3 -> 2.4 ms; 150 species, 48 columns: 33 -> 7.7 ms.  With a lane's loads of
// the row vectors instead of the last warp's copies, the stride of a row's
// lanes a run-time value and x read from global memory in the residual: 7.5 to
// 8.9, 3.0 and 14 ms.
// yscale (may be NULL) widens the convergence floor: k1/k2 enter sol next to y.
constexpr int kBars = 8;                // most blocks in flight
constexpr int kColStage = 8192;         // Jacobian entries whose columns are kept in shared memory
struct RefineSmem { int G, vec, vin, mid, xm, jc, ps, end; };         // byte offsets
__host__ __device__ inline RefineSmem refine_layout(int n, int npc, int nnz, int nwarp, int nb) {
    RefineSmem s;
    int o = kBars * 8;
    s.G = o;   o += nb * block_stride32(n) * 4;
    s.vec = o; o += 3 * 2 * n * 4;               // (coupling, residual or forward result) of three visits
    s.vin = o; o += 2 * n * 4;                   // visit inputs
    s.mid = o; o += 2 * n * 4;                   // (CTA 0) the halves' terms of the middle
    s.xm = o;  o += n * 4;                       // the middle's result
    o = (o + 15) & ~15;
    s.jc = o;  o += nnz <= kColStage ? nnz * 2 : 0;
    // x and the row pieces of each warp's layer: in the block buffer that is
    // free between sweeps where they fit
    o = (o + 15) & ~15;
    s.ps = -1;
    if (nwarp * (npc + n) * 8 > block_stride32(n) * 4) {
        s.ps = o;
        o += nwarp * (npc + n) * 8;
    }
    s.end = (o + 15) & ~15;
    return s;
}

template <int TPR>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(352, 2)
k_refine(DevNet net, DevBatch b, const float *__restrict__ G32, const double *__restrict__ rsc,
         const double *__restrict__ csc, const double *__restrict__ jv,
         const double *__restrict__ dA, const double *__restrict__ dB,
         const double *__restrict__ dC, const double *__restrict__ dt,
         const double *__restrict__ rhs, double *x, float *zf, float *wcf,
         float *wcb, float *raf, float *__restrict__ xf,
         const double *__restrict__ yscale, double *__restrict__ yk2,
         const double *__restrict__ y, int max_sweeps, double tol, int *__restrict__ fallback,
         int *__restrict__ sweeps_out, int *__restrict__ status, double *__restrict__ err_out,
         double *__restrict__ thr64, int *act32, int *__restrict__ failed, int NB) {
    extern __shared__ __align__(16) unsigned char smr[];
    const int n = net.ni, NNP = block_stride32(n);
    const int tid = threadIdx.x, nth = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int nwarp = nth >> 5;
    const RefineSmem L = refine_layout(n, net.npc, net.nnz, nwarp, NB);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smr);           // [NB]
    float *Gbuf = reinterpret_cast<float *>(smr + L.G);          // [NB][NNP]
    float *vec = reinterpret_cast<float *>(smr + L.vec), *vin = reinterpret_cast<float *>(smr + L.vin);
    float *mid_in = reinterpret_cast<float *>(smr + L.mid), *xm = reinterpret_cast<float *>(smr + L.xm);
    uint16_t *jc = reinterpret_cast<uint16_t *>(smr + L.jc);
    const bool staged = net.nnz <= kColStage;
    __shared__ double red[11], s_m[2];
    __shared__ int s_col, s_lost[2];
    uint32_t half;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(half));
    const uint32_t other = half ^ 1u;
    const uint32_t bytes = (uint32_t)NNP * sizeof(float);
    const bool producer = warp == nwarp - 1;
    const int mrow = tid / TPR, mpart = tid - mrow * TPR;
    const bool rowt = mrow < n && !producer, lead = rowt && mpart == 0;
    if (tid == 0) {
        for (int i = 0; i < NB; ++i) mbar_init(&bar[i], 1);
        mbar_fence_init();
        s_lost[0] = s_lost[1] = 0;
    }
    if (staged)
        for (int e = tid; e < net.nnz; e += nth) jc[e] = (uint16_t)net.jcol[e];
    __syncthreads();
    auto remote = [&](const void *p) { return cluster_addr(smem_u32(p), other); };
    auto next = [&]() {
        cluster_sync_all();
        if (half == 0 && tid == 0) {
            const unsigned i = atomicAdd(b.queue, 1u);
            const int c = i < (unsigned)b.ncols ? b.order[i] : -1;
            s_col = c;
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(&s_col)), "r"(c) : "memory");
        }
        cluster_sync_all();
        return s_col;
    };
    int cb = 0;                                  // buffer of the current visit (every thread)
    // the producer's own state: next buffer to fill, phase of buffer cb, copies in flight
    int ib = 0, flying = 0;
    unsigned cph = 0;
    bool gone = false;
    for (int c; !gone && (c = next()) >= 0;) {
        if (b.active && !b.active[c]) continue;
        const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = nz / 2;
        const double c0 = 1.0 / (R_ROS * dt[c]);
        const int cnt = half ? nz - 1 - mid : mid;               // layers of the half but the middle
        const int j0 = half ? mid + 1 : 0, j1 = half ? nz : mid + 1;     // its layers
        const size_t e0 = ((size_t)l0 + j0) * n;
        const int ne = (j1 - j0) * n;
        const int per = 2 * cnt + (half ? 0 : 1);                // visits of a sweep
        const int step = half ? -1 : 1;                          // layers inwards
        const int lf = half ? nz - 1 : 0, lb = half ? mid + 1 : mid - 1;     // first layers inwards, outwards
        const float *wf = half ? wcb : wcf, *wb = half ? wcf : wcb;          // couplings inwards, outwards
        int left = per * max_sweeps, nv = 0;                     // producer: visits not issued, the next in its sweep
        auto issue = [&]() {                                     // producer
            if (left <= 0) return;
            int j;
            if (nv < cnt) j = lf + step * nv;
            else if (!half && nv == cnt) j = mid;
            else j = lb - step * (nv - cnt - (half ? 0 : 1));
            if (lane == 0) tma_load_1d(Gbuf + ib * NNP, G32 + ((size_t)l0 + j) * NNP, bytes, &bar[ib]);
            --left;
            if (++nv == per) nv = 0;
            ++flying;
            if (++ib == NB) ib = 0;
        };
        auto landed = [&]() {                                    // producer: the current visit's block
            if (!s_lost[0] && !mbar_wait(&bar[cb], cph)) *(volatile int *)&s_lost[0] = 1;
            --flying;
            if (cb + 1 == NB) cph ^= 1u;
        };
        // producer: row vectors of visit v of a phase into slot v % 3
        auto fetch = [&](int v, bool inwards) {
            float *s = vec + (v % 3) * 2 * n;
            const size_t ew = ((size_t)l0 + (inwards ? lf + step * (v + 1) : lb - step * (v + 1))) * n;
            const size_t er = inwards ? ew : ((size_t)l0 + lb - step * v) * n;
            const float *w = inwards ? wf : wb, *r = inwards ? raf : zf;
            if (v < cnt)
                for (int e = lane; e < n; e += 32) {
                    if (v + 1 < cnt)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(s + e)), "l"(w + ew + e) : "memory");
                    if (!inwards || v + 1 < cnt)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(s + n + e)), "l"(r + er + e) : "memory");
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        int p = 0;                                               // vin buffer of the current visit
        // the product of the current visit's block with its input
        auto product = [&]() {
            const float *row = Gbuf + cb * NNP + mrow * n, *xin = vin + p * n;
            float s0 = 0.0f, s1 = 0.0f;
            if (rowt) {
                int q = mpart;
                for (; q + 5 * TPR < n; q += 6 * TPR) {
                    float g[6], xv[6];
#pragma unroll
                    for (int u = 0; u < 6; ++u) { g[u] = row[q + u * TPR]; xv[u] = xin[q + u * TPR]; }
#pragma unroll
                    for (int u = 0; u < 6; u += 2) { s0 = fmaf(g[u], xv[u], s0); s1 = fmaf(g[u + 1], xv[u + 1], s1); }
                }
                for (; q < n; q += TPR) s0 = fmaf(row[q], xin[q], s0);
            }
            float s = s0 + s1;
            __syncwarp();
#pragma unroll
            for (int o = 1; o < TPR; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
            return s;
        };
        auto advance = [&]() {                                   // to the next visit's buffers
            p ^= 1;
            if (++cb == NB) cb = 0;
        };
        if (producer)
            for (int i = 0; i < NB - 1; ++i) issue();
        // x = 0, r = b; the scaled couplings of the sweeps (FP32: they feed
        // the FP32 preconditioner) and the scaled first residual
#pragma unroll 4
        for (int e = tid; e < ne; e += nth) {
            const size_t g = e0 + e;
            const int j = j0 + e / n;
            x[g] = 0.0;
            raf[g] = (float)(rsc[g] * rhs[g]);
            wcf[g] = j > 0 ? (float)(rsc[g] * dC[g] * csc[g - n]) : 0.f;
            wcb[g] = j < nz - 1 ? (float)(rsc[g] * dB[g] * csc[g + n]) : 0.f;
        }
        cluster_sync_all();                      // CTA 1 reads the middle's coupling
        int sweep = 0, converged = 0;
        double m_prev = INFINITY;
        for (; sweep < max_sweeps && !converged; ++sweep) {
            // towards the middle
            float z = 0.f;
            if (producer) {
                fetch(0, true);
                fetch(1, true);
            } else if (lead && cnt > 0) {
                vin[p * n + mrow] = raf[((size_t)l0 + lf) * n + mrow];
            }
            for (int v = 0; v < cnt; ++v) {
                if (producer) {
                    landed();
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                }
                __syncthreads();                 // input, vectors and block in place; the last buffers free
                if (producer) {
                    issue();
                    fetch(v + 2, true);
                } else {
                    z = product();
                    if (lead) {
                        const float *s = vec + (v % 3) * 2 * n + mrow;
                        zf[((size_t)l0 + lf + step * v) * n + mrow] = z;
                        if (v + 1 < cnt) vin[(p ^ 1) * n + mrow] = fmaf(s[0], z, s[n]);
                    }
                }
                advance();
            }
            // the middle, in CTA 0; its result to both
            if (lead) {
                const float t = cnt > 0 ? __ldcg(wf + ((size_t)l0 + mid) * n + mrow) * z : 0.f;
                if (half == 0) mid_in[mrow] = t;
                else
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote(mid_in + n + mrow)), "f"(t) : "memory");
            }
            cluster_sync_all();
            if (half == 0) {
                const size_t e = ((size_t)l0 + mid) * n + mrow;
                if (lead) vin[p * n + mrow] = raf[e] + mid_in[mrow] + mid_in[n + mrow];
                if (producer) landed();
                __syncthreads();
                if (producer) {
                    issue();
                } else {
                    const float t = product();
                    if (lead) {
                        xf[e] = t;
                        xm[mrow] = t;
                        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote(xm + mrow)), "f"(t) : "memory");
                    }
                }
                advance();
            }
            cluster_sync_all();
            // and back
            if (producer) {
                fetch(0, false);
                fetch(1, false);
            } else if (lead && cnt > 0) {
                vin[p * n + mrow] = wb[((size_t)l0 + lb) * n + mrow] * xm[mrow];
            }
            for (int v = 0; v < cnt; ++v) {
                if (producer) {
                    landed();
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                }
                __syncthreads();
                if (producer) {
                    issue();
                    fetch(v + 2, false);
                } else {
                    float t = product();
                    if (lead) {
                        const float *s = vec + (v % 3) * 2 * n + mrow;
                        t += s[n];
                        xf[((size_t)l0 + lb - step * v) * n + mrow] = t;
                        if (v + 1 < cnt) vin[(p ^ 1) * n + mrow] = s[0] * t;
                    }
                }
                advance();
            }
            __syncthreads();                     // the last visit's results are visible
            // x += S x~ and the largest |d| / (|x| + |yscale| + 1e-10 n_0) of
            // the sweep, kept as a fraction (num, den) compared by
            // cross-multiplication and divided once per thread (FP64 divisions
            // are long FP64-pipe sequences on this chip)
            double dnum = 0.0, dden = 1.0;
#pragma unroll 4
            for (int e = tid; e < ne; e += nth) {
                const size_t g = e0 + e;
                const double d = csc[g] * (double)xf[g];
                const double xn = x[g] + d;
                x[g] = xn;
                const double n0 = b.atm[((size_t)l0 + j0 + e / n) * VK_ATM_NF + VK_ATM_N0];
                const double sc = fabs(xn) + (yscale ? fabs(yscale[g]) : 0.0) + 1e-10 * n0;
                const double ad = fabs(d);
                if (!isfinite(d)) { dnum = INFINITY; dden = 1.0; }
                else if (ad * dden > dnum * sc) { dnum = ad; dden = sc; }
            }
            double dmax = dnum / dden;
            for (int o = 16; o; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
            if (lane == 0) red[warp] = dmax;
            __syncthreads();
            if (tid == 0) {
                double m = red[0];
                for (int w = 1; w < nwarp; ++w) m = fmax(m, red[w]);
                s_m[half] = m;
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote(&s_m[half])), "d"(m) : "memory");
                if (s_lost[0])
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(&s_lost[1])), "r"(1) : "memory");
            }
            cluster_sync_all();                  // also: both halves' x are visible
            if (s_lost[0] | s_lost[1]) { gone = true; break; }
            const double m = fmax(s_m[0], s_m[1]);
            // converged; or stagnating at the FP64 residual's noise floor (the
            // correction stopped shrinking while already below 1e-6 of |x|+|y|)
            converged = (m <= tol) || (sweep >= 1 && m > 0.25 * m_prev && m <= 1e-6);
            if (!(m <= m_prev) && sweep >= 2) break;        // diverging: leave to the FP64 path
            m_prev = m;
            if (converged) break;
            if (sweep + 1 == max_sweeps) continue;          // no sweep will read it
            // the scaled FP32 residual R (b - A x) of the next sweep (FP64,
            // matrix-free), a layer per warp: the row pieces, then the rows
            double *xw = reinterpret_cast<double *>(
                             L.ps >= 0 ? smr + L.ps
                                       : reinterpret_cast<unsigned char *>(Gbuf + (cb ? cb - 1 : NB - 1) * NNP)) +
                         (size_t)warp * (net.npc + n);
            double *pw = xw + n;
            auto col = [&](int k) { return staged ? (int)jc[k] : net.jcol[k]; };
            for (int j = j0 + warp; j < j1; j += nwarp) {
                const size_t l = (size_t)l0 + j;
                const double *jl = jv + l * net.nnz;
                for (int i = lane; i < n; i += 32) xw[i] = x[l * n + i];
                __syncwarp();
                for (int i = lane; i < net.npc; i += 32) {
                    const int2 q = net.pc[i];
                    double s = 0.0;
                    int k = q.x;
                    const int k1 = q.x + q.y;
                    for (; k + 7 < k1; k += 8) {            // eight entries' loads in flight
                        double v[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) v[u] = jl[k + u];
#pragma unroll
                        for (int u = 0; u < 8; ++u) s += v[u] * xw[col(k + u)];
                    }
                    for (; k < k1; ++k) s += jl[k] * xw[col(k)];
                    pw[i] = s;
                }
                __syncwarp();
                for (int sp = lane; sp < n; sp += 32) {
                    const size_t e = l * n + sp;
                    double ax = (c0 - dA[e]) * xw[sp];
                    for (int k = net.rpcptr[sp]; k < net.rpcptr[sp + 1]; ++k) ax += pw[net.rpc[k]];
                    // (the other half's layer next to the cut was written by the other CTA)
                    if (j > 0) ax -= dC[e] * (j > j0 ? x[e - n] : __ldcg(x + e - n));
                    if (j < nz - 1) ax -= dB[e] * (j < j1 - 1 ? x[e + n] : __ldcg(x + e + n));
                    raf[e] = (float)(rsc[e] * (rhs[e] - ax));
                }
                __syncwarp();
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // a copy lands there next
            __syncthreads();
        }
        // every issued copy lands before the column ends (bounded waits); a
        // copy that never lands ends this cluster's work with a timeout
        if (producer) {
            int cp = cb;
            while (flying > 0) {
                if (!mbar_wait(&bar[cp], cph)) *(volatile int *)&s_lost[0] = 1;
                --flying;
                if (++cp == NB) { cp = 0; cph ^= 1u; }
            }
            if (lane == 0) s_col = cp;                      // where every thread goes on
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncthreads();
        cb = s_col;
        if (tid == 0) {
            if (s_lost[0]) {
                atomicExch(&status[c], VK_ETIMEOUT);
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(&s_lost[1])), "r"(1) : "memory");
            } else if (half == 0 && !gone) {
                if (!converged) {
                    fallback[c] = 1;
                    act32[c] = 0;                   // later mixed launches of this attempt skip it
                    failed[c] = 1;                  // redone in FP64 after the routed columns
                    thr64[c] = fmin(thr64[c], kRouteMargin * dt[c]);
                }
                if (sweeps_out) atomicMax(sweeps_out, sweep + (converged ? 1 : 0));
                if (err_out) err_out[c] = fmax(err_out[c], m_prev);
            }
        }
        if (yk2 && !gone)
            for (int e = tid; e < ne; e += nth) yk2[e0 + e] = y[e0 + e] + x[e0 + e] / R_ROS;
        cluster_sync_all();
        if (s_lost[0] | s_lost[1]) gone = true;
    }
    cluster_sync_all();
}

// fallback[c] = 1: this attempt of column c is solved in FP64 (its step is at or
// above the size at which its refinement last failed); act32[c] = 1: mixed.
// Routing of one attempt: routed[c] = 1: solved in FP64 from the start (its
// step is at or above the size at which its refinement last failed, with the
// margin); act32[c] = 1: mixed; fallback[c] = every FP64 solve of the attempt
// (routed, and mixed columns whose refinement fails, which k_refine adds
// together with failed[c]).
__global__ void k_route(DevBatch b, const double *__restrict__ dt, const double *__restrict__ thr64,
                        int *__restrict__ fallback, int *__restrict__ act32, int *__restrict__ routed,
                        int *__restrict__ failed) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= b.ncols) return;
    const int a = b.active ? b.active[c] : 1;
    const int f64 = a && !(dt[c] < thr64[c]);
    fallback[c] = f64;
    routed[c] = f64;
    act32[c] = a && !f64;
    failed[c] = 0;
}

__global__ void k_reset_route(int ncols, double *__restrict__ thr64, double route_dt0) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < ncols) thr64[c] = route_dt0;
}

void launch_route(const DevBatch &b, const Work &w, cudaStream_t s) {
    k_route<<<(b.ncols + 127) / 128, 128, 0, s>>>(b, w.dt, w.thr64, w.fallback, w.act32, w.routed,
                                                   w.failed);
}

void launch_reset_route(const Work &w, int ncols, double route_dt0, cudaStream_t s) {
    if (w.thr64) k_reset_route<<<(ncols + 127) / 128, 128, 0, s>>>(ncols, w.thr64, route_dt0);
}

namespace {
struct RefineShape { int nth, tpr, nb; size_t smem; };
// ctas: how many of the kernel's CTAs an SM should hold
RefineShape refine_shape(int n, int npc, int nnz, int ctas) {
    RefineShape r;
    // lanes per product row, and a warp more for the copies
    const int rows = n <= 144 ? 288 : 320;
    r.tpr = 4 * n <= rows ? 4 : 2;           // (2 VK_MAX_NI <= 320)
    r.nth = (r.tpr * n + 31) / 32 * 32 + 32;
    r.nb = 4;
    while (r.nb > 2 && ctas * ((size_t)refine_layout(n, npc, nnz, r.nth / 32, r.nb).end + 1200) > 233472) --r.nb;
    r.smem = (size_t)refine_layout(n, npc, nnz, r.nth / 32, r.nb).end;
    return r;
}
}  // namespace

cudaError_t init_mixed_kernels(const DevNet &net) {
    const RefineShape r = refine_shape(net.ni, net.npc, net.nnz, 1);
    return r.tpr == 4 ? raise_smem_limit(k_refine<4>, r.smem) : raise_smem_limit(k_refine<2>, r.smem);
}

void launch_refine(const DevNet &net, const DevBatch &b, const Work &w, const double *rhs,
                   double *x, const double *yscale, double *yk2, int max_sweeps, double tol,
                   cudaStream_t s) {
    const RefineShape r = refine_shape(net.ni, net.npc, net.nnz, 2 * b.ncols <= b.nsm ? 1 : 2);
    reset_queue(b, s);
    const int grid = half_grid(b, VK_TUNE_REFINE, 2) & ~1;    // CTA pairs, one column each
    auto kernel = r.tpr == 4 ? k_refine<4> : k_refine<2>;
    kernel<<<grid, r.nth, r.smem, s>>>(net, b, w.G32, w.rs, w.cs, w.jv, w.dA, w.dB, w.dC, w.dt,
                                      rhs, x, w.zf, w.wcf, w.wcb, w.raf, w.xf, yscale, yk2, w.y,
                                      max_sweeps, tol,
                                      w.fallback, w.sweeps, w.status, w.refine_err, w.thr64,
                                      w.act32, w.failed, r.nb);
}

}  // namespace vk
