// FP64 Gauss-Jordan inversion of one n x n block by a CTA, or by the CTAs of a
// cluster that hold its columns in slices (k_lu64, k_lu64_long; k_solve64_small).
//
// The block lives in shared memory, stored row r / column c standing for the
// block's row rowid[r] and column colid[c].  Step k eliminates stored column
// k.  Its pivot is the unused row with the largest |a| (compared to 2^-12
// relative, the lowest row on ties; rows are never exchanged).  With the
// multipliers m_i = a_ik / a_pk (m_p = 0) the step is
//     a_iq <- a_iq - m_i a_pq  (i != p, q != k),   a_ik <- -m_i,   a_pk <- 1,
// row p staying unscaled until the end (its factor 1/a_pk is kept in srow).
// The result is the inverse with new labels: stored (r, c) is the inverse's
// row colid[step that used r], column rowid[pivot row of step c], so the next
// layer's Schur complement and Gauss-Jordan run in place on the same storage
// and no row or column is ever moved.
//
// Look-ahead: while the bulk warps apply step k, the prep warps (one thread
// per row) update column k+1, find its pivot, and compute step k+1's
// multipliers, so a step costs one block barrier.  In a cluster the CTA that
// owns column k+1 sends its multipliers, pivot row and reciprocal to the others'
// message slot k+1 (a bulk copy completing on
// the receiver's mbarrier); the owner of a run of columns never
// waits for the others, and no cluster barrier is needed inside a column:
// a slot of the next layer is written only after its reader has passed the
// same slot of this layer (each rank's own messages of this layer prove it,
// for n >= 32 and up to 8 CTAs).  Each element sees the same operations in
// the same order however many CTAs share the block, so the result does not
// depend on the cluster size.
//
// What bounds it: the FP64 unit (an SM issues one warp-wide FP64 instruction
// per 19 cycles, one warp at most one per 64 cycles), n^2/32 of them a step
// plus the multipliers and the reciprocal; with few columns the chain of a step
// (the message, update, search, reciprocal, multipliers, barrier), 1 400 cycles at
// 41 species and 1 500 at 69 in a cluster of eight.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "vk_halves.cuh"
#include "vk_tma.cuh"

namespace vk {

constexpr int kLu64MinCluster = 32;    // smallest block a cluster may share

__host__ __device__ inline int lu64_prep_warps(int n) { return (n + 31) / 32; }
// Bulk warps of a CTA that has a block to itself, as many on each of the SM's
// four schedulers (512 NCHO columns: 6, 8, 10, 12 and 14 warps 49.4, 49.5, 47.1,
// 46.0 and 47.4 ms), and of a cluster's (5 to 9 warps: one NCHO column 4.09, 4.03,
// 3.72, 3.82 and 3.82 ms, seven columns of 89 species 5.46, 5.24, 5.09, 5.28 and 5.24).
__host__ __device__ inline int lu64_threads(int n, int csize) {
    return 32 * (lu64_prep_warps(n) + (csize > 1 ? 7 : 12));
}
// doubles of a message: 1/pivot, pivot row, n multipliers, to a multiple of 16 bytes
__host__ __device__ inline int lu64_msg(int n) { return (n + 3) & ~1; }
// first column of rank c's slice
__host__ __device__ inline int lu64_slice(int n, int csize, int c) { return c * n / csize; }
__host__ __device__ inline int lu64_slice_max(int n, int csize) { return (n + csize - 1) / csize; }

// Copy of `bytes` from this CTA's shared memory into another CTA's of the
// cluster, counted there on its mbarrier (all addresses 16-byte aligned).
__device__ __forceinline__ void bulk_send(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "r"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Wait of at most `spin` polls for data other CTAs of the cluster sent; false
// when they run out or a CTA of the cluster has given up (*lost).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity, int spin, const int *lost) {
    for (int i = 0; i < spin; ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if ((i & 63) == 63 && *(const volatile int *)lost) return false;
    }
    return false;
}

// 1/x: the hardware's approximation (about 20 bits) and one third-order
// step x (1 + e + e^2), e = 1 - a x (Householder's iteration), in the range
// where neither can overflow or lose bits; the division (a call, so that it
// is branched around) elsewhere.  Error at most 0.57 ulp if the approximation sees and
// keeps 20 bits (|e| <= 2^-19, so e^3 is at most 1/16 ulp), 0.502 ulp measured over
// 70 000 values of every exponent; the division is exact to 0.5.
__device__ __noinline__ double recip64_edge(double a) { return 1.0 / a; }
__device__ __forceinline__ double recip64(double a) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
    const double e = __fma_rn(-a, x, 1.0);
    return __fma_rn(x, __fma_rn(e, e, e), x);
}
__device__ __forceinline__ bool recip64_edge_case(double a) {
    return (((unsigned)(__double_as_longlong(a) >> 52) & 0x7ffu) - 64u) > 1919u;
}

struct Lu64Mem {
    double *S;            // [n][w] this CTA's columns
    double *msg;          // [nslot][lu64_msg] 1/pivot, pivot row + flag, multipliers
    double *srow;         // [n] scale of each stored row
    double *rowf, *colf;  // [n] factors of the Schur term, by stored row and column
    double *diag;         // [n] c0 - dA, by species
    double *xval;         // [8] the prep warps' candidates' reciprocals
    unsigned *xkey;       // [8] and keys (16-byte aligned; zero beyond the prep warps)
    int *rowid, *colid;   // [n] labels
    int *perm, *kinv;     // [n] pivot row of each step, step of each row
    uint64_t *bar;        // [n] message barriers (cluster)
    int *sing;            // first failure: 1 zero pivot, 2 no finite candidate
    int *dead;            // this CTA gave up a wait for a message (its own threads set it)
    int *lost;            // a CTA of the cluster did (set from there)
    int n, w, c0;         // size, slice width, first column
    int csize, rank, pw;  // cluster size, rank, prep warps
    int spin;             // polls of a wait
};

// A message never came: this CTA's block is void, and the others of the cluster,
// which are all in the kernel until the cluster leaves it together, stop waiting.
__device__ __forceinline__ void lu64_give_up(const Lu64Mem &m) {
    if (*(volatile int *)m.dead) return;
    *(volatile int *)m.dead = 1;
    for (int c = 0; c < m.csize; ++c)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(smem_u32(m.lost), (uint32_t)c)), "r"(1)
                     : "memory");
}

// Inverts the block in m.S and relabels it.  All threads of the CTA call it
// (in a cluster: of every CTA); it starts after a block barrier and ends with
// one.  `phase`: inversions this CTA has done before (message parity).  False, for
// the whole CTA, when a message never came: m.S then holds no inverse, rowid and colid
// are as before, and no other inversion may follow (it would arm message
// barriers whose phase is open, and relabel by pivots that never were).
template <bool CL>
__device__ __forceinline__ bool lu64_invert(const Lu64Mem &m, unsigned phase) {
    const int n = m.n, w = m.w, c0 = m.c0, c1 = c0 + w, ms = lu64_msg(n);
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int npt = m.pw * 32;
    const bool prep_thread = tid < npt;
    const int r = tid;                                  // a prep thread's row
    bool used = false;
    double mult = 0.0;                                  // the last multiplier / pivot row this
    int mp = 0, mk = -1;                                // prep thread computed, and its step
    // column kk's pivot and multipliers; kk > 0: after step kk - 1 with pivot
    // row pp and this row's multiplier mprev
    auto prepare = [&](int kk, double mprev, int pp) {
        double v = 0.0;
        const int qk = kk - c0;
        if (r < n) {
            v = m.S[r * w + qk];
            if (kk > 0) v = __fma_rn(-mprev, m.S[pp * w + qk], v);
        }
        // one key per row: a finite candidate is |a| to 2^-12 over 255 - row, a
        // NaN row only its place (chosen when nothing else is left)
        const unsigned long long bits = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
        unsigned key = 0;
        if (r < n && !used)
            key = bits <= 0x7ff0000000000000ull
                      ? 0x80000000u | ((unsigned)(bits >> 32) & ~255u) | (unsigned)(255 - r) : (unsigned)(256 - r);
        const unsigned mx = __reduce_max_sync(0xffffffffu, key);
        if (lane == 0) m.xkey[warp] = mx;
        // the reciprocal: of every row's candidate while the search runs where the
        // chain of pivots is what takes the time, of the pivot alone (three FP64
        // instructions instead of three per warp) on a full chip
        if (CL) {
            double x = recip64(v);
            if (key == mx && recip64_edge_case(v)) x = recip64_edge(v);
            if (key == mx && key) m.xval[warp] = x;
        }
        asm volatile("barrier.sync 1, %0;" ::"r"(npt) : "memory");
        const uint4 ka = *reinterpret_cast<const uint4 *>(m.xkey), kb = *reinterpret_cast<const uint4 *>(m.xkey + 4);
        const unsigned best = max(max(max(ka.x, ka.y), max(ka.z, ka.w)), max(max(kb.x, kb.y), max(kb.z, kb.w)));
        int p = (best & 0x80000000u) ? 255 - (int)(best & 255u) : 256 - (int)best;
        int flag = (best & 0x80000000u) ? 0 : 2;
        if ((unsigned)p >= (unsigned)n) p = 0;          // (cannot happen: a row is always left)
        const int pwarp = p >> 5;
        double pinv;
        if (CL) {
            pinv = m.xval[pwarp];
        } else {
            if (warp == pwarp) {
                const double pv = __shfl_sync(0xffffffffu, v, p & 31);
                pinv = recip64(pv);
                if (recip64_edge_case(pv)) pinv = recip64_edge(pv);
                if (lane == 0) m.xval[0] = pinv;
            }
            asm volatile("barrier.sync 1, %0;" ::"r"(npt) : "memory");
            pinv = m.xval[0];
        }
        if (r == p && (__double_as_longlong(v) & 0x7fffffffffffffffll) == 0) flag = 1;
        mult = r == p ? 0.0 : v * pinv;
        mp = p;
        mk = kk;
        double *slot = m.msg + (size_t)(CL ? kk : (kk & 1)) * ms;
        const double pword = __longlong_as_double((long long)(unsigned)(p | (flag << 16)));
        if (r < n) {
            slot[2 + r] = mult;
            m.S[r * w + qk] = r == p ? 1.0 : -mult;
        }
        if (r == p) *reinterpret_cast<double2 *>(slot) = make_double2(pinv, pword);
    };
    if (tid >= m.pw && tid < 8) m.xkey[tid] = 0;
    if (CL) {                                           // one message per foreign step
        for (int k = tid; k < n; k += nth)
            if (k < c0 || k >= c1)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                             ::"r"(smem_u32(&m.bar[k])), "r"((uint32_t)ms * 8) : "memory");
    }
    __syncthreads();
    if (prep_thread && c0 == 0) prepare(0, 0.0, 0);
    __syncthreads();
    const int nb = nth - npt, tb = tid - npt;           // bulk threads
    const int ne = n * w;
    const int di = w > 0 ? nb / w : 0, dq = w > 0 ? nb - di * w : 0;
    const int i0 = tb >= 0 && w > 0 ? tb / w : 0, q0 = tb >= 0 && w > 0 ? tb - i0 * w : 0;
    for (int k = 0; k < n; ++k) {
        const double *slot = m.msg + (size_t)(CL ? k : (k & 1)) * ms;
        if (CL && (k < c0 || k >= c1))
            if (!mbar_wait_cluster(&m.bar[k], phase & 1, m.spin, m.lost)) lu64_give_up(m);
        if (prep_thread) {
            if (mk != k) {                              // another CTA's step
                mult = r < n ? slot[2 + r] : 0.0;
                mp = (int)((unsigned)__double_as_longlong(slot[1]) & 0xffffu);
                if (mp >= n) mp = 0;                    // (a message that never came)
            }
            const int p = mp;
            if (r == p) used = true;
            if (k + 1 < n && k + 1 >= c0 && k + 1 < c1) prepare(k + 1, mult, p);
        } else {
            if (CL && warp == m.pw && k >= c0 && k < c1) {
                // send this step's message: one lane per other CTA
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                if (lane < m.csize && lane != m.rank)
                    bulk_send(cluster_addr(smem_u32(slot), (uint32_t)lane), smem_u32(slot), (uint32_t)ms * 8,
                              cluster_addr(smem_u32(&m.bar[k]), (uint32_t)lane));
            }
            int p = (int)((unsigned)__double_as_longlong(slot[1]) & 0xffffu);
            if (CL && p >= n) p = 0;
            if (tb == 0) {
                m.srow[p] = slot[0];
                m.kinv[p] = k;
                m.perm[k] = p;
                const int flag = (int)((unsigned)__double_as_longlong(slot[1]) >> 16);
                if (flag && *m.sing == 0) *m.sing = flag;
            }
            const double *Sp = m.S + p * w;
            const int kq = k - c0, kq1 = k + 1 - c0;
            int i = i0, q = q0, e = tb;
            for (; e + 3 * nb < ne; e += 4 * nb) {      // four elements' loads in flight
                double a[4], rr[4], mi[4];
                bool st[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    a[u] = m.S[e + u * nb];
                    rr[u] = Sp[q];
                    mi[u] = slot[2 + i];
                    st[u] = q != kq && q != kq1 && i != p;
                    q += dq;
                    i += di;
                    if (q >= w) { q -= w; ++i; }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) a[u] = __fma_rn(-mi[u], rr[u], a[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (st[u]) m.S[e + u * nb] = a[u];
            }
            for (; e < ne; e += nb) {
                const double v = __fma_rn(-slot[2 + i], Sp[q], m.S[e]);
                if (q != kq && q != kq1 && i != p) m.S[e] = v;
                q += dq;
                i += di;
                if (q >= w) { q -= w; ++i; }
            }
        }
        __syncthreads();
    }
    if (CL && *(volatile int *)m.dead) return false;    // (set before the last barrier only)
    // labels of the inverse
    int nr = 0, nc = 0;
    if (tid < n) {
        nr = m.colid[m.kinv[tid]];
        nc = m.rowid[m.perm[tid]];
    }
    __syncthreads();
    if (tid < n) {
        m.rowid[tid] = nr;
        m.colid[tid] = nc;
    }
    __syncthreads();
    return true;
}

}  // namespace vk
