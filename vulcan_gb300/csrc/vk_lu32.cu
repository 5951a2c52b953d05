// FP32 block factorisation of the scaled systems (mixed path), two-sided
// block-Thomas over half-columns (vk_halves.cuh):
//   G~_j = D~'_j^-1,  D~_j = R_j D_j S_j  (k_prep32),
//   bottom half  D~'_j = D~_j - diag(R_j dC_j S_{j-1}) G~_{j-1} diag(R_{j-1} dB_{j-1} S_j),
//   top half     D~'_j = D~_j - diag(R_j dB_j S_{j+1}) G~_{j+1} diag(R_{j+1} dC_{j+1} S_j),
// the middle layer has both terms.
//
// A block is inverted by Gauss-Jordan with implicit pivoting (rows are never
// exchanged; a pivot is the unused row with the largest |a| to 2^-15, the
// lowest on ties).  With the multipliers m_i = a_ik / a_pk (m_p = 0) a step is
// a_iq -= m_i a_pq, a_ik = -m_i, a_pk = 1; the pivot rows' factors 1/a_pk wait in
// srow until the inverse is stored.
// The block lives in registers: lane r of every warp holds rows r, r + 32, ..
// (RA of them), warp w of W the columns w, w + W, .. (CW of them).  The warp
// that owns the next column updates it first, finds its pivot and publishes
// the multipliers while the others apply the current step, so a step costs one
// block barrier; the pivot row reaches a warp's lanes through shared memory
// without a barrier (every warp holds its columns of every row).  Every W steps
// the registers rotate by one column, so the current column is always the
// first and the loop body is not unrolled over the columns.
// What bounds it: the chain of n pivots a layer (argmax, reciprocal, one
// barrier each), hidden behind the other CTAs of the SM where columns are
// plenty.  A blocked elimination on the tensor cores shortens the updates, not
// that chain.  With k_prep32, 69 species: 512 columns 11.0 -> 6.3 ms, 64
// columns 7.0 -> 2.95 ms (tcgen05 rank-16 panels before); 150 species, 48
// columns: 54 -> 13.6 ms (a one-sided register elimination with the block
// spread by 8 x 19 tiles before).
//
// Reference: the banded LU of the Ros2 LHS, op.py:2913-2929 (solve_banded on
// the matrix store_bandM builds, op.py:2833-2858).
#include <cuda_runtime.h>
#include <math.h>

#include "vk_halves.cuh"
#include "vk_internal.cuh"
#include "vk_tma.cuh"

namespace vk {

namespace {

constexpr int kSlot = 168;               // multipliers by row, then pivot row, 1/pivot, flag

struct Lu32Smem {                        // float offsets
    int Gs, D, ms, row, alpha, beta, srow, perm, kinv, end;
};
__host__ __device__ inline Lu32Smem lu32_layout(int n, int cw, int w) {
    const int nn4 = block_stride32(n);
    Lu32Smem s;
    int o = 0;
    s.Gs = o;    o += nn4;
    s.D = o;     o += nn4;
    s.ms = o;    o += 2 * kSlot;
    s.row = o;   o += w * ((cw + 3) & ~3);
    s.alpha = o; o += n;
    s.beta = o;  o += n;
    s.srow = o;  o += n;
    s.perm = o;  o += n;
    s.kinv = o;  o += n;
    s.end = o;
    return s;
}

}  // namespace

// The next layer's block is copied to shared memory while this one is inverted.
template <int RA, int CW, int W>
__global__ void __launch_bounds__(32 * W, W == 4 ? (RA * CW <= 54 ? 4 : 3) : 1)
k_lu32(DevNet net, DevBatch b, const float *__restrict__ D32, const double *__restrict__ dB,
       const double *__restrict__ dC, const double *__restrict__ rsc, const double *__restrict__ csc,
       float *G32, int *__restrict__ status) {
    extern __shared__ __align__(16) float smf[];
    __shared__ int s_unit, s_stat;
    constexpr int CP = (CW + 3) & ~3;
    constexpr int NTH = 32 * W;
    const int n = net.ni, NNP = block_stride32(n);
    const Lu32Smem L = lu32_layout(n, CW, W);
    float *Gs = smf + L.Gs, *Db = smf + L.D, *ms = smf + L.ms, *alpha = smf + L.alpha, *beta = smf + L.beta;
    float *srow = smf + L.srow;
    int *perm = reinterpret_cast<int *>(smf + L.perm), *kinv = reinterpret_cast<int *>(smf + L.kinv);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float *row = smf + L.row + warp * CP;                 // this warp's slice of the pivot row
    for (int e = tid; e < n; e += NTH) { perm[e] = 0; kinv[e] = 0; srow[e] = 0.f; }
    __syncthreads();

    float A[RA][CW];
    // The next pivot: the best of a column's unused rows from v[a] (this lane's
    // rows), then its multipliers into message slot kk & 1.  In three parts, so
    // that the latencies of the search, the broadcast and the reciprocal pass
    // under the current step's FMAs.
    auto search = [&](const float (&v)[RA], unsigned used) {
        unsigned key = 0;
#pragma unroll
        for (int a = 0; a < RA; ++a) {
            const unsigned x = __float_as_uint(v[a]) & 0x7fffffffu;
            // a finite candidate; else the row only counts when nothing else is left
            const unsigned c = x < 0x7f800000u ? 0x80000000u | (x & ~255u) : 0u;
            if (!((used >> a) & 1u)) key = max(key, c | (unsigned)(255 - (lane + 32 * a)));
        }
        return __reduce_max_sync(0xffffffffu, key);
    };
    auto pivot_value = [&](unsigned best, const float (&v)[RA], int &p) {
        p = 255 - (int)(best & 255u);
        if (p >= n) p = 0;                                // (cannot happen: a row is always left)
        float pv = 0.f;
#pragma unroll
        for (int a = 0; a < RA; ++a) pv = lane + 32 * a == p ? v[a] : pv;
        return __shfl_sync(0xffffffffu, pv, p & 31);
    };
    auto publish = [&](int kk, unsigned best, const float (&v)[RA], int p, float pv) {
        float pinv;                                       // 1/pivot (FP32 factors: refined in FP64)
        asm("rcp.approx.f32 %0, %1;" : "=f"(pinv) : "f"(pv));
        float *slot = ms + (kk & 1) * kSlot;
#pragma unroll
        for (int a = 0; a < RA; ++a) slot[lane + 32 * a] = lane + 32 * a == p ? 0.f : v[a] * pinv;
        // pivot row, reciprocal, 2: no finite candidate, 1: a zero pivot
        if (lane == 0)
            *reinterpret_cast<float4 *>(slot + 160) =
                make_float4(__int_as_float(p), pinv, __int_as_float(!(best & 0x80000000u) ? 2 : (best & 0x7fffff00u) == 0u), 0.f);
    };
    // Gauss-Jordan on A; all threads, ends with a block barrier
    auto invert = [&]() {
        unsigned used = 0;
#pragma unroll
        for (int a = 0; a < RA; ++a)
            if (lane + 32 * a >= n) used |= 1u << a;
        if (warp == 0) {
            float v[RA];
#pragma unroll
            for (int a = 0; a < RA; ++a) v[a] = A[a][0];
            const unsigned best = search(v, used);
            int p;
            const float pv = pivot_value(best, v, p);
            publish(0, best, v, p, pv);
        }
        __syncthreads();
#pragma unroll 1
        for (int s = 0; s < CW; ++s) {
#pragma unroll 1
            for (int o = 0; o < W; ++o) {
                const int k = s * W + o;
                if (k >= n) break;                        // uniform
                const float *slot = ms + (k & 1) * kSlot;
                const int p = __float_as_int(slot[160]);
                float m[RA], v[RA];
#pragma unroll
                for (int a = 0; a < RA; ++a) {
                    m[a] = slot[lane + 32 * a];
                    if (lane + 32 * a == p) used |= 1u << a;
                }
                // the warp that owns the next column (slot 0, or 1 where the slots are about to rotate)
                const bool next = k + 1 < n && warp == (o + 1 < W ? o + 1 : 0);
                unsigned best = 0;
                if (next) {
                    float c[RA], rn = 0.f;
#pragma unroll
                    for (int a = 0; a < RA; ++a) {
                        c[a] = o + 1 < W ? A[a][0] : A[a][1];
                        rn = lane + 32 * a == p ? c[a] : rn;
                    }
                    rn = __shfl_sync(0xffffffffu, rn, p & 31);
#pragma unroll
                    for (int a = 0; a < RA; ++a) v[a] = fmaf(-m[a], rn, c[a]);
                    best = search(v, used);
                }
                // the pivot row's slice, from its lane to all of the warp
#pragma unroll
                for (int a = 0; a < RA; ++a)
                    if (lane + 32 * a == p) {
#pragma unroll
                        for (int c = 0; c < CP; c += 4) {
                            float4 t;
                            t.x = A[a][c];
                            t.y = A[a][c + 1 < CW ? c + 1 : 0];
                            t.z = A[a][c + 2 < CW ? c + 2 : 0];
                            t.w = A[a][c + 3 < CW ? c + 3 : 0];
                            *reinterpret_cast<float4 *>(row + c) = t;
                        }
                    }
                __syncwarp();
                int pn = 0;
                float pv = 0.f;
                if (next) pv = pivot_value(best, v, pn);
                auto update = [&](int c0) {               // columns c0 .. c0 + 3
                    const float4 t = *reinterpret_cast<const float4 *>(row + c0);
                    const float r[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                    for (int a = 0; a < RA; ++a)
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            if (c0 + x < CW) A[a][c0 + x < CW ? c0 + x : 0] = fmaf(-m[a], r[x], A[a][c0 + x < CW ? c0 + x : 0]);
                };
                constexpr int CH = CP / 8 * 4;
#pragma unroll
                for (int c = 0; c < CH; c += 4) update(c);
                if (next) publish(k + 1, best, v, pn, pv);
#pragma unroll
                for (int c = CH; c < CP; c += 4) update(c);
                if (warp == o) {                          // column k itself: the inverse's column
#pragma unroll
                    for (int a = 0; a < RA; ++a) A[a][0] = lane + 32 * a == p ? 1.f : -m[a];
                }
                if (tid == 32 * ((o + 2) % W)) {          // (a warp that is not on the chain)
                    perm[k] = p;
                    kinv[p] = k;
                    srow[p] = slot[161];
                    const int flag = __float_as_int(slot[162]);
                    if (flag && s_stat == 0) s_stat = flag;
                }
                __syncthreads();
            }
#pragma unroll
            for (int a = 0; a < RA; ++a) {                // rotate: the next column of every warp first
                const float t = A[a][0];
#pragma unroll
                for (int c = 0; c + 1 < CW; ++c) A[a][c] = A[a][c + 1];
                A[a][CW - 1] = t;
            }
        }
    };
    // the inverse in natural order -> Gs -> G32 (layer l)
    auto store = [&](size_t l) {
        int pc[CW];
#pragma unroll
        for (int c = 0; c < CW; ++c) pc[c] = c * W + warp < n ? perm[c * W + warp] : -1;
#pragma unroll
        for (int a = 0; a < RA; ++a) {
            const int rr = lane + 32 * a;
            const float sc = rr < n ? srow[rr] : 0.f;
            float *g = Gs + (rr < n ? kinv[rr] : 0) * n;
#pragma unroll
            for (int c = 0; c < CW; ++c)
                if (rr < n && pc[c] >= 0) g[pc[c]] = A[a][c] * sc;
        }
        __syncthreads();
        float4 *Gl = reinterpret_cast<float4 *>(G32 + l * NNP);
        const float4 *G4 = reinterpret_cast<const float4 *>(Gs);
#pragma unroll 4
        for (int e = tid; e < NNP / 4; e += NTH) Gl[e] = G4[e];
    };
    auto prefetch = [&](size_t l) {                       // D~ of layer l -> Db
        const float *g = D32 + l * NNP;
        for (int e = tid; e < NNP / 4; e += NTH)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(Db + 4 * e)), "l"(g + 4 * e) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    for (int e = n * n + tid; e < NNP; e += NTH) Gs[e] = 0.f;
    for (int u; (u = next_half<false>(b, &s_unit, 0, 1)) >= 0;) {
        const int c = b.order[u >> 1], half = u & 1;
        if (b.active && !b.active[c]) continue;
        const int l0 = b.col_off[c], nz = b.col_end[c] - l0, mid = nz / 2;
        const int cnt = half ? nz - 1 - mid : mid;
        auto layer = [&](int t) { return (size_t)l0 + (half ? nz - 1 - t : t); };
        // the block's rows of this lane and columns of this warp
        auto load = [&](const float *D, bool schur) {
#pragma unroll
            for (int a = 0; a < RA; ++a) {
                const int rr = lane + 32 * a;
                const float al = schur && rr < n ? alpha[rr] : 0.f;
#pragma unroll
                for (int q = 0; q < CW; ++q) {
                    const int col = q * W + warp;
                    float v = 0.f;
                    if (rr < n && col < n) {
                        v = D[rr * n + col];
                        if (schur) v -= al * Gs[rr * n + col] * beta[col];
                    }
                    A[a][q] = v;
                }
            }
        };
        if (tid == 0) s_stat = 0;
        if (cnt > 0) prefetch(layer(0));
        for (int t = 0; t < cnt; ++t) {
            const size_t l = layer(t), lp = half ? l + 1 : l - 1;
            for (int q = tid; q < n && t > 0; q += NTH) {
                const double cr = half ? dB[l * n + q] : dC[l * n + q], cc = half ? dC[lp * n + q] : dB[lp * n + q];
                alpha[q] = (float)(rsc[l * n + q] * cr * csc[lp * n + q]);
                beta[q] = (float)(rsc[lp * n + q] * cc * csc[l * n + q]);
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            load(Db, t > 0);
            __syncthreads();                              // Db and Gs are free
            if (t + 1 < cnt) prefetch(layer(t + 1));
            invert();
            store(l);
        }
        if (second_half<false>(b, c, &s_unit, 0, 1)) {
            const size_t l = (size_t)l0 + mid;
            load(D32 + l * NNP, false);
            for (int side = 0; side < 2; ++side) {
                if (side == 1 && mid + 1 >= nz) break;
                const size_t lp = side ? l + 1 : l - 1;
                __syncthreads();
                for (int q = tid; q < n; q += NTH) {
                    const double cr = side ? dB[l * n + q] : dC[l * n + q], cc = side ? dC[lp * n + q] : dB[lp * n + q];
                    alpha[q] = (float)(rsc[l * n + q] * cr * csc[lp * n + q]);
                    beta[q] = (float)(rsc[lp * n + q] * cc * csc[l * n + q]);
                }
                __syncthreads();
                const float *G = G32 + lp * NNP;
#pragma unroll
                for (int a = 0; a < RA; ++a) {
                    const int rr = lane + 32 * a;
#pragma unroll
                    for (int q = 0; q < CW; ++q) {
                        const int col = q * W + warp;
                        if (rr < n && col < n) A[a][q] -= alpha[rr] * __ldcg(G + rr * n + col) * beta[col];
                    }
                }
            }
            __syncthreads();
            invert();
            store(l);
        }
        __syncthreads();
        if (tid == 0 && s_stat) atomicCAS(&status[c], 0, s_stat == 2 ? VK_ENAN : VK_ESINGULAR);
    }
}

// ---------------------------------------------------------------------------
// The tilings: rows per lane, columns per warp, warps; the
// smallest that covers the block (n <= 32 RA and n <= CW W) has the least work.
#define VK_LU32_TILINGS(X) \
    X(2, 12, 4) X(2, 16, 4) X(3, 18, 4) X(3, 24, 4) X(4, 16, 8) X(5, 10, 16)
static const int kTileCap[6] = {48, 64, 72, 96, 128, 160};
static const int kTileCW[6] = {12, 16, 18, 24, 16, 10}, kTileW[6] = {4, 4, 4, 4, 8, 16};
static int tile_of(int n) {
    int t = 0;
    while (t < 5 && kTileCap[t] < n) ++t;
    return t;
}
static size_t lu32_smem(int n, int t) { return (size_t)lu32_layout(n, kTileCW[t], kTileW[t]).end * 4 + 16; }

// vk_set_launch's variants: the smallest tiling that covers this many species
static const int kVariantCap[6] = {48, 80, 112, 160, 128, 128};
int lu32_tiling_cap(int v) { return v >= 0 && v < 6 ? kVariantCap[v] : 0; }

cudaError_t init_lu32(int n) {
    cudaError_t e = cudaSuccess;
    int t = 0;
#define SETATTR(RA, CW, W) \
    if (e == cudaSuccess && kTileCap[t] >= n) e = raise_smem_limit(k_lu32<RA, CW, W>, lu32_smem(n, t)); \
    ++t;
    VK_LU32_TILINGS(SETATTR)
#undef SETATTR
    return e;
}

void launch_lu32(const DevNet &net, const DevBatch &b, const Work &w, cudaStream_t s) {
    const int n = net.ni, v = b.lu32_tiling;
    // variants 0..3 may ask for a larger tiling than the block needs; 4 and 5 (and -1) take
    // the smallest one
    int tile = tile_of(n);
    if (v >= 0 && v < 4 && tile_of(kVariantCap[v]) > tile) tile = tile_of(kVariantCap[v]);
    const size_t sm = lu32_smem(n, tile);
    reset_queue(b, s);
    const int grid = half_grid(b, VK_TUNE_LU32, tile < 3 ? 4 : tile == 3 ? 3 : 1);
    int t = 0;
#define LAUNCH(RA, CW, W)                                                                                      \
    if (t++ == tile)                                                                                           \
        k_lu32<RA, CW, W><<<grid, 32 * W, sm, s>>>(net, b, w.D32, w.dB, w.dC, w.rs, w.cs, w.G32, w.status);
    VK_LU32_TILINGS(LAUNCH)
#undef LAUNCH
}

}  // namespace vk
