// BF16 MLP kernels for the learned warm start (forward, backward, Adam).
//
// The network proposes a near-steady log mixing-ratio profile per layer; it
// has no counterpart in the reference.  Weights and activations are BF16,
// accumulation FP32 (tensor-core mma.sync m16n8k16), master weights and
// optimiser state FP32.  All buffers are device pointers owned by the caller.
//
//   forward layer   Z = X W + b,  H = silu(Z) (or Z)          X [B,K], W [K,N]
//   backward layer  dZ = dH o silu'(Z);  dW = X^T dZ;  db = sum_rows dZ;
//                   dX = dZ W^T
//   Adam            m, v, w (FP32) and the BF16 copy of w
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "vk_internal.cuh"

namespace {

constexpr int BM = 128, BN = 64, BK = 64;     // CTA tile; 8 warps of 32x32
constexpr int STAGES = 3;                     // K tiles in flight (cp.async)
constexpr int PAD = 8;                        // bf16s: 16-byte rows, conflict-free ldmatrix
constexpr int GEMM_THREADS = 256;

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

enum Epi { EPI_FWD = 0, EPI_F32 = 1 };

// A ROWS x COLS tile of the row-major matrix src[nr][nc] at (r0, c0), zero
// outside it, into dst[ROWS][COLS + PAD]: asynchronous copies of CH elements,
// the largest chunk (16, 8 or 4 bytes) every row starts on, element loads
// (eight in flight) where rows start on 2 bytes only.
template <int ROWS, int COLS, int CH>
__device__ __forceinline__ void load_chunks(__nv_bfloat16 *dst, const __nv_bfloat16 *__restrict__ src, int nr,
                                            int nc, int r0, int c0) {
    constexpr int PER = COLS / CH;
#pragma unroll 8
    for (int e = threadIdx.x; e < ROWS * PER; e += GEMM_THREADS) {
        const int r = e / PER, c = (e - r * PER) * CH;
        const int gr = r0 + r, gc = c0 + c;
        const int bytes = (gr < nr && gc < nc) ? 2 * min(CH, nc - gc) : 0;
        const __nv_bfloat16 *g = bytes ? src + (long long)gr * nc + gc : src;
        const uint32_t d = smem_addr(dst + r * (COLS + PAD) + c);
        if (CH == 8)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g), "r"(bytes) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;"
                         ::"r"(d), "l"(g), "n"(CH * 2), "r"(bytes) : "memory");
    }
}
template <int ROWS, int COLS>
__device__ __forceinline__ void load_tile(__nv_bfloat16 *dst, const __nv_bfloat16 *__restrict__ src, int nr,
                                          int nc, int r0, int c0, int chunk) {
    if (chunk == 8) load_chunks<ROWS, COLS, 8>(dst, src, nr, nc, r0, c0);
    else if (chunk == 4) load_chunks<ROWS, COLS, 4>(dst, src, nr, nc, r0, c0);
    else if (chunk == 2) load_chunks<ROWS, COLS, 2>(dst, src, nr, nc, r0, c0);
    else {
        const __nv_bfloat16 zero = __float2bfloat16(0.0f);
        for (int e = threadIdx.x; e < ROWS * COLS; e += 8 * GEMM_THREADS) {
            __nv_bfloat16 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int f = e + u * GEMM_THREADS, r = f / COLS, c = f - r * COLS;
                const int gr = r0 + r, gc = c0 + c;
                v[u] = (gr < nr && gc < nc) ? src[(long long)gr * nc + gc] : zero;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int f = e + u * GEMM_THREADS, r = f / COLS, c = f - r * COLS;
                dst[r * (COLS + PAD) + c] = v[u];
            }
        }
    }
}

template <bool AT, bool BT>
struct GemmSmem {                              // bf16s of one stage
    static constexpr int A = AT ? BK * (BM + PAD) : BM * (BK + PAD);
    static constexpr int B = BT ? BN * (BK + PAD) : BK * (BN + PAD);
    static constexpr int bytes = STAGES * (A + B) * 2;
};

// C[M,N] = sum_k A(m,k) B(k,n) of row-major matrices: A is [M][K], or [K][M]
// with AT; B is [K][N], or [N][K] with BT.
// EPI_FWD: Z = C + bias (FP32, optional), H = bf16(silu?(Z)) (optional).
// EPI_F32: Cf = C.
// Tensor-core mma.sync with FP32 accumulators; a layer is 2 GFLOP at most, so
// the latency of filling a tile's K loop and the launches bound it, not the
// tensor rate.  A product with few tiles and a long K (dW: 32 tiles, K = the
// batch) is split over the CTAs of a cluster (gridDim.z); they add their
// partial tiles through distributed shared memory in rank order, so the
// result is deterministic.  4096 x 512 x 512 on a GB300, before (64 x 64 tiles,
// element loads, no split) -> now, warm caches: forward 124 -> 17 us, dW
// 548 -> 17 us, dX 113 -> 12 us.
template <bool AT, bool BT, int EPI, bool VEC>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
k_gemm_bf16(int M, int N, int K, const __nv_bfloat16 *__restrict__ A, int chunkA,
            const __nv_bfloat16 *__restrict__ B, int chunkB, const float *__restrict__ bias,
            float *__restrict__ Z, __nv_bfloat16 *__restrict__ H, int act, float *__restrict__ Cf, bool even) {
    using L = GemmSmem<AT, BT>;
    const int chA = VEC ? 8 : chunkA, chB = VEC ? 8 : chunkB;    // VEC: the other paths compile away
    extern __shared__ __align__(16) unsigned char smraw[];
    __nv_bfloat16 *As = reinterpret_cast<__nv_bfloat16 *>(smraw);
    __nv_bfloat16 *Bs = As + STAGES * L::A;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    const int kt = (K + BK - 1) / BK;                       // K tiles, this CTA's share
    const int split = gridDim.z, t0 = (int)((long long)kt * blockIdx.z / split);
    const int t1 = (int)((long long)kt * (blockIdx.z + 1) / split);
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0f;
    auto fetch = [&](int t) {
        if (t < t1) {
            const int s = (t - t0) % STAGES, k0 = t * BK;
            if (AT) load_tile<BK, BM>(As + s * L::A, A, K, M, k0, m0, chA);
            else load_tile<BM, BK>(As + s * L::A, A, M, K, m0, k0, chA);
            if (BT) load_tile<BN, BK>(Bs + s * L::B, B, N, K, n0, k0, chB);
            else load_tile<BK, BN>(Bs + s * L::B, B, K, N, k0, n0, chB);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) fetch(t0 + s);
    // ldmatrix row addresses of this lane: matrix g = lane / 8, row lane % 8
    const int lr = lane & 7, lg = lane >> 3;
    for (int t = t0; t < t1; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                    // tile t landed; tile t - 1 is free
        fetch(t + STAGES - 1);
        __syncwarp();                                       // ldmatrix and mma need the whole warp
        const __nv_bfloat16 *as = As + ((t - t0) % STAGES) * L::A, *bs = Bs + ((t - t0) % STAGES) * L::B;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
            uint32_t af[2][4], bf[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                // matrices (m, k): (0,0) (8,0) (0,8) (8,8)
                const int mr = wm + 16 * i + (lg & 1) * 8, kc = kk + (lg >> 1) * 8;
                if (AT) ldmatrix_x4_trans(af[i], smem_addr(as + (kc + lr) * (BM + PAD) + mr));
                else ldmatrix_x4(af[i], smem_addr(as + (mr + lr) * (BK + PAD) + kc));
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                // matrices (k, n): (0,0) (8,0) of columns 16 j, then of 16 j + 8
                const int kc = kk + (lg & 1) * 8, nc = wn + 16 * j + (lg >> 1) * 8;
                if (BT) ldmatrix_x4(bf[j], smem_addr(bs + (nc + lr) * (BK + PAD) + kc));
                else ldmatrix_x4_trans(bf[j], smem_addr(bs + (kc + lr) * (BN + PAD) + nc));
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t b2[2] = {bf[j >> 1][(j & 1) * 2], bf[j >> 1][(j & 1) * 2 + 1]};
                    mma_bf16(acc[i][j], af[i], b2);
                }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const int g = lane >> 2, tq = lane & 3;
    if (split > 1) {
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        float *P = reinterpret_cast<float *>(smraw);        // [BM][BN + 4] partial tile
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 4; q += 2)
                    *reinterpret_cast<float2 *>(P + (wm + 16 * i + g + (q ? 8 : 0)) * (BN + 4) + wn + 8 * j + 2 * tq) =
                        make_float2(acc[i][j][q], acc[i][j][q + 1]);
        cl.sync();
        // rank z adds rows [z BM / split, (z + 1) BM / split) of every partial
        // tile, all ranks' values of an element in flight at once
        const int rows = BM / split;
        for (int e = tid; e < rows * (BN / 4); e += GEMM_THREADS) {
            const int r = (int)blockIdx.z * rows + e / (BN / 4), c = (e % (BN / 4)) * 4;
            float4 p[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < split) p[u] = *reinterpret_cast<const float4 *>(cl.map_shared_rank(P, u) + r * (BN + 4) + c);
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < split) { v[0] += p[u].x; v[1] += p[u].y; v[2] += p[u].z; v[3] += p[u].w; }
            if (m0 + r >= M) continue;
            float *o = Cf + (long long)(m0 + r) * N + n0 + c;
#pragma unroll
            for (int x = 0; x < 4; ++x)
                if (n0 + c + x < N) o[x] = v[x];
        }
        cl.sync();
        return;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                const int m = m0 + wm + 16 * i + g + (q ? 8 : 0);
                const int n = n0 + wn + 8 * j + 2 * tq;
                if (m >= M || n >= N) continue;
                float v[2] = {acc[i][j][q], acc[i][j][q + 1]};
                const long long o = (long long)m * N + n;
                const int cnt = n + 1 < N ? 2 : 1;
                if (EPI == EPI_FWD) {
                    float h[2];
                    for (int x = 0; x < cnt; ++x) {
                        v[x] += bias ? bias[n + x] : 0.0f;
                        h[x] = act ? silu(v[x]) : v[x];
                    }
                    if (Z) {
                        if (even) *reinterpret_cast<float2 *>(Z + o) = make_float2(v[0], v[1]);
                        else for (int x = 0; x < cnt; ++x) Z[o + x] = v[x];
                    }
                    if (H) {
                        if (even) *reinterpret_cast<__nv_bfloat162 *>(H + o) = __floats2bfloat162_rn(h[0], h[1]);
                        else for (int x = 0; x < cnt; ++x) H[o + x] = __float2bfloat16(h[x]);
                    }
                } else if (even) {
                    *reinterpret_cast<float2 *>(Cf + o) = make_float2(v[0], v[1]);
                } else {
                    for (int x = 0; x < cnt; ++x) Cf[o + x] = v[x];
                }
            }
}

// dZ = dH o silu'(Z) (or dH) -> BF16 and its column sums db (may be NULL), in
// one pass over the rows: a cluster of gridDim.y CTAs takes 16 columns, each
// CTA a contiguous part of the rows (16 threads a row, 16 rows at a time, eight
// such steps' loads in flight: reading dH and Z, 16.8 MB at 4096 x 512, bounds
// it); the partial sums are added in a fixed order, so db is deterministic.
// Two kernels before, 8 + 237 us (one thread per column sum), now 7 us.
constexpr int ACT_COLS = 16, ACT_U = 8;
__global__ void __launch_bounds__(256)
k_act_bwd(int M, int N, const float *__restrict__ dH, const float *__restrict__ Z, int act,
          __nv_bfloat16 *__restrict__ dZ, float *__restrict__ db) {
    __shared__ float part[256];
    __shared__ float mine[ACT_COLS];
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int col = threadIdx.x & (ACT_COLS - 1), row = threadIdx.x / ACT_COLS;
    constexpr int RSTEP = 256 / ACT_COLS;
    const int n = blockIdx.x * ACT_COLS + col;
    const int r0 = (int)((long long)M * blockIdx.y / gridDim.y);
    const int r1 = (int)((long long)M * (blockIdx.y + 1) / gridDim.y);
    float s = 0.0f;
    if (n < N) {
        for (int m = r0 + row; m < r1; m += ACT_U * RSTEP) {
            float d[ACT_U], z[ACT_U];
#pragma unroll
            for (int u = 0; u < ACT_U; ++u) {
                const int mm = m + u * RSTEP;
                const long long o = (long long)mm * N + n;
                d[u] = mm < r1 ? dH[o] : 0.0f;
                z[u] = act && mm < r1 ? Z[o] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < ACT_U; ++u) {
                const int mm = m + u * RSTEP;
                if (mm >= r1) break;
                const __nv_bfloat16 v = __float2bfloat16(act ? d[u] * dsilu(z[u]) : d[u]);
                dZ[(long long)mm * N + n] = v;
                s += __bfloat162float(v);
            }
        }
    }
    if (!db) return;                                        // uniform
    part[threadIdx.x] = s;
    __syncthreads();
    if (row == 0) {
        float t = part[col];
        for (int w = 1; w < RSTEP; ++w) t += part[w * ACT_COLS + col];
        mine[col] = t;
    }
    cl.sync();
    if (blockIdx.y == 0 && row == 0 && n < N) {
        float t = 0.0f;
        for (int u = 0; u < (int)gridDim.y; ++u) t += cl.map_shared_rank(mine, u)[col];
        db[n] = t;
    }
    cl.sync();
}

__global__ void k_adam(long long n, float *__restrict__ w, __nv_bfloat16 *__restrict__ wb,
                       const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16(wi);
}

int mlp_fail(const char *msg) {
    vk::set_global_error(msg);
    return VK_EINVAL;
}

int launch_check(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        vk::set_global_error(std::string(what) + ": " + cudaGetErrorString(e));
        return VK_ECUDA;
    }
    return VK_OK;
}

}  // namespace

namespace {

// Elements of the largest copy (16, 8, 4 or 2 bytes) every row of ld elements starts on.
int row_chunk(const void *p, int ld) {
    for (int c = 8; c > 1; c /= 2)
        if (((uintptr_t)p & (2 * c - 1)) == 0 && ld % c == 0) return c;
    return 1;
}

// CTAs a product's K loop is split over: none while its tiles fill the chip's
// SMs or its K loop is short, else up to a portable cluster's 8.
int gemm_split(int M, int N, int K) {
    const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN), kt = (K + BK - 1) / BK;
    int s = 1;
    while (s < 8 && tiles * s < 128 && kt / (2 * s) >= 2) s *= 2;
    return s;
}

template <bool AT, bool BT, int EPI>
cudaError_t launch_gemm(int M, int N, int K, const __nv_bfloat16 *A, const __nv_bfloat16 *B, const float *bias,
                        float *Z, __nv_bfloat16 *H, int act, float *Cf, cudaStream_t s) {
    constexpr int sm = GemmSmem<AT, BT>::bytes;
    static_assert(sm >= BM * (BN + 4) * 4, "the partial tile of a split product reuses the stages");
    const int chA = row_chunk(A, AT ? M : K), chB = row_chunk(B, BT ? K : N);
    auto kernel = chA == 8 && chB == 8 ? k_gemm_bf16<AT, BT, EPI, true> : k_gemm_bf16<AT, BT, EPI, false>;
    cudaError_t e = raise_smem_limit(kernel, sm);
    if (e != cudaSuccess) return e;
    const int split = EPI == EPI_F32 ? gemm_split(M, N, K) : 1;
    // pairs of output columns are stored at once where that is aligned
    const bool pairs = N % 2 == 0 && (((uintptr_t)Z | (uintptr_t)Cf) & 7) == 0 && ((uintptr_t)H & 3) == 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = (unsigned)split;
    cfg.gridDim = dim3((N + BN - 1) / BN, (M + BM - 1) / BM, split);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = split > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, M, N, K, A, chA, B, chB, bias, Z, H, act, Cf, pairs);
}

}  // namespace

extern "C" int vk_mlp_forward(int B, int K, int N, const void *X, const void *W, const float *bias,
                              float *Z, void *H, int silu_act, void *stream) {
    if (B <= 0 || K <= 0 || N <= 0 || !X || !W) return mlp_fail("vk_mlp_forward: bad arguments");
    if (!Z && !H) return mlp_fail("vk_mlp_forward: no output");
    launch_gemm<false, false, EPI_FWD>(B, N, K, (const __nv_bfloat16 *)X, (const __nv_bfloat16 *)W, bias, Z,
                                       (__nv_bfloat16 *)H, silu_act, nullptr, (cudaStream_t)stream);
    return launch_check("vk_mlp_forward");
}

extern "C" int vk_mlp_backward(int B, int K, int N, const void *X, const void *W, const float *Z,
                               const float *dH, int silu_act, void *dZ_scratch, float *dW,
                               float *db, float *dX, void *stream) {
    if (B <= 0 || K <= 0 || N <= 0 || !X || !W || !Z || !dH || !dZ_scratch)
        return mlp_fail("vk_mlp_backward: bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    __nv_bfloat16 *dZ = (__nv_bfloat16 *)dZ_scratch;
    {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = at[0].val.clusterDim.z = 1;
        at[0].val.clusterDim.y = 8;
        cfg.gridDim = dim3((N + ACT_COLS - 1) / ACT_COLS, 8);
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k_act_bwd, B, N, dH, Z, silu_act, dZ, db);
    }
    if (dW)     // dW[K,N] = X^T dZ
        launch_gemm<true, false, EPI_F32>(K, N, B, (const __nv_bfloat16 *)X, dZ, nullptr, nullptr, nullptr, 0,
                                          dW, s);
    if (dX)     // dX[B,K] = dZ W^T
        launch_gemm<false, true, EPI_F32>(B, K, N, dZ, (const __nv_bfloat16 *)W, nullptr, nullptr, nullptr, 0,
                                          dX, s);
    return launch_check("vk_mlp_backward");
}

extern "C" int vk_mlp_adam(long long n, float *w, void *w_bf16, const float *g, float *m, float *v,
                           float lr, float beta1, float beta2, float eps, int step, void *stream) {
    if (n <= 0 || !w || !g || !m || !v || step < 1) return mlp_fail("vk_mlp_adam: bad arguments");
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    k_adam<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        n, w, (__nv_bfloat16 *)w_bf16, g, m, v, lr, beta1, beta2, eps, c1, c2);
    return launch_check("vk_mlp_adam");
}
