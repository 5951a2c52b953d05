// Preparation of the mixed path's FP32 factorisation (vk_lu32.cu): per layer the
// scales R_j, S_j and the dense scaled block R_j D_j S_j.
#include <cuda_runtime.h>
#include <math.h>

#include "vk_internal.cuh"
#include "vk_tma.cuh"

namespace vk {

// Biased IEEE exponent field of a double.
__device__ __forceinline__ int bexp64(double v) {
    return (int)((__double_as_longlong(v) >> 52) & 0x7ff);
}
// |v| as integer bits with NaN mapped to 0 (fmax ignores NaN operands).
__device__ __forceinline__ long long absbits_nonan(double v) {
    const long long a = __double_as_longlong(v) & 0x7fffffffffffffffll;
    return a > 0x7ff0000000000000ll ? 0ll : a;
}
// v x 2^k by the exponent field when the result stays normal (exact, as the
// FP64 product with a power of two is); returns false otherwise.
__device__ __forceinline__ bool scale_pow2(double v, int k, double &out) {
    const int E = bexp64(v);
    if (E < 1 || E > 2046 || E + k < 1 || E + k > 2046) return false;
    const long long bits = __double_as_longlong(v);
    out = __longlong_as_double((bits & ~(0x7ffll << 52)) | ((long long)(E + k) << 52));
    return true;
}
constexpr int kNoExp = -100000;        // "this row's scale has no exponent form"

// The FP64 expressions for values outside the normal range, as calls so the
// compiler branches around them instead of evaluating them for every element
// and selecting (they are FP64-pipe work).
__device__ __noinline__ int frexp_of_scaled(double v, double rs) {
    const double a = fabs(v * rs);
    if (!(a > 0.0) || !isfinite(a)) return kNoExp;
    int ex;
    frexp(a, &ex);
    return ex;
}
__device__ __noinline__ float scaled_f32(double rs, double v, double cs) {
    return (float)(rs * v * cs);
}

// Per-layer preparation for the FP32 factorisation (fully parallel over
// layers): power-of-two row scales (row maxima of D_j) and column scales
// (column maxima of R_j D_j), and the dense scaled block R_j D_j S_j rounded
// once to FP32, written with a 16-byte-aligned stride (block_stride32) for the
// bulk copies of k_lu32.
// The scales are exact powers of two, so maxima, exponents and the scaled
// values are taken from the IEEE exponent fields with integer operations --
// the FP64 pipe (about 1/60 of the FP32 rate on this chip) only adds the
// diagonal and converts to FP32; values outside the normal range take the
// FP64 expressions, which give the same results.
__global__ void __launch_bounds__(256, 6)
k_prep32(DevNet net, DevBatch b, const double *__restrict__ jv, const double *__restrict__ dA,
         const double *__restrict__ dt, float *__restrict__ D32, double *__restrict__ rsc,
         double *__restrict__ csc) {
    extern __shared__ double sp[];
    const int n = net.ni, nn = n * n, nnz = net.nnz;
    __shared__ double s_c0;
    // the CTAs stride over the layers (inactive columns' layers cost a test
    // each); every layer ends with a block barrier
    for (int l = blockIdx.x; l < b.L; l += gridDim.x) {
    const int c = b.lay_col[l];
    if (c < 0 || (b.active && !b.active[c])) continue;
    double *jls = sp;                       // [nnz]
    double *rs = jls + nnz;                 // [n]
    double *cs = rs + n;                    // [n]
    double *dg = cs + n;                    // [n] c0 - dA
    double *dd = dg + n;                    // [n] diagonal of D: -J_rr + c0 - dA_r
    float *dense = reinterpret_cast<float *>(dd + n);   // [nn]
    int *cexp = reinterpret_cast<int *>(dense + nn);    // [n]
    int *rexp = cexp + n;                   // [n] log2 rs (kNoExp: use rs)
    int *cxp = rexp + n;                    // [n] log2 cs
    const int tid = threadIdx.x, nth = blockDim.x;
    if (tid == 0) s_c0 = 1.0 / (R_ROS * dt[c]);     // one FP64 division per layer
    const double *jl = jv + (size_t)l * nnz;
    for (int e = tid; e < nnz; e += nth) jls[e] = jl[e];
    for (int e = tid; e < nn; e += nth) dense[e] = 0.0f;
    for (int t = tid; t < n; t += nth) cexp[t] = kNoExp;
    __syncthreads();
    for (int r = tid; r < n; r += nth) {
        dg[r] = s_c0 - dA[(size_t)l * n + r];
        const int e = net.jmap[r * n + r];
        dd[r] = e >= 0 ? jls[e] + dg[r] : dg[r];
    }
    __syncthreads();
    // row scales: 2^-e with |max| in [2^(e-1), 2^e)  (frexp / ldexp)
    for (int r = tid; r < n; r += nth) {
        long long m = absbits_nonan(dg[r]);
        for (int e = net.jrowptr[r]; e < net.jrowptr[r + 1]; ++e)
            m = max(m, absbits_nonan(net.jcol[e] == r ? dd[r] : jls[e]));
        const int E = (int)(m >> 52);
        if (m == 0 || E == 2047) {              // no positive finite maximum
            rs[r] = 1.0;
            rexp[r] = 0;
        } else if (E >= 1 && E <= 2044) {
            rexp[r] = 1022 - E;
            rs[r] = __longlong_as_double((long long)(1023 + 1022 - E) << 52);
        } else {                                // subnormal or huge maximum
            const double md = __longlong_as_double(m);
            int ex;
            frexp(md, &ex);
            rs[r] = ldexp(1.0, -ex);
            rexp[r] = kNoExp;
        }
    }
    __syncthreads();
    // column exponents of R_j D_j
    for (int e = tid; e < nnz + n; e += nth) {
        int r, q;
        double v;
        if (e < nnz) {
            r = net.jrow[e]; q = net.jcol[e];
            v = r == q ? dd[r] : jls[e];
        } else {
            r = q = e - nnz;
            v = dg[r];
        }
        if ((__double_as_longlong(v) & 0x7fffffffffffffffll) == 0) continue;    // v * rs = 0
        const int E = bexp64(v), k = rexp[r];
        if (k != kNoExp && E >= 1 && E <= 2046 && E + k >= 1 && E + k <= 2046) {
            atomicMax(&cexp[q], E + k - 1022);
        } else {
            const int ex = frexp_of_scaled(v, rs[r]);
            if (ex != kNoExp) atomicMax(&cexp[q], ex);
        }
    }
    __syncthreads();
    for (int t = tid; t < n; t += nth) {
        cs[t] = cexp[t] > kNoExp ? ldexp(1.0, -cexp[t]) : 1.0;
        cxp[t] = cexp[t] > kNoExp ? -cexp[t] : 0;
    }
    __syncthreads();
    // dense scaled block: (rs v) cs rounded once to FP32
    for (int e = tid; e < nnz + n; e += nth) {
        int r, q;
        double v;
        if (e < nnz) {
            r = net.jrow[e]; q = net.jcol[e];
            v = r == q ? dd[r] : jls[e];
        } else {
            r = q = e - nnz;
            if (net.jmap[r * n + r] >= 0) continue;     // the diagonal came with the Jacobian
            v = dg[r];
        }
        const int k = rexp[r];
        const long long vb = __double_as_longlong(v);
        double t1, t2;
        if ((vb & 0x7fffffffffffffffll) == 0)             // +-0 stays +-0
            dense[r * n + q] = __int_as_float((int)((unsigned long long)vb >> 32) & (int)0x80000000);
        else if (k != kNoExp && scale_pow2(v, k, t1) && scale_pow2(t1, cxp[q], t2))
            dense[r * n + q] = __double2float_rn(t2);
        else
            dense[r * n + q] = scaled_f32(rs[r], v, cs[q]);
    }
    __syncthreads();
    float *Dl = D32 + (size_t)l * block_stride32(n);
    for (int e = tid; e < nn; e += nth) Dl[e] = dense[e];
    for (int t = tid; t < n; t += nth) {
        rsc[(size_t)l * n + t] = rs[t];
        csc[(size_t)l * n + t] = cs[t];
    }
    __syncthreads();
    }
}

static size_t smem_prep(const DevNet &net) {
    const int n = net.ni;
    return (size_t)(net.nnz + 4 * n) * sizeof(double) + (size_t)n * n * sizeof(float) + 3 * n * sizeof(int) + 16;
}

// Resident CTAs per SM of k_prep32 for this network's shared memory.
int prep_blocks_per_sm(const DevNet &net) {
    int a = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_prep32, 256, smem_prep(net)) != cudaSuccess) a = 0;
    return a;
}

cudaError_t init_prep32(const DevNet &net) { return raise_smem_limit(k_prep32, smem_prep(net)); }

void launch_prep32(const DevNet &net, const DevBatch &b, const Work &w, cudaStream_t s) {
    k_prep32<<<layer_grid(b, b.grid_prep), 256, smem_prep(net), s>>>(net, b, w.jv, w.dA, w.dt, w.D32, w.rs,
                                                                     w.cs);
}

}  // namespace vk
