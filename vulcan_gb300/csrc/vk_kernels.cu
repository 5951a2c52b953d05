// Device kernels of the Ros2 kinetics-diffusion step: rates and stage (the
// block-tridiagonal solves: vk_lu64.cu, vk_mixed.cu).
//
//   k_rates      (a) rate/source: net rate of every reaction pair of one layer
//                    and the production/loss gather dy/dt, plus the transport
//                    operator; with JAC also (b): the sparse per-layer
//                    chemistry Jacobian and the diffusion coefficients that form
//                    the block-tridiagonal LHS.
//   k_stage      (d) sol, truncation error delta (masked, column max), ymix.
//
// Reference semantics: chem_funs.chemdf / neg_symjac (generated by
// make_chem_funs.py:113-430, 686-717), op.ODESolver.diffdf / diffdf_no_mol
// (op.py:1438-1597), lhs_jac_tot / lhs_jac_no_mol (op.py:1973-2042,
// 2122-2166), Ros2.solver (op.py:2860-3007).
#include <cuda_runtime.h>
#include <math.h>

#include "vk_internal.cuh"
#include "vk_geo.cuh"

namespace vk {

__device__ __forceinline__ double ipow(double x, int e) {
    double r = x;
    for (int i = 1; i < e; ++i) r = __dmul_rn(r, x);
    return r;
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Value of one side of pair p in the generated lambda order k*t1*t2*...
__device__ __forceinline__ double side_rate(double kk, const PairDesc *pd, int side,
                                            const double *yl, double M) {
    double v = kk;
    const int nt = __ldg(&pd->nt[side]);
    for (int t = 0; t < nt; ++t) {
        const int s = __ldg(&pd->tsp[side][t]);
        const double f = s < 0 ? M : yl[s];
        const int e = __ldg(&pd->tnu[side][t]);
        v = __dmul_rn(v, e == 1 ? f : ipow(f, e));
    }
    return v;
}

// ---------------------------------------------------------------------------
// (a)+(b) rate / source / Jacobian kernel: a CTA per layer at a time.  The FP64 pipe
// bounds it, so every gathered term is one FP64 instruction (the gather form
// of vk_network.cpp) and the loops a warp runs have similar lengths (pairs,
// species, half terms and Jacobian entries in decreasing order of length).
template <bool JAC>
__global__ void __launch_bounds__(128, 8)
k_rates(DevNet net, DevBatch b, const double *__restrict__ y, double *__restrict__ f,
        double *__restrict__ jv, double *__restrict__ dA, double *__restrict__ dB,
        double *__restrict__ dC, const double *__restrict__ k1, const double *__restrict__ dt,
        const double *__restrict__ geo, int flags, int chem_only) {
    extern __shared__ double sm[];
    const int ni = net.ni;
    // the CTAs stride over the layers, so layers of inactive columns cost a
    // test each rather than a CTA launch (an attempt in which few columns
    // still run launches few CTAs' worth of work); every layer ends with a
    // block barrier before the next one's shared-memory writes
    for (int l = blockIdx.x; l < b.L; l += gridDim.x) {
    const int c = b.lay_col[l];
    if (c < 0 || (b.active && !b.active[c])) continue;   // gap layer of a slot, or inactive
    const int l0 = b.col_off[c], nz = b.col_end[c] - l0;
    const int j = l - l0;
    double *yl = sm;                       // [ni + 1] layer j, then M (factor index ni)
    double *ym = yl + ni + 1;              // [ni] layer j-1
    double *yp = ym + ni;                  // [ni] layer j+1
    double *sums = yp + ni;                // [8] column sums, ysum ratios, 2/(r dt)
    double *v = sums + 8;                  // [max(npair + nxm, nh)]
    const int tid = threadIdx.x, nth = blockDim.x;
    const double *al = b.atm + (size_t)l * VK_ATM_NF;
    const double M = al[VK_ATM_M];
    for (int t = tid; t < 3 * ni; t += nth) {
        const int w = t / ni, s = t - w * ni, jj = j - 1 + w;
        const double val = (jj >= 0 && jj < nz) ? y[(size_t)(l0 + jj) * ni + s] : 0.0;
        (w == 0 ? ym : (w == 1 ? yl : yp))[s] = val;
    }
    if (tid == 0) yl[ni] = M;
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    const bool has_up = j + 1 < nz, has_dn = j > 0;
    if (warp == 0) {
        // layer sums and the state-dependent ysum ratios of the transport
        // operator, once per layer (FP64 divisions are costly on this chip)
        double s3[3];
        const double *yw[3] = {ym, yl, yp};
#pragma unroll
        for (int w = 0; w < 3; ++w) {
            double s = 0;
            for (int i = lane; i < ni; i += 32) s += yw[w][i];
            s3[w] = warp_sum(s);
        }
        if (lane == 0) {
            const double ysm = s3[0], ys0 = s3[1], ysp = s3[2];
            sums[0] = has_up ? (ysp + ys0) / (2. * ys0) : 0.0;
            sums[1] = has_dn ? (ys0 + ysm) / (2. * ys0) : 0.0;
            sums[2] = has_up ? (ysp + ys0) / (2. * ysp) : 0.0;
            sums[3] = has_dn ? (ys0 + ysm) / (2. * ysm) : 0.0;
            sums[4] = k1 ? 2. / (R_ROS * dt[c]) : 0.0;
        }
    }
    const double *kl = b.k + (size_t)l * net.nr;
    // net rate of each pair (written-order products: bit-identical to chemdf)
    for (int i = tid; i < net.npair; i += nth) {
        const int p = net.porder[i];
        const PairDesc *pd = net.pairs + p;
        const double2 kk = reinterpret_cast<const double2 *>(kl)[p];
        v[p] = side_rate(kk.x, pd, 0, yl, M) - side_rate(kk.y, pd, 1, yl, M);
    }
    __syncthreads();
    if (net.nxm > 0) {                     // products by coefficients that are not powers of two
        for (int m = tid; m < net.nxm; m += nth)
            v[net.npair + m] = __dmul_rn(net.xmul_fac[m], v[net.xmul_pair[m]]);
        __syncthreads();
    }
    // ysum ratios of the transport operator (state dependent part)
    const double qU0 = sums[0], qD0 = sums[1], qUp = sums[2], qDm = sums[3];
    const double hinv = sums[4];
    const double *gl = geo + (size_t)l * GEO_NF * ni;
    const double *spf = b.spf + (size_t)c * VK_SP_NF * ni;
    // production - loss gather (generated chemdf order, one fma per term) +
    // transport; species in decreasing order of term count
    for (int si = tid; si < ni; si += nth) {
        const int s = net.src_order[si];
        double acc = 0.0;
        for (int e = net.src_ptr[s]; e < net.src_ptr[s + 1]; ++e)
            acc = __fma_rn(net.src_c[e], v[net.src_slot[e]], acc);
        const double gU = gl[s], gD = gl[ni + s];
        double cA = -gU * qU0 - gD * qD0 + gl[2 * ni + s];
        double cB = has_up ? gU * qUp + gl[3 * ni + s] : 0.0;
        double cC = has_dn ? gD * qDm + gl[4 * ni + s] : 0.0;
        double out = acc;
        if (!chem_only) {
            double dif = cA * yl[s];
            if (has_up) dif += cB * yp[s];
            if (has_dn) dif += cC * ym[s];
            if ((flags & VK_F_TOPFLUX) && j == nz - 1)
                dif += spf[VK_SP_TOPFLUX * ni + s] / b.atm[(size_t)(l - 1) * VK_ATM_NF + VK_ATM_DZI];
            if ((flags & VK_F_BOTFLUX) && j == 0)
                dif += (spf[VK_SP_BOTFLUX * ni + s] - yl[s] * spf[VK_SP_BOTVDEP * ni + s]) / al[VK_ATM_DZI];
            out = acc + dif;
            if (k1) out = out - hinv * k1[(size_t)l * ni + s];
        }
        f[(size_t)l * ni + s] = out;
        if (JAC) {
            if ((flags & VK_F_BOTFLUX) && j == 0) cA -= spf[VK_SP_BOTVDEP * ni + s] / al[VK_ATM_DZI];
            dA[(size_t)l * ni + s] = cA;
            dB[(size_t)l * ni + s] = cB;
            dC[(size_t)l * ni + s] = cC;
        }
    }
    if (JAC) {
        __syncthreads();
        // derivative half terms: k_side x product of the side's remaining factors
        for (int h = tid; h < net.nh; h += nth) {
            double d = kl[net.hk[h]];
            for (int t = net.hptr[h]; t < net.hptr[h + 1]; ++t) d = __dmul_rn(d, yl[net.hfac[t]]);
            v[h] = d;
        }
        __syncthreads();
        double *jl = jv + (size_t)l * net.nnz;
        for (int ei = tid; ei < net.nnz; ei += nth) {
            const int e = net.jorder[ei];
            double acc = 0.0;
            for (int t = net.hjptr[e]; t < net.hjptr[e + 1]; ++t)
                acc = __fma_rn(net.hjcoef[t], v[net.hjterm[t]], acc);
            jl[e] = -acc;                      // entries of -J (neg_symjac)
        }
    }
    __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// (d) stage: sol, masked relative truncation error (column max), ymix.
__global__ void __launch_bounds__(256)
k_stage(DevNet net, DevBatch b, const double *__restrict__ y, const double *__restrict__ ymix,
        const double *__restrict__ k1, const double *__restrict__ k2,
        const double *__restrict__ yk2, double *__restrict__ sol, double *__restrict__ ymix_out,
        double *__restrict__ delta, int *__restrict__ status, int flags, double mtol, double atol) {
    __shared__ double wmax[8];
    const int n = net.ni;
    const int c = blockIdx.x;
    if (b.active && !b.active[c]) return;
    const int l0 = b.col_off[c], nz = b.col_end[c] - l0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = blockDim.x >> 5;
    const double c1 = 3. / (2. * R_ROS), c2 = 1 / (2. * R_ROS);
    // the column's largest d / sol, kept as a fraction (num, den) compared by
    // cross-multiplication and divided once per thread (an FP64 division is a
    // long FP64-pipe sequence on this chip)
    double dnum = 0.0, dden = 1.0;
    int bad = 0;
    for (int j = warp; j < nz; j += nwarp) {
        const size_t l = (size_t)l0 + j;
        double s = 0.0;
        for (int i = lane; i < n; i += 32) {
            const size_t e = l * n + i;
            double sv = __dadd_rn(__dadd_rn(y[e], __dmul_rn(c1, k1[e])), __dmul_rn(c2, k2[e]));
            sol[e] = sv;
            bad |= !isfinite(sv);
            s += sv;
            double d = fabs(sv - yk2[e]);
            if (ymix[e] < mtol) d = 0.0;
            if (sv < atol) d = 0.0;
            if ((flags & VK_F_BOTFLUX) && j == 0) d = 0.0;
            if (sv > 0.0 && d * dden > dnum * sv) { dnum = d; dden = sv; }
        }
        s = warp_sum(s);
        for (int i = lane; i < n; i += 32) ymix_out[l * n + i] = sol[l * n + i] / s;
    }
    double dmax = dnum / dden;
    for (int o = 16; o; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    if (lane == 0) wmax[warp] = dmax;
    bad = __syncthreads_or(bad);
    if (tid == 0) {
        if (bad && status[c] == 0) status[c] = VK_ENAN;
        double m = 0.0;
        for (int w = 0; w < nwarp; ++w) m = fmax(m, wmax[w]);
        delta[c] = m;
    }
}

// Transport geometry of every (layer, species) of the active columns.
__global__ void __launch_bounds__(256)
k_geometry(DevNet net, DevBatch b, double *__restrict__ geo, int flags) {
    const int ni = net.ni;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)b.L * ni) return;
    const int l = (int)(e / ni), i = (int)(e - (long long)l * ni);
    const int c = b.lay_col[l];
    if (c < 0 || (b.active && !b.active[c])) return;
    const GeoCol cv = make_geocol(b.atm, b.Dzz, b.spf, b.col_off, b.col_end, c, ni);
    double out[GEO_NF];
    geo_coef(cv, l - cv.l0, i, flags, out);
    double *gl = geo + (size_t)l * GEO_NF * ni;
    for (int k = 0; k < GEO_NF; ++k) gl[k * ni + i] = out[k];
}

void launch_geometry(const DevNet &net, const DevBatch &b, double *geo, int flags, cudaStream_t s) {
    long long n = (long long)b.L * net.ni;
    k_geometry<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(net, b, geo, flags);
}

// ---------------------------------------------------------------------------
static size_t rates_smem(const DevNet &net);
// Opt the kernels into the dynamic shared memory this network needs; called
// once per handle, outside any stream capture.
cudaError_t init_kernels(const DevNet &net) {
    size_t sr = rates_smem(net);
    cudaError_t e;
    if ((e = raise_smem_limit(k_rates<true>, (int)sr))) return e;
    if ((e = raise_smem_limit(k_rates<false>, (int)sr))) return e;
    if ((e = init_lu64(net.ni))) return e;
    return cudaSuccess;
}

static size_t rates_smem(const DevNet &net) {
    const int m = net.npair + net.nxm > net.nh ? net.npair + net.nxm : net.nh;
    return (size_t)(3 * net.ni + 1 + 8 + m) * sizeof(double);
}

void launch_rates(const DevNet &net, const DevBatch &b, const double *y, double *f,
                  double *jv, double *dA, double *dB, double *dC, const double *k1,
                  const double *dt, const double *geo, int flags, bool with_jac, cudaStream_t s) {
    size_t sm = rates_smem(net);
    const int grid = layer_grid(b, b.grid_rates);
    if (with_jac)
        k_rates<true><<<grid, 128, sm, s>>>(net, b, y, f, jv, dA, dB, dC, k1, dt, geo, flags, 0);
    else
        k_rates<false><<<grid, 128, sm, s>>>(net, b, y, f, jv, dA, dB, dC, k1, dt, geo, flags, 0);
}

// Resident CTAs per SM of k_rates (the larger of its two forms' register
// footprints sets it) for this network's shared memory.
int rates_blocks_per_sm(const DevNet &net) {
    const size_t sm = rates_smem(net);
    int a = 0, c = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_rates<true>, 128, sm) != cudaSuccess) a = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k_rates<false>, 128, sm) != cudaSuccess) c = 0;
    return a < c ? a : c;
}

void launch_chem_only(const DevNet &net, const DevBatch &b, const double *y, double *f,
                      const double *geo, cudaStream_t s) {
    size_t sm = rates_smem(net);
    k_rates<false><<<layer_grid(b, b.grid_rates), 128, sm, s>>>(net, b, y, f, nullptr, nullptr, nullptr, nullptr,
                                        nullptr, nullptr, geo, 0, 1);
}

void launch_stage(const DevNet &net, const DevBatch &b, const Work &w, int flags, double mtol,
                  double atol, cudaStream_t s) {
    k_stage<<<b.ncols, 256, 0, s>>>(net, b, w.y, w.ymix, w.k1, w.k2, w.yk2, w.sol, w.ymix_out,
                                    w.delta, w.status, flags, mtol, atol);
}

}  // namespace vk
