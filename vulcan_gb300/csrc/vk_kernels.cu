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
// (species s at yl[s TL]).
template <int TL>
__device__ __forceinline__ double side_rate(double kk, const PairDesc *pd, int side,
                                            const double *yl, double M) {
    double v = kk;
    const int nt = __ldg(&pd->nt[side]);
    for (int t = 0; t < nt; ++t) {
        const int s = __ldg(&pd->tsp[side][t]);
        const double f = s < 0 ? M : yl[s * TL];
        const int e = __ldg(&pd->tnu[side][t]);
        v = __dmul_rn(v, e == 1 ? f : ipow(f, e));
    }
    return v;
}

// ---------------------------------------------------------------------------
// (a)+(b) rate / source / Jacobian kernel: a CTA per tile of TL layers at a time,
// TL = 1, 2 or 4; lane = (item, layer of the tile), the layer fastest, so a warp
// runs 32 / TL items (pairs, species, half terms, Jacobian entries, sorted by
// decreasing length) and shared memory is [item][layer].
// What bounds it: the FP64 unit.  Every gathered term is one FP64 instruction (the
// gather form of vk_network.cpp), and a warp issues as many as its longest item
// has: with 32 items a warp the 69-species network takes 157 FMAs for a layer's
// sources, 50 if the lanes were all busy, 284 for its Jacobian instead of 174.
// The call with the Jacobian: 512 columns (66 560 layers) of 69 species 3.82 ->
// 2.49 ms, 48 columns of 150 species 1.53 -> 1.30 (a CTA a layer, before).
template <int TL, bool JAC>
__global__ void __launch_bounds__(TL == 1 ? 128 : 256, TL == 1 ? 8 : 4)
k_rates(DevNet net, DevBatch b, const double *__restrict__ y, double *__restrict__ f,
         double *__restrict__ jv, double *__restrict__ dA, double *__restrict__ dB,
         double *__restrict__ dC, const double *__restrict__ k1, const double *__restrict__ dt,
         const double *__restrict__ geo, int flags, int chem_only) {
    extern __shared__ double sm[];
    const int ni = net.ni;
    const int tid = threadIdx.x, nth = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int li = tid & (TL - 1);         // this thread's layer of the tile
    const int i0 = tid / TL, di = nth / TL;
    double *yl = sm + li;                  // [ni + 1][TL] the layer, then M (factor index ni)
    double *ym = sm + (ni + 1) * TL + li;  // [ni][TL] the layer below
    double *yp = ym + ni * TL;             // [ni][TL] the layer above
    double *sums = sm + (3 * ni + 1) * TL + li;     // [5][TL] ysum ratios, 2/(r dt)
    double *rsum = sm + (3 * ni + 6) * TL; // [TL + 2] sums over the species
    double *v = sm + (3 * ni + 9) * TL + li;        // [max(npair + nxm, nh)][TL]
    // the CTAs stride over the tiles, so layers of inactive columns cost a
    // test each rather than a CTA launch (an attempt in which few columns
    // still run launches few CTAs' worth of work); every tile ends with a
    // block barrier before the next one's shared-memory writes
    const int ntile = (b.L + TL - 1) / TL;
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int lt = tile * TL;
    // this thread's layer: a gap layer of a slot and an inactive column's have no work
    const int l = lt + li;
    const int c = l < b.L ? b.lay_col[l] : -1;
    const bool on = c >= 0 && !(b.active && !b.active[c]);
    if (TL == 1) {
        if (!on) continue;
    } else {
        if (!__syncthreads_or(on)) continue;
    }
    const int l0 = on ? b.col_off[c] : 0, nz = on ? b.col_end[c] - l0 : 0;
    const int j = l - l0;
    const bool has_up = on && j + 1 < nz, has_dn = on && j > 0;
    const double *al = b.atm + (size_t)l * VK_ATM_NF;
    const double M = on ? al[VK_ATM_M] : 0.0;
    if (TL == 1) {
        for (int t = tid; t < 3 * ni; t += nth) {
            const int w = t / ni, s = t - w * ni, jj = j - 1 + w;
            const double val = (jj >= 0 && jj < nz) ? y[(size_t)(l0 + jj) * ni + s] : 0.0;
            (w == 0 ? ym : (w == 1 ? yl : yp))[s] = val;
        }
    } else {
        // rows of the tile and its two neighbours, each to the layers it serves
        for (int t = tid; t < (TL + 2) * ni; t += nth) {
            const int w = t / ni, s = t - w * ni, row = lt - 1 + w;
            const double val = row >= 0 && row < b.L ? y[(size_t)row * ni + s] : 0.0;
            if (w >= 1 && w <= TL) sm[s * TL + w - 1] = val;
            if (w < TL) sm[(ni + 1 + s) * TL + w] = val;
            if (w >= 2) sm[(2 * ni + 1 + s) * TL + w - 2] = val;
        }
    }
    if (i0 == 0) yl[ni * TL] = M;
    __syncthreads();
    // sums of the tile's rows and its two neighbours', a warp each
    for (int w = warp; w < TL + 2; w += nth >> 5) {
        // (row lt - 1 + w: the layer below the first, the layers, the one above the last)
        const double *yw = w == 0 ? sm + (ni + 1) * TL : w <= TL ? sm + w - 1 : sm + (2 * ni + 1) * TL + TL - 1;
        double t = 0;
        for (int i = lane; i < ni; i += 32) t += yw[i * TL];
        t = warp_sum(t);
        if (lane == 0) rsum[w] = t;
    }
    const double *kl = b.k + (size_t)l * net.nr;
    // net rate of each pair (written-order products: bit-identical to chemdf)
    if (on)
        for (int i = i0; i < net.npair; i += di) {
            const int p = net.porder[i];
            const PairDesc *pd = net.pairs + p;
            const double2 kk = reinterpret_cast<const double2 *>(kl)[p];
            v[p * TL] = side_rate<TL>(kk.x, pd, 0, yl, M) - side_rate<TL>(kk.y, pd, 1, yl, M);
        }
    __syncthreads();
    // the state-dependent ysum ratios of the transport operator and 2/(r dt):
    // one division per lane of one warp (an FP64 division is a long sequence
    // on this chip, however many lanes take part)
    if (warp == (nth >> 5) - 1 && lane < 5 * TL) {
        const int q = lane / TL;
        const double ysm = rsum[li], ys0 = rsum[li + 1], ysp = rsum[li + 2];
        const bool there = q == 4 ? k1 && on : q & 1 ? has_dn : has_up;
        const double num = q == 4 ? 2. : q & 1 ? ys0 + ysm : ysp + ys0;
        const double den = q == 4 ? (there ? R_ROS * dt[c] : 1.) : 2. * (q < 2 ? ys0 : q == 2 ? ysp : ysm);
        sums[q * TL] = there ? num / den : 0.0;
    }
    if (net.nxm > 0 && on)                 // products by coefficients that are not powers of two
        for (int m = i0; m < net.nxm; m += di)
            v[(net.npair + m) * TL] = __dmul_rn(net.xmul_fac[m], v[net.xmul_pair[m] * TL]);
    __syncthreads();
    // ysum ratios of the transport operator (state dependent part)
    const double qU0 = sums[0], qD0 = sums[TL], qUp = sums[2 * TL], qDm = sums[3 * TL];
    const double hinv = sums[4 * TL];
    const double *gl = geo + (size_t)l * GEO_NF * ni;
    const double *spf = b.spf + (size_t)(on ? c : 0) * VK_SP_NF * ni;
    // production - loss gather (generated chemdf order, one fma per term) +
    // transport; species in decreasing order of term count
    if (on)
        for (int si = i0; si < ni; si += di) {
            const int s = net.src_order[si];
            double acc = 0.0;
            for (int e = net.src_ptr[s]; e < net.src_ptr[s + 1]; ++e)
                acc = __fma_rn(net.src_c[e], v[net.src_slot[e] * TL], acc);
            const double gU = gl[s], gD = gl[ni + s];
            // (written out: every TL rounds alike)
            double cA = __dadd_rn(__fma_rn(-gD, qD0, __dmul_rn(-gU, qU0)), gl[2 * ni + s]);
            double cB = has_up ? __fma_rn(gU, qUp, gl[3 * ni + s]) : 0.0;
            double cC = has_dn ? __fma_rn(gD, qDm, gl[4 * ni + s]) : 0.0;
            double out = acc;
            if (!chem_only) {
                double dif = __dmul_rn(cA, yl[s * TL]);
                if (has_up) dif = __fma_rn(cB, yp[s * TL], dif);
                if (has_dn) dif = __fma_rn(cC, ym[s * TL], dif);
                if ((flags & VK_F_TOPFLUX) && j == nz - 1)
                    dif += spf[VK_SP_TOPFLUX * ni + s] / b.atm[(size_t)(l - 1) * VK_ATM_NF + VK_ATM_DZI];
                if ((flags & VK_F_BOTFLUX) && j == 0)
                    dif += __fma_rn(-yl[s * TL], spf[VK_SP_BOTVDEP * ni + s], spf[VK_SP_BOTFLUX * ni + s]) / al[VK_ATM_DZI];
                out = acc + dif;
                if (k1) out = __fma_rn(-hinv, k1[(size_t)l * ni + s], out);
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
        if (on)
            for (int h = i0; h < net.nh; h += di) {
                double d = kl[net.hk[h]];
                for (int t = net.hptr[h]; t < net.hptr[h + 1]; ++t) d = __dmul_rn(d, yl[net.hfac[t] * TL]);
                v[h * TL] = d;
            }
        __syncthreads();
        double *jl = jv + (size_t)l * net.nnz;
        if (on)
            for (int ei = i0; ei < net.nnz; ei += di) {
                const int e = net.jorder[ei];
                double acc = 0.0;
                for (int t = net.hjptr[e]; t < net.hjptr[e + 1]; ++t)
                    acc = __fma_rn(net.hjcoef[t], v[net.hjterm[t] * TL], acc);
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

// Transport geometry of every (layer, species) of the active columns, a CTA per
// kGeoTile layers.  FP64 divisions bound it: those of a layer alone are done
// once a layer, 10 of 28 are left per species.  66 752 layers of 69 species
// 1.88 -> 1.08 ms (every division per species before).
constexpr int kGeoTile = 8;
__global__ void __launch_bounds__(256)
k_geometry(DevNet net, DevBatch b, double *__restrict__ geo, int flags) {
    __shared__ GeoLayer lay[kGeoTile];
    const int ni = net.ni, lt = blockIdx.x * kGeoTile;
    auto column = [&](int l) {             // -1: no work
        const int c = l < b.L ? b.lay_col[l] : -1;
        return c >= 0 && !(b.active && !b.active[c]) ? c : -1;
    };
    if (threadIdx.x < kGeoTile) {
        const int l = lt + threadIdx.x, c = column(l);
        if (c >= 0) {
            const GeoCol cv = make_geocol(b.atm, b.Dzz, b.spf, b.col_off, b.col_end, c, ni);
            lay[threadIdx.x] = geo_layer(cv, l - cv.l0, flags);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kGeoTile * ni; e += blockDim.x) {
        const int t = e / ni, i = e - t * ni, l = lt + t, c = column(l);
        if (c < 0) continue;
        const GeoCol cv = make_geocol(b.atm, b.Dzz, b.spf, b.col_off, b.col_end, c, ni);
        double out[GEO_NF];
        geo_species(cv, lay[t], l - cv.l0, i, flags, out);
        double *gl = geo + (size_t)l * GEO_NF * ni;
        for (int k = 0; k < GEO_NF; ++k) gl[k * ni + i] = out[k];
    }
}

void launch_geometry(const DevNet &net, const DevBatch &b, double *geo, int flags, cudaStream_t s) {
    k_geometry<<<(b.L + kGeoTile - 1) / kGeoTile, 256, 0, s>>>(net, b, geo, flags);
}

// ---------------------------------------------------------------------------
static size_t rates_smem(const DevNet &net, int tl) {
    const int m = net.npair + net.nxm > net.nh ? net.npair + net.nxm : net.nh;
    return (size_t)tl * (3 * net.ni + 1 + 8 + m) * sizeof(double);
}
// A tile of more than one layer leaves room for a second CTA on the SM.
static bool rates_fits(const DevNet &net, int tl) { return tl == 1 || rates_smem(net, tl) <= 112 * 1024; }
// Layers per tile (log2): one while every layer can have an SM of its own, four
// where the tiles still give each SM three CTAs, two between (the two calls of
// an attempt, 69 species, with tiles of 1, 2 and 4: 150 layers 0.046, 0.045 and
// 0.066 ms, 1200 layers 0.077, 0.068 and 0.076, 2400 layers 0.151, 0.129 and
// 0.101; of 8 layers 0.098).
static int rates_tile(const DevNet &net, const DevBatch &b) {
    int i = b.L <= b.nsm ? 0 : b.L < 12 * b.nsm ? 1 : 2;
    while (i > 0 && !rates_fits(net, 1 << i)) --i;
    return i;
}
// Opt the kernels into the dynamic shared memory this network needs; called
// once per handle, outside any stream capture.
cudaError_t init_kernels(const DevNet &net) {
    cudaError_t e = init_lu64(net.ni);
#define SET(TL)                                                                                     \
    if (e == cudaSuccess && rates_fits(net, TL)) e = raise_smem_limit(k_rates<TL, true>, rates_smem(net, TL)); \
    if (e == cudaSuccess && rates_fits(net, TL)) e = raise_smem_limit(k_rates<TL, false>, rates_smem(net, TL));
    SET(1) SET(2) SET(4)
#undef SET
    return e;
}

void launch_rates(const DevNet &net, const DevBatch &b, const double *y, double *f,
                  double *jv, double *dA, double *dB, double *dC, const double *k1,
                  const double *dt, const double *geo, int flags, bool with_jac, bool chem_only, cudaStream_t s) {
    const int i = rates_tile(net, b), ntile = (b.L + (1 << i) - 1) >> i;
    const int want = b.grid_rates[i], grid = want > 0 && want < ntile ? want : (ntile > 0 ? ntile : 1);
#define GO(I)                                                                                       \
    if (i == I)                                                                                     \
        (with_jac ? k_rates<1 << I, true> : k_rates<1 << I, false>)<<<grid, I ? 256 : 128, rates_smem(net, 1 << I), s>>>( \
            net, b, y, f, jv, dA, dB, dC, k1, dt, geo, flags, chem_only);
    GO(0) GO(1) GO(2)
#undef GO
}

// Resident CTAs per SM of k_rates with tiles of 1, 2 and 4 layers (the larger of
// its two forms' register footprints sets it) for this network's shared memory.
void rates_blocks_per_sm(const DevNet &net, int occ[3]) {
#define OCC(I)                                                                                                   \
    {                                                                                                            \
        int a = 0, c = 0;                                                                                        \
        const size_t sm = rates_smem(net, 1 << I);                                                               \
        if (rates_fits(net, 1 << I)) {                                                                           \
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_rates<1 << I, true>, I ? 256 : 128, sm) != cudaSuccess) a = 0; \
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k_rates<1 << I, false>, I ? 256 : 128, sm) != cudaSuccess) c = 0; \
        }                                                                                                        \
        occ[I] = a < c ? a : c;                                                                                  \
    }
    OCC(0) OCC(1) OCC(2)
#undef OCC
}

void launch_chem_only(const DevNet &net, const DevBatch &b, const double *y, double *f,
                      const double *geo, cudaStream_t s) {
    launch_rates(net, b, y, f, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, geo, 0, false, true, s);
}

void launch_stage(const DevNet &net, const DevBatch &b, const Work &w, int flags, double mtol,
                  double atol, cudaStream_t s) {
    k_stage<<<b.ncols, 256, 0, s>>>(net, b, w.y, w.ymix, w.k1, w.k2, w.yk2, w.sol, w.ymix_out,
                                    w.delta, w.status, flags, mtol, atol);
}

}  // namespace vk
