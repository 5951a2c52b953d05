// Rate constants on the device for batches whose temperature varies by
// column (op.ReadRate.read_rate and rev_rate, op.py:63-309; the host
// restatement is network.Network.rate_constants).
//
//   forward  A T^B exp(-C/T)                       (two-body, k0-only three-body)
//            k0 / (1 + k0 M / k_inf)               (fall-off three-body)
//            the pressure-dependent OH + CH3 + M form (op.py:197-207)
//            photolysis / ionisation / condensation: the slot is left as uploaded
//            low-temperature caps (op.py:320-342), where set: at T <= T_max the
//            cap's Arrhenius or fall-off form replaces the forward rate
//   reverse  k_f / Keq,  Keq = exp(-(sum_p nu g_p - sum_r nu g_r)) (kB T / P0)^(n_r - n_p)
//            with g/RT from two-range NASA-9 polynomials switched at 1000 K
//            (chem_funs Gibbs / gibbs_sp), for pairs before '# reverse stops'.
//
// FP64 throughout (exp / pow / log of CUDA's math library).
//
// What bounds it: the FP64 unit, and there pow, exp and the divisions.  So a CTA
// takes a tile of TL layers (lane = (item, layer)) and first tabulates
// T^B and exp(-C/T) of the distinct B and C of its pairs, T-only
// factors of g/RT and (kB T / P0)^d once a layer; a pair is then a few products, one
// exponential (Keq) and a division.  Networks with more distinct exponents than
// the table holds go through it in chunks of pairs.  11 340 layers of 391 pairs: 3.2 -> 0.90 ms
// (a layer per CTA, everything per pair, before).
#include <cuda_runtime.h>
#include <math.h>

#include <string>

#include "vk_internal.cuh"

namespace vk {

constexpr int kCorr = 6;             // (kB T / P0)^d is tabulated for |d| <= kCorr

__device__ __noinline__ double arrhenius(double A, double B, double C, double T) {
    return A * pow(T, B) * exp(-C / T);
}

// The exponents of the OH + CH3 + M form, tabulated with the pairs' own
// (kRateSpecial of vk_internal.cuh, in this order: three B, four C).
template <int TL>
__device__ __forceinline__ double special_oh_ch3(double T, double M, const double *tab, const int *ix) {
    const double k = 1.932E3 * tab[ix[0] * TL] * tab[ix[3] * TL] + 5.109E-11 * tab[ix[1] * TL] * tab[ix[4] * TL];
    const double kinf = 1.031E-10 * tab[ix[2] * TL] * tab[ix[5] * TL];
    const double Fc = 0.1855 * exp(-T / 155.8) + 0.8145 * exp(-T / 1675.) + tab[ix[6] * TL];
    const double nn = 0.75 - 1.27 * log(Fc);
    const double x = log(k * M / kinf) / nn;
    const double ff = exp(log(Fc) / (1. + x * x));
    return k / (1 + k * M / kinf) * ff;
}

template <int TL>
__global__ void __launch_bounds__(256)
k_rate_consts(DevNet net, DevBatch b, RateTab rt, const int *__restrict__ kind, const int *__restrict__ rev,
              const int *__restrict__ cap_kind, const double *__restrict__ cap_T,
              const double *__restrict__ cap_params, const double *__restrict__ params,
              const double *__restrict__ nasa9, double *k) {
    extern __shared__ double sm[];
    const int li = threadIdx.x & (TL - 1), i0 = threadIdx.x / TL, di = blockDim.x / TL;
    double *gs = sm + li;                                // [ni][TL] g/RT
    double *phi = gs + net.ni * TL;                      // [10][TL] its T-only factors
    double *corr = phi + 10 * TL;                        // [2 kCorr + 1][TL] (kB T / P0)^d
    double *tab = corr + (2 * kCorr + 1) * TL;           // [rt.cap][TL] T^B, exp(-C/T) of a chunk
    const int l = blockIdx.x * TL + li;
    const bool on = l < b.L && b.lay_col[l] >= 0;        // (not a gap layer of a slot)
    const double *al = b.atm + (size_t)(on ? l : 0) * VK_ATM_NF;
    const double T = on ? al[VK_ATM_TCO] : 1.0, M = on ? al[VK_ATM_M] : 0.0;
    for (int i = i0; i < 2 * kCorr + 2; i += di) {
        if (i < 2 * kCorr + 1) {
            corr[i * TL] = pow(VK_CORR * T, (double)(i - kCorr));
        } else {
            // g/RT = h/RT - s/R, the two polynomials' terms taken together
            const double lnT = log(T), T2 = T * T;
            phi[0] = -0.5 / T2;
            phi[TL] = (lnT + 1.) / T;
            phi[2 * TL] = 1. - lnT;
            phi[3 * TL] = -T / 2.;
            phi[4 * TL] = -T2 / 6.;
            phi[5 * TL] = -T2 * T / 12.;
            phi[6 * TL] = -T2 * T2 / 20.;
            phi[8 * TL] = 1. / T;
        }
    }
    __syncthreads();
    for (int s = i0; s < net.ni; s += di) {
        const double *a = nasa9 + (size_t)s * 20 + (T < 1000. ? 0 : 10);
        double g = a[8] * phi[8 * TL] - a[9];
#pragma unroll
        for (int q = 6; q >= 0; --q) g = fma(a[q], phi[q * TL], g);
        gs[s * TL] = g;
    }
    double *kl = k + (size_t)l * net.nr;
    for (int ch = 0; ch < rt.nchunk; ++ch) {
        const int tb = rt.tab_off[2 * ch], tc = rt.tab_off[2 * ch + 1], te = rt.tab_off[2 * ch + 2];
        __syncthreads();                                 // the last chunk's table is read
        for (int i = tb + i0; i < te; i += di)
            tab[(i - tb) * TL] = i < tc ? pow(T, rt.val[i]) : exp(-rt.val[i] / T);
        __syncthreads();
        if (!on) continue;
        for (int p = rt.pair_off[ch] + i0; p < rt.pair_off[ch + 1]; p += di) {
            const double *pp = params + (size_t)p * 6;
            const int4 ix = rt.idx[p];
            double kf;
            switch (kind[p]) {
            case VK_K_ARRHENIUS: kf = pp[0] * tab[ix.x * TL] * tab[ix.y * TL]; break;
            case VK_K_FALLOFF: {
                const double k0 = pp[0] * tab[ix.x * TL] * tab[ix.y * TL];
                const double kinf = pp[3] * tab[ix.z * TL] * tab[ix.w * TL];
                kf = k0 / (1 + k0 * M / kinf);
                break;
            }
            case VK_K_SPECIAL_OH_CH3: kf = special_oh_ch3<TL>(T, M, tab, rt.special + 7 * ch); break;
            default: kf = kl[2 * p];                     // photolysis etc.: as uploaded
            }
            if (cap_kind && cap_kind[p] != VK_K_NONE && T <= cap_T[p]) {
                const double *cp = cap_params + (size_t)p * 6;
                double c = arrhenius(cp[0], cp[1], cp[2], T);
                if (cap_kind[p] == VK_K_FALLOFF) {
                    const double cinf = arrhenius(cp[3], cp[4], cp[5], T);
                    c = c / (1. + c * M / cinf);
                }
                kf = c;
            }
            double kr = 0.0;
            if (rev[p]) {
                const PairDesc *pd = net.pairs + p;
                double dg = 0.0;
                int nr_ = 0, np_ = 0;
                for (int t = 0; t < pd->nf; ++t) { dg -= pd->fnu[t] * gs[pd->fsp[t] * TL]; nr_ += pd->fnu[t]; }
                for (int t = 0; t < pd->nr; ++t) { dg += pd->rnu[t] * gs[pd->rsp[t] * TL]; np_ += pd->rnu[t]; }
                double kq = exp(-dg);
                const int d = nr_ - np_;
                if (d != 0) kq *= abs(d) <= kCorr ? corr[(d + kCorr) * TL] : pow(VK_CORR * T, (double)d);
                kr = kf / kq;
            }
            *reinterpret_cast<double2 *>(kl + 2 * p) = make_double2(kf, kr);
        }
    }
}

static size_t rate_smem(const DevNet &net, const RateTab &rt, int tl) {
    return (size_t)tl * (net.ni + 10 + 2 * kCorr + 1 + rt.cap) * sizeof(double);
}

// Tiles of four layers where every SM still gets one, else a layer each (one
// and four, 69 species: 150 layers 0.039 and 0.072 ms, 600 layers 0.084 and 0.072,
// 1200 layers 0.156 and 0.111).
void launch_rate_consts(const DevNet &net, const DevBatch &b, const RateTab &rt, const int *kind, const int *rev,
                        const int *cap_kind, const double *cap_T, const double *cap_params,
                        const double *params, const double *nasa9, double *k, cudaStream_t s) {
    if (b.L >= 4 * b.nsm)
        k_rate_consts<4><<<(b.L + 3) / 4, 256, rate_smem(net, rt, 4), s>>>(net, b, rt, kind, rev, cap_kind, cap_T,
                                                                           cap_params, params, nasa9, k);
    else
        k_rate_consts<1><<<b.L, 256, rate_smem(net, rt, 1), s>>>(net, b, rt, kind, rev, cap_kind, cap_T, cap_params,
                                                                 params, nasa9, k);
}

}  // namespace vk
