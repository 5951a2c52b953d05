// Photochemistry radiative transfer on the device: optical depth, two-stream
// actinic flux and photolysis rates for every column of a batch.
//
// Restates op.ODESolver.compute_tau (op.py:2580-2599), compute_flux
// (op.py:2603-2739, isotropic scattering, ag0 = 0 in phy_const.py) and
// compute_J (op.py:2751-2786) on the binned cross sections the host set-up
// provides (make_bins_read_cross, read_sflux).  The T-dependent branches of
// compute_tau (op.py:2591-2592) and compute_J (op.py:2770-2774) read
// per-layer tables where vk_photo_set_cross_T gave them.
//
// Measured, 128 columns x 150 layers x 446 bins x 48 channels on a GB300: one
// thread per (column, bin) for the fluxes, everything recomputed in each sweep,
// and a block reduction per channel 10.5 + 3.7 ms; now 1.03 + 0.03 + 1.75 + 0.24 +
// 0.87 ms (one column: 0.30 ms).
// The FP64 unit bounds all of it (19 cycles per warp-wide instruction and SM),
// so every quantity of a (layer, bin) is computed once, and what a column's
// layers depend on in sequence is kept to one add or two FMAs a layer:
//   k_photo_opt    (layers x bins) optical depth of each layer and the
//                  single-scattering albedo, a thread per bin and eight layers:
//                  one read of a cross section serves all eight;
//   k_photo_scan   (columns x bins) tau from the top;
//   k_photo_coef   (layers x bins) the two-stream coefficients divided by chi,
//                  and the layer's mean direct flux (one exp per interface);
//   k_photo_sweep  (columns x bins) the downward then the upward sweep of the
//                  diffuse fluxes (the downward sweep reads the previous call's
//                  upward flux, as the reference's arrays persist) and the
//                  actinic flux.  Staggered arrays (nz+1 interfaces) of column
//                  c start at row col_off[c] + c;
//   k_photo_J      J of every channel = sum over bins of actinic flux x
//                  (cross_J x bin weight), a thread per (layer, three channels)
//                  with both factors staged in shared memory, written times
//                  f_diurnal into the channel's k slot; the column's largest
//                  relative actinic-flux change (aflux_change) by atomicMax on
//                  the bit pattern (non-negative doubles order like integers).
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>

#include "vk_internal.cuh"

namespace vk {

constexpr double kHC = 1.98644582E-9;        // erg nm (phy_const.py)

constexpr int kPT = 128;                     // threads (bins) of the per-layer kernels
constexpr int kPL = 8;                       // layers a thread of k_photo_opt / _coef takes
constexpr int kMaxTerms = 192;               // absorbers + scatterers staged at once

// a / c with rc = 1 / c: the quotient's rounding error is corrected by one
// residual, so it is as good as the division
__device__ __forceinline__ double div_const(double a, double c, double rc) {
    const double q = a * rc;
    return isfinite(q) ? __fma_rn(__fma_rn(-q, c, a), rc, q) : q;
}

__global__ void __launch_bounds__(kPT)
k_photo_opt(DevNet net, DevBatch b, PhotoDev ph, const double *__restrict__ y,
            const double *__restrict__ ymix) {
    __shared__ double2 yy[kMaxTerms][kPL];   // (y dz, ymix) of each term and layer
    __shared__ int lcol[kPL], s_any;
    const int ni = net.ni, NB = ph.nbins, tid = threadIdx.x;
    const int n = blockIdx.y * kPT + tid, lt = blockIdx.x * kPL;
    if (tid == 0) s_any = 0;
    __syncthreads();
    if (tid < kPL) {
        const int l = lt + tid;
        int c = l < b.L ? b.lay_col[l] : -1;
        if (c >= 0 && b.active && !b.active[c]) c = -1;
        lcol[tid] = c;
        if (c >= 0) s_any = 1;
    }
    __syncthreads();
    if (!s_any) return;
    double t[kPL], tabs[kPL], tsc[kPL];
#pragma unroll
    for (int u = 0; u < kPL; ++u) t[u] = tabs[u] = tsc[u] = 0.0;
    const int nt = ph.nabs + ph.nscat;
    for (int a0 = 0; a0 < nt; a0 += kMaxTerms) {
        const int na = nt - a0 < kMaxTerms ? nt - a0 : kMaxTerms;
        __syncthreads();
        for (int e = tid; e < na * kPL; e += kPT) {
            const int a = e / kPL, u = e - a * kPL, ai = a0 + a;
            double2 v = make_double2(0.0, 0.0);
            if (lcol[u] >= 0) {
                const size_t l = (size_t)lt + u;
                const int s = ai < ph.nabs ? ph.abs_sp[ai] : ph.scat_sp[ai - ph.nabs];
                v.x = y[l * ni + s] * b.atm[l * VK_ATM_NF + VK_ATM_DZ];
                v.y = ymix[l * ni + s];
            }
            yy[a][u] = v;
        }
        __syncthreads();
        if (n >= NB) continue;
        for (int a = 0; a < na; ++a) {
            const int ai = a0 + a;
            if (ai < ph.nabs) {
                const double cr = ph.cross[(size_t)ai * NB + n];
                const int ts = ph.abs_tslot ? ph.abs_tslot[ai] : -1;
                if (ts < 0) {
#pragma unroll
                    for (int u = 0; u < kPL; ++u) t[u] += yy[a][u].x * cr;
                } else {
#pragma unroll
                    for (int u = 0; u < kPL; ++u)
                        if (lcol[u] >= 0) t[u] += yy[a][u].x * ph.cross_T[((size_t)ts * ph.lstride + lt + u) * NB + n];
                }
                if (ph.abs_photo[ai]) {
#pragma unroll
                    for (int u = 0; u < kPL; ++u) tabs[u] += yy[a][u].y * cr;
                }
            } else {
                const double cr = ph.cross_scat[(size_t)(ai - ph.nabs) * NB + n];
#pragma unroll
                for (int u = 0; u < kPL; ++u) {
                    t[u] += yy[a][u].x * cr;
                    tsc[u] += yy[a][u].y * cr;
                }
            }
        }
    }
    if (n >= NB) return;
#pragma unroll
    for (int u = 0; u < kPL; ++u) {
        if (lcol[u] < 0) continue;
        const size_t l = (size_t)lt + u;
        ph.tau[(l + lcol[u]) * NB + n] = t[u];           // the layer's own; summed by k_photo_scan
        // numpy's nan_to_num, then the cap below 1 (pure scatterers)
        double w0 = tsc[u] / (tabs[u] + tsc[u]);
        if (isnan(w0)) w0 = 0.0;
        else if (isinf(w0)) w0 = w0 > 0 ? DBL_MAX : -DBL_MAX;
        ph.w0[l * NB + n] = fmin(w0, 1. - 1.E-8);
    }
}

// tau of a column's interfaces: the layers' optical depths added from the top
__global__ void __launch_bounds__(64) k_photo_scan(DevBatch b, PhotoDev ph) {
    const int c = blockIdx.y, n = blockIdx.x * 64 + threadIdx.x, NB = ph.nbins;
    if (n >= NB || (b.active && !b.active[c])) return;
    const int l0 = b.col_off[c], nz = b.col_end[c] - l0;
    double *tau = ph.tau + (size_t)(l0 + c) * NB + n;
    tau[(size_t)nz * NB] = 0.0;
    double s = 0.0;
    constexpr int U = 10;                    // loads in flight
    for (int j = nz - 1; j >= 0; j -= U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = j - u >= 0 ? tau[(size_t)(j - u) * NB] : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j - u < 0) break;
            s += v[u];
            tau[(size_t)(j - u) * NB] = s;
        }
    }
}

// Two-stream coefficients of every (layer, bin), over chi: with
//   Dd_j = (phi Dd_{j+1} - xi Du_j + id/mu) / chi,  Du_{j+1} = (phi Du_j - xi Dd_{j+1} + iu/mu) / chi
// w0 becomes phi/chi, cX xi/chi, cD id/(mu chi), cU iu/(mu chi), and aflux_prev the mean direct flux
// (k_photo_sweep turns it into the previous actinic flux).
__global__ void __launch_bounds__(kPT)
k_photo_coef(DevBatch b, PhotoDev ph) {
    const int NB = ph.nbins, n = blockIdx.y * kPT + threadIdx.x, lt = blockIdx.x * kPL;
    if (n >= NB) return;
    const double cosz = cos(ph.sl_angle), rcosz = 1. / cosz, mu = -cosz, rmu = 1. / mu;
    const double redd = 1. / ph.edd, imu2 = 1. / (mu * mu), iedd2 = 1. / (ph.edd * ph.edd);
    const double hp = 0.5 * (redd + rmu), hm = 0.5 * (redd - rmu);
    const double ftop = ph.sflux_top[n];
    double t_hi = 0.0, s_hi = 0.0;           // tau and direct flux of the interface below
    int have = -1;                           // the layer they belong to as its lower interface
    for (int u = 0; u < kPL; ++u) {
        const int l = lt + u;
        const int c = l < b.L ? b.lay_col[l] : -1;
        if (c < 0 || (b.active && !b.active[c])) continue;
        const double *tau = ph.tau + (size_t)(l + c) * NB + n;
        double tj, slo;
        if (have == l && l != b.col_off[c]) {
            tj = t_hi;
            slo = s_hi;
        } else {
            tj = tau[0];
            slo = ftop * exp(-div_const(tj, cosz, rcosz));
        }
        const double tj1 = tau[NB], shi = ftop * exp(-div_const(tj1, cosz, rcosz));
        t_hi = tj1;
        s_hi = shi;
        have = l + 1;
        const size_t o = (size_t)l * NB + n;
        const double w0 = ph.w0[o];
        const double sq = sqrt(1. - w0);
        const double tran = exp(-1. * redd * sq * (tj - tj1));
        const double zp = 0.5 * (1. + sq), zm = 0.5 * (1. - sq);
        const double ll = -w0 / (imu2 - iedd2 * (1. - w0));
        const double gp = ll * hp, gm = ll * hm;
        const double tr2 = tran * tran;
        const double chi = zm * zm * tr2 - zp * zp;
        const double xi = zp * zm * (1. - tr2);
        const double phi = (zm * zm - zp * zp) * tran;
        const double dlo = slo * cosz, dhi = shi * cosz;            // direct flux, lower / upper interface
        const double iu = phi * gp * dlo - (xi * gm + chi * gp) * dhi;
        const double id = phi * gm * dhi - (chi * gm + xi * gp) * dlo;
        const double rc = 1. / chi, rcm = rc * rmu;
        ph.w0[o] = phi * rc;
        ph.cX[o] = xi * rc;
        ph.cD[o] = id * rcm;
        ph.cU[o] = iu * rcm;
        ph.aflux_prev[o] = 0.5 * (slo + shi);
    }
}

__global__ void __launch_bounds__(64) k_photo_sweep(DevBatch b, PhotoDev ph) {
    const int c = blockIdx.y, n = blockIdx.x * 64 + threadIdx.x, NB = ph.nbins;
    if (n >= NB || (b.active && !b.active[c])) return;
    const int l0 = b.col_off[c], nz = b.col_end[c] - l0;
    const size_t lo = (size_t)l0 * NB + n, so = (size_t)(l0 + c) * NB + n;
    const double *cA = ph.w0 + lo, *cX = ph.cX + lo, *cD = ph.cD + lo, *cU = ph.cU + lo;
    double *Du = ph.dflux_u + so, *Dd = ph.dflux_d + so;
    constexpr int U = 6;                     // layers whose loads are in flight
    double d = Dd[(size_t)nz * NB];
    for (int j = nz - 1; j >= 0; j -= U) {
        double va[U], vx[U], vc[U], vu[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t o = (size_t)(j - u >= 0 ? j - u : 0) * NB;
            va[u] = cA[o]; vx[u] = cX[o]; vc[u] = cD[o]; vu[u] = Du[o];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j - u < 0) break;
            d = va[u] * d - vx[u] * vu[u] + vc[u];
            Dd[(size_t)(j - u) * NB] = d;
        }
    }
    const double e = kHC / ph.bins[n], re = 1. / e, hedd = 0.5 / ph.edd;
    double *af = ph.aflux + lo, *ap = ph.aflux_prev + lo;
    double uu = Du[0], dlow = d;
    for (int j = 0; j < nz; j += U) {
        double va[U], vx[U], vc[U], vd[U], vm[U], vf[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const size_t o = (size_t)(j + u < nz ? j + u : nz - 1) * NB;
            va[u] = cA[o]; vx[u] = cX[o]; vc[u] = cU[o]; vd[u] = Dd[o + NB]; vm[u] = ap[o]; vf[u] = af[o];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (j + u >= nz) break;
            const size_t o = (size_t)(j + u) * NB;
            const double un = va[u] * uu - vx[u] * vd[u] + vc[u];
            Du[o + NB] = un;
            const double tot = vm[u] + (uu + un + vd[u] + dlow) * hedd;
            ap[o] = vf[u];
            af[o] = div_const(tot, e, re);
            uu = un;
            dlow = vd[u];
        }
    }
}

// TL layers per CTA; a thread takes one layer and every (256 / TL)-th channel,
// kJC at a time, over bins staged kJB at a time.
constexpr int kJB = 32, kJT = 256;
template <int TL, int kJC>
__global__ void __launch_bounds__(kJT)
k_photo_J(DevNet net, DevBatch b, PhotoDev ph, double *k, unsigned long long *change) {
    constexpr int G = kJT / TL;              // threads per layer = channels per pass / kJC
    __shared__ double sa[TL][kJB + 1];
    __shared__ double sw[G * kJC][kJB + 1];
    __shared__ int lcol[TL], s_any;
    const int lt = blockIdx.x * TL, tid = threadIdx.x, NB = ph.nbins;
    const int tl = tid % TL, g = tid / TL, lane = tid & 31;
    if (tid == 0) s_any = 0;
    __syncthreads();
    if (tid < TL) {
        const int l = lt + tid;
        int c = l < b.L ? b.lay_col[l] : -1;
        if (c >= 0 && b.active && !b.active[c]) c = -1;
        lcol[tid] = c;
        if (c >= 0) s_any = 1;
    }
    __syncthreads();
    if (!s_any) return;
    const size_t l = (size_t)lt + tl;
    const int c = lcol[tl];
    for (int ch0 = 0; ch0 < ph.nch; ch0 += G * kJC) {
        double acc[kJC];
        const double *wT[kJC];               // this layer's own table of a T-dependent channel
#pragma unroll
        for (int x = 0; x < kJC; ++x) {
            const int ch = ch0 + g + x * G;
            acc[x] = 0.0;
            const int ts = ph.ch_tslot && ch < ph.nch && c >= 0 ? ph.ch_tslot[ch] : -1;
            wT[x] = ts < 0 ? nullptr : ph.wcross_J_T + ((size_t)ts * ph.lstride + l) * NB;
        }
        for (int n0 = 0; n0 < NB; n0 += kJB) {
            const int nn = NB - n0 < kJB ? NB - n0 : kJB;
            __syncthreads();
            for (int e = tid; e < TL * kJB; e += kJT) {
                const int r = e / kJB, n = e - r * kJB;
                sa[r][n] = lcol[r] >= 0 && n < nn ? ph.aflux[((size_t)lt + r) * NB + n0 + n] : 0.0;
            }
            for (int e = tid; e < G * kJC * kJB; e += kJT) {
                const int r = e / kJB, n = e - r * kJB;
                sw[r][n] = ch0 + r < ph.nch && n < nn ? ph.wcross_J[(size_t)(ch0 + r) * NB + n0 + n] : 0.0;
            }
            __syncthreads();
            for (int n = 0; n < nn; ++n) {
                const double a = sa[tl][n];
#pragma unroll
                for (int x = 0; x < kJC; ++x)
                    acc[x] += a * (wT[x] ? wT[x][n0 + n] : sw[g + x * G][n]);
            }
        }
#pragma unroll
        for (int x = 0; x < kJC; ++x) {
            const int ch = ch0 + g + x * G;
            if (c >= 0 && ch < ph.nch) {
                ph.J[l * ph.nch + ch] = acc[x];
                const int ki = ph.ch_kindex[ch];
                if (ki > 0) k[l * net.nr + ki - 1] = acc[x] * ph.f_diurnal;
            }
        }
    }
    // relative change of the actinic flux where it exceeds flux_atol
    for (int r = tid >> 5; r < TL; r += kJT / 32) {
        if (lcol[r] < 0) continue;
        const double *af = ph.aflux + ((size_t)lt + r) * NB, *ap = ph.aflux_prev + ((size_t)lt + r) * NB;
        double m = 0.0;
        for (int n = lane; n < NB; n += 32)
            if (af[n] > ph.flux_atol) m = fmax(m, fabs(af[n] - ap[n]) / af[n]);
        for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0 && m > 0.0) atomicMax(change + lcol[r], (unsigned long long)__double_as_longlong(m));
    }
}

// zero the change of the columns this update covers
__global__ void k_photo_clear(DevBatch b, unsigned long long *change) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < b.ncols && (!b.active || b.active[c])) change[c] = 0ull;
}

void launch_photo_clear(const DevBatch &b, unsigned long long *change, cudaStream_t s) {
    k_photo_clear<<<(b.ncols + 127) / 128, 128, 0, s>>>(b, change);
}

void launch_photo(const DevNet &net, const DevBatch &b, const PhotoDev &ph, const double *y,
                  const double *ymix, double *k, unsigned long long *change, cudaStream_t s) {
    const dim3 gl((b.L + kPL - 1) / kPL, (ph.nbins + kPT - 1) / kPT), gc((ph.nbins + 63) / 64, b.ncols);
    k_photo_opt<<<gl, kPT, 0, s>>>(net, b, ph, y, ymix);
    k_photo_scan<<<gc, 64, 0, s>>>(b, ph);
    k_photo_coef<<<gl, kPT, 0, s>>>(b, ph);
    k_photo_sweep<<<gc, 64, 0, s>>>(b, ph);
    // sixteen layers share each staged weight (0.87 ms at 19 200 layers); four where
    // that would leave SMs idle (0.07 ms at 150 layers, where it is 10 CTAs)
    if (b.L >= 16 * b.nsm) k_photo_J<16, 3><<<(b.L + 15) / 16, kJT, 0, s>>>(net, b, ph, k, change);
    else k_photo_J<4, 1><<<(b.L + 3) / 4, kJT, 0, s>>>(net, b, ph, k, change);
}

}  // namespace vk
