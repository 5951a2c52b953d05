// Transport-operator geometry: the parts of the eddy + molecular diffusion
// coefficients that do not depend on the state (op.py:1496-1597 diffdf,
// op.py:1438-1494 diffdf_no_mol, op.py:1973-2166 lhs_jac_tot / no_mol).
//
// For species i in layer j the reference's operator is
//     dy_j/dt = A y_j + B y_{j+1} + C y_{j-1}      (eddy A,B,C + molecular Ai,Bi,Ci)
// and every term has the form  g * (ysum_a + ysum_b) / (2 ysum_c) + p  with a
// state-free factor g and offset p.  Per (layer, species) we store
//     gU  factor of the upper-interface flux   (K_{j+1/2} + D_{j+1/2,i}) / (dz_ave dzi_j)
//     gD  factor of the lower-interface flux   (K_{j-1/2} + D_{j-1/2,i}) / (dz_ave dzi_{j-1})
//     pA, pB, pC  advection and thermal/gravitational molecular terms
// so that, with q = ysum ratios,
//     cA = -gU (ys_{j+1}+ys_j)/(2 ys_j) - gD (ys_j+ys_{j-1})/(2 ys_j) + pA
//     cB =  gU (ys_{j+1}+ys_j)/(2 ys_{j+1}) + pB
//     cC =  gD (ys_j+ys_{j-1})/(2 ys_{j-1}) + pC.
// The divisions then happen once per atmosphere update instead of per RHS.
#pragma once
#include <cuda_runtime.h>

#include "vk_internal.cuh"

namespace vk {

constexpr double GEO_KB = 1.38064852E-16;
constexpr double GEO_NAVO = 6.02214086E+23;
constexpr int GEO_NF = 5;           // gU, gD, pA, pB, pC

struct GeoCol {
    const double *atm;   // [layer][VK_ATM_NF]
    const double *Dzz;   // [layer][ni]
    const double *ms, *alpha;
    int l0, nz, ni;
    __device__ double a(int j, int f) const { return atm[(size_t)(l0 + j) * VK_ATM_NF + f]; }
    __device__ double dzz(int j, int i) const { return Dzz[(size_t)(l0 + j) * ni + i]; }
};

__device__ __forceinline__ GeoCol make_geocol(const double *atm, const double *Dzz,
                                              const double *spf, const int *col_off,
                                              const int *col_end, int c, int ni) {
    GeoCol g;
    g.atm = atm;
    g.Dzz = Dzz;
    g.ms = spf + (size_t)c * VK_SP_NF * ni + VK_SP_MS * ni;
    g.alpha = spf + (size_t)c * VK_SP_NF * ni + VK_SP_ALPHA * ni;
    g.l0 = col_off[c];
    g.nz = col_end[c] - g.l0;
    g.ni = ni;
    return g;
}

// The thermal and gravitational term of an interface: phi(i, g) = h + ms_i g / q
// + alpha_i / Ti dT / dz, of which only ms and alpha are the species'.
struct GeoFace { double h, q, Ti, dT, dz; };
// What a layer's coefficients have in common: eddy parts and the interfaces.
struct GeoLayer {
    double eU, eD, pA, pB, pC;      // eddy and advection
    double w, w2;                   // 1/da and 1/(2 da), at the ends 1/dzi
    double g0, gU, gD;              // gravity of the layer, above, below
    GeoFace up, dn;
};

__device__ __forceinline__ GeoFace geo_face(const GeoCol &cv, int j) {
    GeoFace f;
    f.Ti = cv.a(j, VK_ATM_TI);
    f.h = -1. / cv.a(j, VK_ATM_HPI);
    f.q = GEO_NAVO * GEO_KB * f.Ti;
    f.dT = cv.a(j + 1, VK_ATM_TCO) - cv.a(j, VK_ATM_TCO);
    f.dz = cv.a(j, VK_ATM_DZI);
    return f;
}

__device__ __forceinline__ GeoLayer geo_layer(const GeoCol &cv, int j, int flags) {
    const int nz = cv.nz;
    const bool mol = flags & VK_F_MOLDIFF;
    GeoLayer L = {};
    if (j == 0) {
        const double dzi = cv.a(0, VK_ATM_DZI), K = cv.a(0, VK_ATM_KZZ), vz = cv.a(0, VK_ATM_VZ);
        L.w = 1. / dzi;
        L.eU = L.w * (K / dzi);
        L.pA = -((vz > 0) * vz) / dzi;
        L.pB = -((vz < 0) * vz) / dzi;
        L.gU = cv.a(0, VK_ATM_G);
        if (mol) L.up = geo_face(cv, 0);
    } else if (j == nz - 1) {
        const int t = nz - 2;
        const double dzi = cv.a(t, VK_ATM_DZI), K = cv.a(t, VK_ATM_KZZ), vz = cv.a(t, VK_ATM_VZ);
        L.w = 1. / dzi;
        L.eD = L.w * (K / dzi);
        L.pA = ((vz < 0) * vz) / dzi;
        L.pC = ((vz > 0) * vz) / dzi;
        L.gD = cv.a(nz - 1, VK_ATM_G);
        if (mol) L.dn = geo_face(cv, t);
    } else {
        const double dm = cv.a(j - 1, VK_ATM_DZI), dp = cv.a(j, VK_ATM_DZI);
        const double Km = cv.a(j - 1, VK_ATM_KZZ), Kp = cv.a(j, VK_ATM_KZZ);
        const double vm = cv.a(j - 1, VK_ATM_VZ), vp = cv.a(j, VK_ATM_VZ);
        const double da = 0.5 * (dm + dp);
        const double inv = mol ? 1. / da : 2. / (dm + dp);
        L.eU = inv * (Kp / dp);
        L.eD = inv * (Km / dm);
        L.pA = -((vp > 0) * vp - (vm < 0) * vm) / da;
        L.pB = -((vp < 0) * vp) / da;
        L.pC = ((vm > 0) * vm) / da;
        if (mol) {
            L.w = 1. / da;
            L.w2 = 1. / (2. * da);
            L.g0 = cv.a(j, VK_ATM_G);
            L.gU = cv.a(j + 1, VK_ATM_G);
            L.gD = cv.a(j - 1, VK_ATM_G);
            L.up = geo_face(cv, j);
            L.dn = geo_face(cv, j - 1);
        }
    }
    return L;
}

// Geometry of species i in layer j -> out[0..4] = gU, gD, pA, pB, pC.
__device__ __forceinline__ void geo_species(const GeoCol &cv, const GeoLayer &L, int j, int i, int flags, double *out) {
    const int nz = cv.nz;
    double gU = L.eU, gD = L.eD, pA = L.pA, pB = L.pB, pC = L.pC;
    if (flags & VK_F_MOLDIFF) {
        const double ms = cv.ms[i], al = cv.alpha[i];
        auto thermal = [&](const GeoFace &f) { return al / f.Ti * f.dT / f.dz; };
        auto phi = [&](const GeoFace &f, double g, double th) { return f.h + ms * g / f.q + th; };
        if (j == 0) {
            const double D = cv.dzz(0, i), ph = phi(L.up, L.gU, thermal(L.up));
            gU += L.w * (D / L.up.dz);
            pA += L.w * D / 2. * ph;
            pB += L.w * D / 2. * ph;
        } else if (j == nz - 1) {
            const double D = cv.dzz(nz - 2, i), ph = phi(L.dn, L.gD, thermal(L.dn));
            gD += L.w * (D / L.dn.dz);
            pA += -L.w * D / 2. * ph;
            pC += -L.w * D / 2. * ph;
        } else {
            const double Dm = cv.dzz(j - 1, i), Dp = cv.dzz(j, i);
            const double tU = thermal(L.up), tD = thermal(L.dn);
            gU += L.w * (Dp / L.up.dz);
            gD += L.w * (Dm / L.dn.dz);
            pA += L.w2 * (Dp * phi(L.up, L.g0, tU) - Dm * phi(L.dn, L.g0, tD));
            pB += L.w2 * Dp * phi(L.up, L.gU, tU);
            pC += -L.w2 * Dm * phi(L.dn, L.gD, tD);
        }
    }
    out[0] = gU; out[1] = gD; out[2] = pA; out[3] = pB; out[4] = pC;
}
__device__ __forceinline__ void geo_coef(const GeoCol &cv, int j, int i, int flags, double *out) {
    geo_species(cv, geo_layer(cv, j, flags), j, i, flags, out);
}

}  // namespace vk
