// qeffcoef.cuh -- the bilinear coefficients of lrsphereqeff
// (december2023/mstm-scatprops-26.f90:676-776) of one sphere, filled by the
// CTA that sums its efficiencies.
#pragma once
#include "special.cuh"

#define QEFF_NT 64   // threads of a sphere's CTA (two warps: the items of order 7, 63, in one go)

// per degree n: aam, ggm, agm, index (s-1) + 2(t-1)
struct QeffCoef {
    zd aam[MSTMG_LMAX][4], ggm[MSTMG_LMAX][4], agm[MSTMG_LMAX][4];
    zd psi[MSTMG_LMAX + 2], xi[MSTMG_LMAX + 2], scr[2][2 * (MSTMG_LMAX + 2)];
};

// all QEFF_NT threads; ends with a barrier
__device__ inline void qeff_coefficients(QeffCoef& c, int L, double xsp, zd ri0)
{
    const zd xri = xsp * ri0;
    // a lossless medium: j and y by real recurrences on one thread, psi = z j
    // and xi = z (j + i y); else the two complex routines, a warp each
    const bool real = xri.y == 0.0 && xri.x >= MSTM_REAL_BESSEL_MIN;
    if (real) {
        if (threadIdx.x == 0) mstm_bessel_real(L, xri, c.scr[0]);
    } else {
        if (threadIdx.x == 0) mstm_cricbessel(L, xri, c.psi, c.scr[0]);
        if (threadIdx.x == 32) mstm_crichankel(L, xri, c.xi, c.scr[1]);
    }
    __syncthreads();
    for (int n = threadIdx.x + 1; n <= L; n += QEFF_NT) {
        zd ps0, ps1, x0, x1;
        if (real) {
            x0 = xri.x * c.scr[0][n - 1];
            x1 = xri.x * c.scr[0][n];
            ps0 = mk(x0.x, 0.0);
            ps1 = mk(x1.x, 0.0);
        } else {
            ps0 = c.psi[n - 1];
            ps1 = c.psi[n];
            x0 = c.xi[n - 1];
            x1 = c.xi[n];
        }
        const zd psip = ps0 - cdiv((double)n * ps1, xri);
        const zd xip = x0 - cdiv((double)n * x1, xri);
        const zd cterm = imul(cdiv(cj(cdivr(1.0, ri0)), ri0));
        for (int s = 0; s < 2; s++)
            for (int t = 0; t < 2; t++) {
                const double sg = pm1(s + t);
                const int k = s + 2 * t;
                c.aam[n - 1][k] = cterm * (xip * cj(x1) - sg * (x1 * cj(xip)));
                c.ggm[n - 1][k] = cterm * (psip * cj(ps1) - sg * (ps1 * cj(psip)));
                c.agm[n - 1][k] = cterm * (xip * cj(ps1) - sg * (x1 * cj(psip)));
            }
    }
    __syncthreads();
}

// sums over the CTA of K doubles a thread; thread 0 has them after (red: 2 K doubles)
template <int K>
__device__ inline void qeff_reduce(double* v, double* red)
{
    for (int k = 0; k < K; k++)
        for (int w = 16; w > 0; w >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], w);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < K; k++) red[(threadIdx.x >> 5) * K + k] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < K; k++) v[k] = red[k] + red[K + k];
}

// (m, n) of slot t of a sphere's first-mode half: degree n
__device__ __forceinline__ int slot_degree(int t, int L)
{
    const int row = t % (L + 2), col = t / (L + 2) + 1;
    return row <= col ? col : row - 1;
}
