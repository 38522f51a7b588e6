// gsfrows.cuh -- the four generalised spherical functions of every degree at
// one polar angle that the averaged scattering matrices expand in: elements of
// rotcoef(ct, 2, nmax) (december2023/mstm-modules-33.f90:1098-1175).
#pragma once
#include "common.cuh"

#define GSF_NT 128
#define GSF_ROW 9     // doubles per degree: columns k = -4 .. 4 of the m = 0 row, then the values below
#define GSF_D00 0     // dc(0, n(n+1))
#define GSF_D02 1     // dc(0, n(n+1)+2)
#define GSF_D20 2     // row 2, column 0
#define GSF_D22 3     // row 2, column 2
#define GSF_D2M 4     // row 2, column -2
#define GSF_DM22 5    // row -2, column 2

// nmax reaches 400: 28.9 KB
inline int gsf_smem_bytes(int nmax) { return (int)sizeof(double) * GSF_ROW * (nmax + 1); }

// All GSF_NT threads; g: GSF_ROW (nmax + 1) doubles of shared memory, the
// values of degree n >= 1 at g + GSF_ROW n afterwards; ends with a barrier.
// Rows 2 and -2 at columns 0 and +-2 reach columns -4 .. 4 of row 0 only, so
// nine threads run the recurrence over the degrees, each its own column, and a
// thread per degree goes on from there: serial in nmax once, where a CTA-wide
// barrier per row and degree took 202 us at 181 angles for a 350-sphere
// aggregate; now 19 us.
__device__ inline void gsf_columns(int nmax, double ct, const double* fnr, const double* bcofd, double* g)
{
    const double sbe = (fabs(ct) >= 1.0) ? 0.0 : sqrt(fabs((1.0 + ct) * (1.0 - ct)));
    const double cbe2 = 0.5 * (1.0 + ct), sbe2 = 0.5 * (1.0 - ct);
    if (threadIdx.x < GSF_ROW) {
        const int k = (int)threadIdx.x - 4, ak = k < 0 ? -k : k;
        double d0 = 1.0, d01 = 0.0, sben = 1.0;
        for (int n = 1; n <= ak; n++) {
            sben = sben * sbe / 2.0;
            if (sben < 1.0e-30) sben = 0.0;
        }
        for (int n = 1; n < ak && n <= nmax; n++) g[GSF_ROW * n + threadIdx.x] = 0.0;
        if (ak > 0) {
            d0 = pm1(ak) * sben * bcofd[ak];
            if (k < 0) d0 = pm1(ak) * d0;
            if (ak <= nmax) g[GSF_ROW * ak + threadIdx.x] = d0;
        }
        for (int n = ak + 1; n <= nmax; n++) {
            const double v = (ct * (double)(n + n - 1) * d0 - fnr[n - k - 1] * fnr[n + k - 1] * d01) / (fnr[n + k] * fnr[n - k]);
            d01 = d0;
            d0 = v;
            g[GSF_ROW * n + threadIdx.x] = v;
        }
    }
    __syncthreads();
    for (int n = 1 + (int)threadIdx.x; n <= nmax; n += GSF_NT) {
        double* r = g + GSF_ROW * n;
        // row m at column k from row m - 1 at k - 1, k, k + 1
        auto step = [&](int m, int k, double dm, double d, double dp) {
            if (k < -n || k > n) return 0.0;
            const double fmn = 1.0 / fnr[n - m + 1] / fnr[n + m];
            return (fnr[n + k] * fnr[n - k + 1] * cbe2 * dm - fnr[n - k] * fnr[n + k + 1] * sbe2 * dp - (double)k * sbe * d) * fmn;
        };
        double r1[7];   // row 1, columns -3 .. 3
        for (int k = -3; k <= 3; k++) r1[k + 3] = step(1, k, r[k + 3], r[k + 4], r[k + 5]);
        const double d00 = r[4], d02 = r[6];
        double d2[3] = {0.0, 0.0, 0.0};
        if (n >= 2)
            for (int k = -2; k <= 2; k += 2) d2[(k + 2) / 2] = step(2, k, r1[k + 2], r1[k + 3], r1[k + 4]);
        r[GSF_D00] = d00;
        r[GSF_D02] = d02;
        r[GSF_D20] = d2[1];
        r[GSF_D22] = d2[2];
        r[GSF_D2M] = d2[0];
        r[GSF_DM22] = d2[0];   // dc(-m, -k) = (-1)^(k + m) dc(m, k)
    }
    __syncthreads();
}
