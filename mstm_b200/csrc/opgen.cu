// opgen.cu -- FP64 generation of the per-pair VSWF translation operators on the
// device, in the folded layout the translation kernel streams.
//
// A pair (i, j), i < j, gets one operator record, computed once per cluster
// (MSTM's store_translation_matrix=.true. mode, december2023/mstm-modules-33.f90:6390-6525):
//   - e^{i phi} of the pair vector r_i - r_j                (cartosphere/ephicoef, modules:1986-2004, 2075-2085)
//   - Wigner-d d^n_{km}(theta) for |k| <= min(n,nmin), folded
//     by the symmetry d_{-k,-m} = (-1)^{k+m} d_{k,m} into
//     E_n(k,m) = (d_{k,m} + (-1)^m d_{k,-m})/2  (0<=k<=kk, 0<=m<=n) and
//     O_n(k,m) = (d_{k,m} - (-1)^m d_{k,-m})/2  (1<=k<=kk, 1<=m<=n)   (rotcoef, modules:1098-1175)
//   - axial translation blocks Z_m(n,l), m = 0..nmin, both modes for m>0 and
//     one mode for m=0; the -m block equals the +m block with modes swapped
//     (axialtrancoefrecurrence, modules:1566-1676; constants axialtrancoefinit, modules:1680-1722).
//     Every element is the vector-coupling sum over the Hankel orders w that the
//     reference uses for the first row and the last column of each block,
//     Z_m(n,l) = sum_w vcc(n, l(l+1)+m, w) xi_w / z with the odd-offset terms
//     times +-i for the two modes; the reference fills the interior by a
//     three-term recurrence in n instead, the same quantity up to rounding.
//     The sums are independent.
// Three launches, each shaped for its own parallelism: the per-pair scalars and
// the Riccati-Hankel functions xi_w / z (serial in w) one thread per pair,
// into a scratch of 2 LMAX + 1 complex per pair; the Wigner-d rows (serial in
// the degree and the restricted index, parallel over the other index) one
// warp per pair; the axial blocks one CTA per AX_P pairs, a thread per (m, n, l).
// Record layout (doubles; R rotation values, oplayout.cuh):
//   [0, H)           e^{i m phi}, then e^{-i m phi}, m = 0 .. nmax (H = 4 nmax + 4)
//   [H, H+R)         E_1, O_1, E_2, O_2, ...   (row-major, restricted index first;
//                    O_n has the rows and columns of E_n, k = 0 and m = 0 zero)
//   [zb, zb+2Z)      Z_0[p=0], Z_1[p=0], Z_1[p=1], Z_2[p=0], ... complex, [row n][col l];
//                    zb is H+R rounded up to an even number
//   zeros up to zb and to a multiple of 4 doubles.
// Passes of either precision read these records.
#include "common.cuh"
#include "special.cuh"
#include "kernels.cuh"

#define DW (2 * MSTMG_LMAX + 1)
#define XIW (2 * MSTMG_LMAX + 1)   // Hankel orders w = 0 .. nt + ns <= 2 LMAX per pair

static_assert(2 * MSTMG_LMAX - 1 <= 32, "the m = 0 recurrence gives each lane one k");

struct PairGeom {
    int i, j, nt, ns, nmin, nmax;
    double r, ct;
    zd ephi;
    bool ok;
};

// cartosphere (modules:1986-2004) of r_i - r_j; ok is false for coincident centres
__device__ __forceinline__ PairGeom pair_geom(const OpGenArgs& a, int q)
{
    PairGeom g;
    g.i = a.pairs[q].x;
    g.j = a.pairs[q].y;
    g.nt = a.order[g.i];
    g.ns = a.order[g.j];
    g.nmin = g.nt < g.ns ? g.nt : g.ns;
    g.nmax = g.nt > g.ns ? g.nt : g.ns;
    const double rv0 = a.pos[3 * g.i] - a.pos[3 * g.j], rv1 = a.pos[3 * g.i + 1] - a.pos[3 * g.j + 1],
                 rv2 = a.pos[3 * g.i + 2] - a.pos[3 * g.j + 2];
    const double rr = rv0 * rv0 + rv1 * rv1 + rv2 * rv2;
    if (rr == 0.0) {
        g.r = 0.0;
        g.ct = 1.0;
        g.ephi = mk(1.0, 0.0);
    } else {
        g.r = sqrt(rr);
        g.ct = rv2 / g.r;
        if (rv0 == 0.0 && rv1 == 0.0) g.ephi = mk(1.0, 0.0);
        else {
            const double h = sqrt(rv0 * rv0 + rv1 * rv1);
            g.ephi = mk(rv0 / h, rv1 / h);
        }
    }
    g.ok = rr >= 1.0e-12;
    return g;
}

// e^{i phi} into the record and xi_w(z) / z, z = r m_medium, w = 0 .. nt + ns
// into the scratch (psi_w(z) / z for regular translations): one thread per pair
__global__ void __launch_bounds__(128) opgen_pair_kernel(OpGenArgs a)
{
    zd hs[2 * (XIW + 1)];   // spherical Bessel scratch of the complex-argument branch
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < a.npairs; q += gridDim.x * blockDim.x) {
        const PairGeom g = pair_geom(a, q);
        if (!g.ok) {
            atomicExch(a.err, MSTMG_ERR_UNSUPPORTED);
            continue;
        }
        // e^{i m phi} by the recurrence (ephicoef)
        double* h = a.op64 + a.opoff[q];
        if (op_z_base(g.nmax, g.nmin) > op_head(g.nmax) + op_rot_size(g.nmax, g.nmin)) h[op_z_base(g.nmax, g.nmin) - 1] = 0.0;
        const int units = op_record_units(g.nt, g.ns);
        for (int k = op_z_base(g.nmax, g.nmin) + 2 * op_z_offset(g.nmin + 1, g.nt, g.ns); k < units; k++) h[k] = 0.0;
        zd e = mk(1.0, 0.0);
        for (int m = 0; m <= g.nmax; m++) {
            h[2 * m] = e.x;
            h[2 * m + 1] = e.y;
            h[2 * (g.nmax + 1 + m)] = e.x;
            h[2 * (g.nmax + 1 + m) + 1] = -e.y;
            e = g.ephi * e;
        }
        zd* xi = a.xi + (size_t)q * XIW;
        const int nl = g.nt + g.ns;
        const zd z = a.pmed ? mk(g.r * a.pmed[2 * q], g.r * a.pmed[2 * q + 1]) : mk(g.r * a.rimed_re, g.r * a.rimed_im);
        if (mstm_bessel_real(nl, z, xi)) {
            if (a.regular)
                for (int k = 0; k <= nl; k++) xi[k].y = 0.0;
            continue;
        }
        if (a.regular) mstm_cricbessel(nl, z, xi, hs);
        else mstm_crichankel(nl, z, xi, hs);
        for (int k = 0; k <= nl; k++) xi[k] = cdiv(xi[k], z);
    }
}

// rotcoef(ct, nmin, nmax) (modules:1098-1175), degree by degree, folded into
// E_n, O_n: one warp per pair.  Per-warp shared scratch: D, rows k = 0..kk of
// (2 LMAX + 1) doubles (restricted index first), and the m = 0 columns dk0,
// dk01 of the degree recurrence (index -LMAX-1 .. LMAX+1).
#define ROT_WARP_DOUBLES ((MSTMG_LMAX + 1) * DW + 2 * (2 * MSTMG_LMAX + 3))
__global__ void __launch_bounds__(128) opgen_rot_kernel(OpGenArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* D = reinterpret_cast<double*>(smem_raw) + (size_t)warp * ROT_WARP_DOUBLES;
    double* dk0 = D + (MSTMG_LMAX + 1) * DW + (MSTMG_LMAX + 1);
    double* dk01 = dk0 + (2 * MSTMG_LMAX + 3);
    const int nwarps = blockDim.x >> 5;
    const double* fnr = a.fnr;
    const double* rfnr = a.rfnr;
    for (int q = blockIdx.x * nwarps + warp; q < a.npairs; q += gridDim.x * nwarps) {
        const PairGeom g = pair_geom(a, q);
        if (!g.ok) continue;
        const int nmin = g.nmin, nmax = g.nmax;
        const double ct = g.ct;
        double* rec64 = a.op64 + a.opoff[q];
        const double sbe = (fabs(ct) >= 1.0) ? 0.0 : sqrt(fabs((1.0 + ct) * (1.0 - ct)));
        const double cbe2 = 0.5 * (1.0 + ct), sbe2 = 0.5 * (1.0 - ct);
        for (int k = lane; k < 2 * MSTMG_LMAX + 3; k += 32) {
            dk0[k - (MSTMG_LMAX + 1)] = 0.0;
            dk01[k - (MSTMG_LMAX + 1)] = 0.0;
        }
        __syncwarp();
        if (lane == 0) {
            dk0[0] = 1.0;
            dk01[0] = 0.0;
        }
        __syncwarp();
        int sgn = 1;
        double sben = 1.0;
        for (int n = 1; n <= nmax; n++) {
            const int kk = n < nmin ? n : nmin;
            sgn = -sgn;
            sben = sben * sbe / 2.0;
            if (sben < 1.0e-30) sben = 0.0;
            // m = 0 column by the three-term recurrence in n (lane k + n - 1 takes
            // k = -n+1 .. n-1: at most 2 LMAX - 1 <= 31 lanes)
            {
                const int k = -n + 1 + lane;
                const bool on = k <= n - 1;
                double newv = 0.0;
                if (on)
                    newv = (ct * (double)(n + n - 1) * dk0[k] - fnr[n - k - 1] * fnr[n + k - 1] * dk01[k]) * (rfnr[n + k] * rfnr[n - k]);
                __syncwarp();
                if (on) {
                    dk01[k] = dk0[k];
                    dk0[k] = newv;
                }
            }
            if (lane == 0) {
                dk0[n] = sgn * sben * a.bcofd[n];
                dk0[-n] = sgn * dk0[n];
                dk01[n] = 0.0;
                dk01[-n] = 0.0;
            }
            __syncwarp();
            for (int k = -n + lane; k <= n; k += 32) D[k + MSTMG_LMAX] = dk0[k];
            __syncwarp();
            for (int m = 1; m <= kk; m++) {
                const double fmn = rfnr[n - m + 1] * rfnr[n + m];
                const int m1 = m - 1;
                // rows with a negative restricted index are never read (the
                // fold below takes rows 0..kk), so only row m is written
                for (int k = -n + lane; k <= n; k += 32) {
                    const double dkm1 = (k == -n) ? 0.0 : D[m1 * DW + (k - 1 + MSTMG_LMAX)];
                    const double dkn1 = (k == n) ? 0.0 : D[m1 * DW + (k + 1 + MSTMG_LMAX)];
                    const double v = (fnr[n + k] * fnr[n - k + 1] * cbe2 * dkm1 - fnr[n - k] * fnr[n + k + 1] * sbe2 * dkn1
                                      - (double)k * sbe * D[m1 * DW + (k + MSTMG_LMAX)]) * fmn;
                    D[m * DW + (k + MSTMG_LMAX)] = v;
                }
                __syncwarp();
            }
            // fold into E_n, O_n
            const int roff = op_head(nmax) + op_rot_offset(n, nmin);
            const int ne = (kk + 1) * (n + 1);
            // row and column of element e by a float reciprocal: e < 2^10 and
            // e / (n + 1) sits at least 1 / (2 (n + 1)) from the next integer
            const float rn1 = 1.0f / (float)(n + 1);
            for (int e = lane; e < ne; e += 32) {
                const int rr_ = (int)(((float)e + 0.5f) * rn1), f = e - rr_ * (n + 1);
                const double dp = D[rr_ * DW + (f + MSTMG_LMAX)], dm = pm1(f) * D[rr_ * DW + (-f + MSTMG_LMAX)];
                rec64[roff + e] = f == 0 ? 0.5 * dp : 0.5 * (dp + dm);
                rec64[roff + ne + e] = f == 0 || rr_ == 0 ? 0.0 : 0.5 * (dp - dm);
            }
            __syncwarp();
        }
    }
}

// Axial translation blocks (itype 3, outgoing; itype 1, regular, with the
// Bessel functions in the scratch) of AX_P consecutive pairs per CTA, their
// xi_w / z side by side in shared memory: thread t takes the mode-0 elements
// t, t + 128, ... of the concatenated blocks Z_0, Z_1, ..., for all the pairs
// when their orders agree, else for one after the other.  The table lies by
// term, degree m, n and l, so that the lanes (consecutive l) read it
// contiguously and every value serves AX_P pairs; one pair a CTA from a table
// by w, n fastest, took 1.62 ms for the 124,750 pairs of 500 spheres of order 9
// (their 1.3 GB of blocks take 0.2 ms to write) and 0.34 ms for 180,000 of
// order 3; now 1.04 and 0.10 ms.
#define AX_P 4
template <int NP> __device__ __forceinline__ void axial_blocks(const OpGenArgs& a, int nt, int ns, double* const* rec, const zd (*xs)[AX_P], int p0)
{
    const int nmin = nt < ns ? nt : ns, nmax = nt > ns ? nt : ns, vn = a.vnmax;
    const int zbase = op_z_base(nmax, nmin);
    const size_t ks = (size_t)(vn + 1) * vn * vn;   // one term of the sums further
    // walk the blocks forward: block m holds rc(m) elements, mode-1 copies
    // after the mode-0 ones for m > 0 (op_z_offset)
    int m = 0, e = threadIdx.x, zoff = 0;
    while (m <= nmin) {
        const int m1 = m < 1 ? 1 : m;
        const int cols = ns - m1 + 1, rc = (nt - m1 + 1) * cols;
        if (e >= rc) {
            e -= rc;
            zoff += (m == 0 ? 1 : 2) * rc;
            m++;
            continue;
        }
        const int qn = (int)(((float)e + 0.5f) * (1.0f / (float)cols));   // e / cols (e < 2^10)
        const int n = m1 + qn, l = m1 + e - qn * cols;
        const int wmin = n > l ? n - l : l - n, nw = n < l ? n : l;   // terms w = wmin, wmin + 1, ..., wmin + 2 nw
        const double* vc = a.vcc + ((size_t)m * vn + (n - 1)) * vn + (l - 1);
        const zd(*x)[AX_P] = xs + wmin;
        zd s1[NP], s2[NP];
        {
            const double v = *vc;
#pragma unroll
            for (int p = 0; p < NP; p++) {
                s1[p] = v * x[0][p0 + p];
                s2[p] = mk(0.0, 0.0);
            }
        }
#pragma unroll 2
        for (int k = 0; k < nw; k++) {
            const double v2 = vc[ks * (2 * k + 1)], v1 = vc[ks * (2 * k + 2)];
#pragma unroll
            for (int p = 0; p < NP; p++) {
                s2[p] = s2[p] + v2 * x[2 * k + 1][p0 + p];
                s1[p] = s1[p] + v1 * x[2 * k + 2][p0 + p];
            }
        }
        const int zo = zbase + 2 * (zoff + e);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            const zd t = imul(s2[p]), v0 = s1[p] + t, v1 = s1[p] - t;
            double* r = rec[p0 + p];
            *reinterpret_cast<double2*>(r + zo) = make_double2(v0.x, v0.y);   // an even offset of a record aligned to 32 bytes
            if (m > 0) *reinterpret_cast<double2*>(r + zo + 2 * rc) = make_double2(v1.x, v1.y);
        }
        e += blockDim.x;
    }
}

// grp: pairs a CTA takes, AX_P or 1
__global__ void __launch_bounds__(128) opgen_axial_kernel(OpGenArgs a, int grp)
{
    __shared__ zd xs[XIW][AX_P];
    __shared__ int nts[AX_P], nss[AX_P];   // orders; 0 for coincident centres and past the last pair
    __shared__ double* rec[AX_P];
    for (int q0 = blockIdx.x * grp; q0 < a.npairs; q0 += gridDim.x * grp) {
        __syncthreads();   // the previous pairs' reads are done
        if (threadIdx.x < AX_P) {
            const int q = q0 + threadIdx.x;
            const bool in = (int)threadIdx.x < grp && q < a.npairs;
            const PairGeom g = pair_geom(a, in ? q : q0);
            nts[threadIdx.x] = in && g.ok ? g.nt : 0;
            nss[threadIdx.x] = in && g.ok ? g.ns : 0;
            rec[threadIdx.x] = a.op64 + a.opoff[in ? q : q0];
        }
        __syncthreads();
        bool same = nts[0] > 0;
        for (int p = 1; p < AX_P; p++) same = same && nts[p] == nts[0] && nss[p] == nss[0];
        for (int t = threadIdx.x; t < AX_P * XIW; t += blockDim.x) {
            const int p = t / XIW, k = t % XIW;
            if (nts[p] > 0 && k <= nts[p] + nss[p]) xs[k][p] = a.xi[(size_t)(q0 + p) * XIW + k];
        }
        __syncthreads();
        if (same) axial_blocks<AX_P>(a, nts[0], nss[0], rec, xs, 0);
        else
            for (int p = 0; p < AX_P; p++)
                if (nts[p] > 0) axial_blocks<1>(a, nts[p], nss[p], rec, xs, p);
    }
}

size_t opgen_xi_scratch(int npairs) { return (size_t)npairs * XIW; }

void launch_opgen(const OpGenArgs& a, int nsm, cudaStream_t st)
{
    if (a.npairs <= 0) return;
    int b1 = (a.npairs + 127) / 128;
    if (b1 > nsm * 16) b1 = nsm * 16;
    opgen_pair_kernel<<<b1, 128, 0, st>>>(a);
    const int warps = 4;
    const size_t smem = sizeof(double) * ROT_WARP_DOUBLES * warps;
    allow_smem(opgen_rot_kernel, smem);
    int b2 = (a.npairs + warps - 1) / warps;
    if (b2 > nsm * 16) b2 = nsm * 16;
    opgen_rot_kernel<<<b2, warps * 32, smem, st>>>(a);
    // pairs together once they fill the chip with groups; 780 pairs of order 14
    // take 76 us in groups and 62 alone, 20,503 of order 9 193 and 290
    const int grp = a.npairs >= AX_P * 8 * nsm ? AX_P : 1;
    const int ng = (a.npairs + grp - 1) / grp, b3 = ng < nsm * 16 ? ng : nsm * 16;
    opgen_axial_kernel<<<b3, 128, 0, st>>>(a, grp);
    launch_counter() += 3;
}
