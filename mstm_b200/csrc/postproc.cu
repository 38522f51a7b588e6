// postproc.cu -- FP64 device post-processing of a solved cluster:
//   * translation orders of each sphere to the cluster origin
//     (tranordertest, december2023/mstm-modules-33.f90:1896-1942);
//   * merge to the common origin: regular (J) translation of every sphere's
//     expansion to the origin, converted from the LR to the TE/TM basis and
//     summed (merge_to_common_origin, mstm-scatprops-26.f90:447-559), and the
//     reverse translation of an origin expansion to every sphere
//     (distribute_from_common_origin, mstm-scatprops-26.f90:561-669);
//   * GSF expansion of the azimuth-averaged scattering matrix
//     (fosmexpansion, mstm-scatprops-26.f90:1820-1951);
//   * its evaluation at polar angles (fosmcalc, mstm-scatprops-26.f90:1750-1810);
//   * the scattering matrix at single directions without azimuthal averaging
//     (scatteringmatrix, mstm-scatprops-26.f90:1498-1573).
// Orders reach t_matrix_order (up to 100), so the per-sphere translation keeps
// its Wigner-d rows, Bessel values and axial blocks in global scratch.
#include "common.cuh"
#include "special.cuh"
#include "postproc.cuh"
#include "vcoupling.cuh"
#include "gsfrows.cuh"
#include <algorithm>

#define PP_NT 256

// vector-coupling coefficients: vc_func / vc_uprec of vcoupling.cuh

__device__ __forceinline__ zd ipow_z(int k)
{
    int e = ((k % 4) + 4) % 4;
    return (e == 0) ? mk(1.0, 0.0) : (e == 1 ? mk(0.0, 1.0) : (e == 2 ? mk(-1.0, 0.0) : mk(0.0, -1.0)));
}

// ---------------------------------------------------------------------------
// tranordertest per sphere: a warp per sphere, its lanes evaluating the
// terms of 32 consecutive orders n at a time; one lane adds them in order of
// n, exactly as the reference's loop does, and stops at the first order whose
// partial sum meets the criterion.
// ---------------------------------------------------------------------------
// One Bessel evaluation serves all 32 orders, and each lane's coupling row lies
// in shared memory; with an evaluation per order and rows in global scratch
// the kernel took 1224 us for 350 spheres; now 47 us.  Arguments the real
// recurrence leaves to the complex routine have an evaluation per order: each
// lane in the rest of its coupling row for the first 32 orders, where such
// arguments meet the criterion, else the lanes in turn with one pair of arrays.
#define TRANORDER_NLIM 200
#define TRANORDER_ROW (TRANORDER_NLIM + 31 + MSTMG_LMAX + 2)
__global__ void __launch_bounds__(32) tranorder_kernel(int nsph, const double* pos, const int* order, double ox, double oy, double oz,
                                                       double rire, double eps, int maxt, VCTab tab, int* tord)
{
    extern __shared__ __align__(16) unsigned char tr_smem[];
    zd* xs = reinterpret_cast<zd*>(tr_smem);                  // j_l(z) i^l
    zd* work = xs + TRANORDER_ROW;                            // of the complex routine
    double* vc1 = reinterpret_cast<double*>(work + TRANORDER_ROW) + threadIdx.x * TRANORDER_ROW;
    __shared__ double terms[32];
    const int lane = threadIdx.x;
    for (int i = blockIdx.x; i < nsph; i += gridDim.x) {
        const int lmax = order[i];
        const double dx = pos[3 * i] - ox, dy = pos[3 * i + 1] - oy, dz = pos[3 * i + 2] - oz;
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        int nmax = lmax;
        if (r != 0.0) {
            const zd z = mk(r * rire, 0.0);
            double sum = 0.0;
            int found = 0;
            for (int n0 = 1; n0 <= TRANORDER_NLIM && !found; n0 += 32) {
                const int n = n0 + lane;
                int shared_xi = 0;
                __syncwarp();
                if (lane == 0) shared_xi = mstm_bessel_real(min(n0 + 31, TRANORDER_NLIM) + lmax, z, xs);
                shared_xi = __shfl_sync(0xffffffffu, shared_xi, 0);
                __syncwarp();
                if (shared_xi)
                    for (int l = lane; l <= min(n0 + 31, TRANORDER_NLIM) + lmax; l += 32) xs[l] = mk(xs[l].x, 0.0) * ipow_z(l);
                __syncwarp();
                double term = 0.0;
                if (n <= TRANORDER_NLIM) vc_func(tab, -1, n, 1, lmax, vc1);
                auto sum_terms = [&](const zd* xi) {
                    const int l = lmax;
                    const zd c = (tab.fr(n + n + 1) * tab.fr(l + l + 1)) * ipow_z(n - l);
                    const int wmin = abs(n - l), wmax = n + l;
                    zd a = mk(0.0, 0.0), b = mk(0.0, 0.0);
                    for (int w = wmin; w <= wmax; w++) {
                        const double alnw = vc1[w] * vc1[w];
                        if ((n + l + w) % 2 == 0) a = a + alnw * xi[w];
                        else b = b + alnw * xi[w];
                    }
                    a = c * a;
                    b = c * b;
                    return (a * cj(a) + b * cj(b)).x;
                };
                auto own_terms = [&](zd* xi, zd* scr) {
                    mstm_cricbessel(n + lmax, z, xi, scr);
                    for (int l = 0; l <= n + lmax; l++) xi[l] = cdiv(xi[l], z) * ipow_z(l);
                    return sum_terms(xi);
                };
                constexpr int first = 32 + MSTMG_LMAX + 1;   // values of an order up to 32
                static_assert(first + 1 + 2 * 2 * first <= TRANORDER_ROW, "a coupling row and two arrays of the first orders");
                if (shared_xi) {
                    if (n <= TRANORDER_NLIM) term = sum_terms(xs);
                } else if (n0 == 1) {
                    zd* xi = reinterpret_cast<zd*>(vc1 + first + 1);
                    term = own_terms(xi, xi + first);
                } else {
                    for (int q = 0; q < 32; q++) {
                        if (lane == q && n <= TRANORDER_NLIM) term = own_terms(xs, work);
                        __syncwarp();
                    }
                }
                terms[lane] = term;
                __syncwarp();
                if (lane == 0)
                    for (int k = 0; k < 32 && n0 + k <= TRANORDER_NLIM; k++) {
                        sum = sum + terms[k];
                        if (fabs(1.0 - sum) < eps) {
                            found = n0 + k;
                            break;
                        }
                    }
                found = __shfl_sync(0xffffffffu, found, 0);
                __syncwarp();
            }
            nmax = found ? found : TRANORDER_NLIM;
            nmax = max(nmax, lmax);
        }
        if (lane == 0) tord[i] = min(nmax, maxt);
    }
}

// ---------------------------------------------------------------------------
// coupling constants of a regular translation (axialtrancoefinit,
// modules:1680-1722): one CTA per (n, l), a thread per degree m and one for
// the m-independent row, rows in shared memory (min(n, l) <= MSTMG_LMAX: one
// side is a sphere).  The host took 2 ms for the tables of a 350-sphere
// scattering matrix before the first kernel that reads them could start.
// ---------------------------------------------------------------------------
#define RC_NT 64
static_assert(RC_NT >= 2 * MSTMG_LMAX + 2, "a thread per degree m and one more");
__global__ void __launch_bounds__(RC_NT) regular_couplings_kernel(int Tt, int Ls, VCTab tab, double* vcc)
{
    extern __shared__ __align__(16) double rc_smem[];
    const int n = Tt - (int)blockIdx.x, l = Ls - (int)blockIdx.y, VL = Tt + Ls + 1;
    const int nlmin = min(n, l), wmin = abs(n - l), wmax = n + l, nm = 2 * nlmin + 1;
    const int r = threadIdx.x;
    // every axial element is a sum of these, where the reference has most of
    // them by a recurrence: 0.5 keeps their errors below those it had
    if (r < nm) vc_func(tab, nlmin - r, n, r - nlmin, l, rc_smem + r * VL, 0.5);   // vcfunc(-m,n,m,l), m = r - nlmin
    else if (r == nm) vc_func(tab, -1, n, 1, l, rc_smem + nm * VL, 0.5);
    __syncthreads();
    const double c1 = tab.fr(n + n + 1) * tab.fr(l + l + 1);
    const double* v2 = rc_smem + nm * VL;
    const int nw = wmax - wmin + 1;
    for (int e = threadIdx.x; e < nm * nw; e += RC_NT) {
        const int q = e / nw, w = wmin + e % nw, m = q - nlmin, ml = l * (l + 1) + m;
        const int ph = ((n - l + w) % 4 + 4) % 4;
        const double ri = (ph == 0 || ph == 1) ? 1.0 : -1.0;
        vcc[(size_t)(n - 1) + (size_t)Tt * ((size_t)(ml - 1) + (size_t)Ls * (Ls + 2) * w)] = -c1 * pm1(m) * rc_smem[q * VL + w] * v2[w] * ri;
    }
}

// ---------------------------------------------------------------------------
// merge to / distribute from the common origin: CTAs over (sphere, chunk of
// MERGE_PC columns), spheres grid-strided, scratch per CTA.  Per sphere the
// translation's tables are made once -- e^{i m phi} powers, the regular
// radial functions, the Wigner-d rows (rotcoef recurrence) and the axial
// blocks of every degree m -- and then applied to the chunk's columns
// together: forward rotation, axial translation, back rotation, each phase
// one barrier for all the columns.
// The tables are latency bound, so each is split where it has no recurrence:
// a thread owns a column of the m = 0 rows through every degree, a warp owns a
// degree of the other rows (its two last rows in shared memory, no barrier),
// and every axial element is its own vector-coupling sum (the reference's
// three-term recurrence over n gives the same numbers).  With CTA-wide
// barriers at every step of every recurrence, through global scratch, a launch
// took 318 us for the columns of one order of a T matrix of 60 spheres and
// 1330 us for 350 spheres of order 9 merged to one origin expansion; now 124
// and 287 us.
// Source expansions whose only nonzero degrees are lsrc and up (the unit
// fields of one order that a T matrix distributes) skip the degrees below.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(PP_NT) merge_kernel(MergeArgs a)
{
    extern __shared__ __align__(16) unsigned char mg_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = a.T;
    zd* base = a.scratch + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * a.scratch_stride;
    const bool dist = (a.mode == 1);
    const int p0 = blockIdx.y * MERGE_PC, np = min(MERGE_PC, a.npol - p0);
    if (np <= 0) return;
    for (int i = blockIdx.x; i < a.nsph; i += gridDim.x) {
        if (a.active && !a.active[i]) continue;   // uniform over the CTA
        const int Li = a.order[i];
        const int L = dist ? T : Li;                       // source order
        const int nt = dist ? Li : min(T, a.tord[i]);      // target order
        const int nmin = min(L, nt), nmax = max(L, nt);
        const int l0 = max(1, a.lsrc);                     // first source degree
        const int W = 2 * nmin + 1;
        const double sv = dist ? -1.0 : 1.0;               // translation vector: target - source
        const double rv0 = sv * (a.r0[0] - a.pos[3 * i]), rv1 = sv * (a.r0[1] - a.pos[3 * i + 1]), rv2 = sv * (a.r0[2] - a.pos[3 * i + 2]);
        const size_t soff = dist ? 0 : (size_t)a.offset[i];
        const double rr = rv0 * rv0 + rv1 * rv1 + rv2 * rv2;
        // scratch layout
        zd* xi = base;                                        // nt+L+2
        zd* hs = xi + (nmax + L + 4);                         // Bessel scratch 2*(nt+L+2)
        zd* eph = hs + 2 * (nmax + L + 4);                    // e^{i m phi}, m = -nmax..nmax
        double* D = (double*)(eph + (2 * nmax + 1));          // Wigner rows: per degree n, W x (2n+1) at W n n, restricted index first
        zd* Zall = (zd*)(D + ((size_t)W * (nmax + 1) * (nmax + 1) + 1) / 2 * 2);   // axial blocks, per degree ma: 2 x nt x L
        zd* AP = Zall + (size_t)(nmin + 1) * 2 * nt * L;      // a'(k, l, q) per column: np x 2 x L x W
        zd* G = AP + (size_t)np * 2 * L * W;                  // g(m, n, q) per column: np x 2 x nt x W
        zd* XP = G + (size_t)np * 2 * nt * W;                 // x(m, l, q) e^{i m phi} per column: np x 2 x L (L + 2)
        const zd* src = a.amnp;
        __syncthreads();
        if (rr < 1.0e-12) {
            // zero translation of regular functions: copy the overlapping orders (mtransfer)
            int nc = min(L, nt);
            for (int e = tid; e < np * nc * (nc + 2); e += PP_NT) {
                const int pc = e / (nc * (nc + 2)), ee = e - pc * (nc * (nc + 2));
                const int p = p0 + pc;
                int n = 1;
                while (n * (n + 2) <= ee) n++;
                int m = ee - (n * n - 1) - n;   // ee = n(n+1)-1+m ... -> m in -n..n
                zd v1 = src[(size_t)p * a.ld + soff + aidx(m, n, 0, L)];
                zd v2 = src[(size_t)p * a.ld + soff + aidx(m, n, 1, L)];
                if (dist) {
                    zd* o = a.out + (size_t)p * a.ldo + a.offset[i];
                    o[aidx(m, n, 0, nt)] = v1;
                    o[aidx(m, n, 1, nt)] = v2;
                    continue;
                }
                int s_ = aidx(m, n, 0, T);
                atomicAdd(&a.amnp0[(size_t)p * a.ld0 + s_].x, v1.x + v2.x);
                atomicAdd(&a.amnp0[(size_t)p * a.ld0 + s_].y, v1.y + v2.y);
                atomicAdd(&a.amnp0[(size_t)p * a.ld0 + s_ + T * (T + 2)].x, v1.x - v2.x);
                atomicAdd(&a.amnp0[(size_t)p * a.ld0 + s_ + T * (T + 2)].y, v1.y - v2.y);
            }
            __syncthreads();
            continue;
        }
        const double r = sqrt(rr);
        const double ct = rv2 / r;
        const zd ephi = (rv0 == 0.0 && rv1 == 0.0) ? mk(1.0, 0.0) : mk(rv0 / sqrt(rv0 * rv0 + rv1 * rv1), rv1 / sqrt(rv0 * rv0 + rv1 * rv1));
        // Bessel functions psi_n(r)/r (cricbessel), n = 0..nt+L; e^{i m phi}
        if (tid == PP_NT - 1) {
            const zd z = mk(r * a.rimed_re, r * a.rimed_im);
            if (mstm_bessel_real(nt + L, z, xi))
                for (int k = 0; k <= nt + L; k++) xi[k].y = 0.0;
            else {
                mstm_cricbessel(nt + L, z, xi, hs);
                for (int k = 0; k <= nt + L; k++) xi[k] = cdiv(xi[k], z);
            }
        }
        if (tid == PP_NT - 33) {
            zd* e = eph + nmax;
            zd em = mk(1.0, 0.0);
            e[0] = em;
            for (int m = 1; m <= nmax; m++) {
                em = ephi * em;
                e[m] = em;
                e[-m] = cj(em);
            }
        }
        // Wigner-d rows by the rotcoef recurrence (kmax = nmin, nmax), of the
        // degrees the rotations use
        auto used = [&](int n) { return n <= nt || (n >= l0 && n <= L); };
        const double sbe = (fabs(ct) >= 1.0) ? 0.0 : sqrt(fabs((1.0 + ct) * (1.0 - ct)));
        const double cbe2 = 0.5 * (1.0 + ct), sbe2 = 0.5 * (1.0 - ct);
        for (int k = tid - nmax; k <= nmax; k += PP_NT) {
            const int ak = abs(k);
            double d0 = 1.0, d01 = 0.0, sben = 1.0;
            for (int n = 1; n <= ak; n++) {
                sben = sben * sbe / 2.0;
                if (sben < 1.0e-30) sben = 0.0;
            }
            if (ak > 0) {
                d0 = pm1(ak) * sben * a.bcofd[ak];
                if (k < 0) d0 = pm1(ak) * d0;
                if (used(ak)) D[(size_t)W * ak * ak + nmin * (2 * ak + 1) + k + ak] = d0;
            }
            for (int n = ak + 1; n <= nmax; n++) {
                const double v = (ct * (double)(n + n - 1) * d0 - a.fnr[n - k - 1] * a.fnr[n + k - 1] * d01) / (a.fnr[n + k] * a.fnr[n - k]);
                d01 = d0;
                d0 = v;
                if (used(n)) D[(size_t)W * n * n + nmin * (2 * n + 1) + k + n] = v;
            }
        }
        // phase (shift_op = F: e^{+i m phi} on the source) needs eph: after the barrier
        __syncthreads();
        {
            double* row0 = reinterpret_cast<double*>(mg_smem) + (size_t)warp * 2 * (2 * nmax + 3);
            double* row1 = row0 + 2 * nmax + 3;
            for (int n = nmax - warp; n >= 1; n -= PP_NT / 32) {
                if (!used(n)) continue;
                const int kk = min(n, nmin), ld = 2 * n + 1;
                double* Dn = D + (size_t)W * n * n + nmin * ld + n;   // (m, k) at m ld + k
                double *cur = row0, *nxt = row1;                      // column k at k + n + 1, a zero at either end
                for (int k = -n + lane; k <= n; k += 32) cur[k + n + 1] = Dn[k];
                if (lane < 2) {
                    row0[lane * (ld + 1)] = 0.0;
                    row1[lane * (ld + 1)] = 0.0;
                }
                double fm = 0.0;   // of m = lane + 1
                if (lane < kk) fm = 1.0 / a.fnr[n - lane] / a.fnr[n + lane + 1];
                __syncwarp();
                for (int m = 1; m <= kk; m++) {
                    const double fmn = __shfl_sync(0xffffffffu, fm, m - 1), im = pm1(m);
                    for (int k = -n + lane; k <= n; k += 32) {
                        const double v = (a.fnr[n + k] * a.fnr[n - k + 1] * cbe2 * cur[k + n] - a.fnr[n - k] * a.fnr[n + k + 1] * sbe2 * cur[k + n + 2] -
                                          (double)k * sbe * cur[k + n + 1]) * fmn;
                        nxt[k + n + 1] = v;
                        Dn[m * ld + k] = v;
                        Dn[-m * ld - k] = v * pm1(k) * im;
                    }
                    __syncwarp();
                    double* t = cur;
                    cur = nxt;
                    nxt = t;
                }
            }
        }
        // axial blocks of every degree ma (regular functions), kept for all columns:
        // every element its vector-coupling sum, n fastest as the table lies
        for (int e = tid; e < (nmin + 1) * (L - l0 + 1) * nt; e += PP_NT) {
            const int n = e % nt + 1, l = l0 + (e / nt) % (L - l0 + 1), ma = e / (nt * (L - l0 + 1));
            if (n < ma || l < ma) continue;
            const int wmin = abs(n - l), wmax = n + l, ml = l * (l + 1) + ma;
            const double* vc = a.vcc + (n - 1) + (size_t)a.vcT * (ml - 1);
            const size_t vw = (size_t)a.vcT * a.vcML;
            zd s1 = vc[vw * wmin] * xi[wmin], s2 = mk(0.0, 0.0);
#pragma unroll 2
            for (int w = wmin + 1; w < wmax; w += 2) {
                s2 = s2 + vc[vw * w] * xi[w];
                s1 = s1 + vc[vw * (w + 1)] * xi[w + 1];
            }
            s2 = imul(s2);
            zd* Z = Zall + (size_t)ma * 2 * nt * L + (n - 1) * L + (l - 1);
            Z[0] = s1 + s2;
            Z[nt * L] = s1 - s2;
        }
        const zd* e = eph + nmax;
        const int xl = L * (L + 2);
        for (int it = tid; it < np * 2 * xl; it += PP_NT) {
            const int pc = it / (2 * xl), q = (it / xl) % 2, loc = it % xl;
            const int row = loc % (L + 2), col = loc / (L + 2) + 1;
            const int l = row <= col ? col : row - 1, m = row <= col ? row : -col;
            if (l >= l0) XP[((size_t)pc * 2 + q) * xl + l * l - 1 + l + m] = src[(size_t)(p0 + pc) * a.ld + soff + (size_t)q * xl + loc] * e[m];
        }
        __syncthreads();
        // forward rotation of the source degrees, every column
        for (int it = tid; it < np * 2 * (L - l0 + 1) * W; it += PP_NT) {
            const int k = it % W - nmin, l = l0 + (it / W) % (L - l0 + 1), pq = it / (W * (L - l0 + 1));
            zd acc = mk(0.0, 0.0);
            if (abs(k) <= min(l, nt)) {
                const double* Dl = D + (size_t)W * l * l + (k + nmin) * (2 * l + 1);
                const zd* x = XP + (size_t)pq * xl + l * l - 1;
#pragma unroll 4
                for (int m = 0; m <= 2 * l; m++) acc = acc + Dl[m] * x[m];
            }
            AP[((size_t)pq * L + (l - 1)) * W + (k + nmin)] = acc;
        }
        __syncthreads();
        // g(+ma, n, p) = Z[mode p] a'(+ma) ; g(-ma, n, p) = Z[mode 1-p] a'(-ma), every degree ma and column
        {
            // items (column, ma, sign, mode, n) with n = max(1, ma) .. nt
            const int per_col = 2 * 2 * (nt + nt * nmin - (nmin * (nmin - 1)) / 2);   // 4 x sum over ma of the rows
            for (int it = tid; it < np * per_col; it += PP_NT) {
                const int pc = it / per_col;
                int rem = it - pc * per_col;
                int ma = 0;
                for (;; ma++) {
                    const int rows = nt - max(1, ma) + 1;
                    if (rem < 4 * rows) break;
                    rem -= 4 * rows;
                }
                const int m1 = max(1, ma), rows = nt - m1 + 1;
                const int sg = rem / (2 * rows);
                rem -= sg * 2 * rows;
                const int pm = rem / rows, n = m1 + rem % rows;
                if (ma == 0 && sg == 1) continue;
                const int mm = sg ? -ma : ma;
                const int pz = (ma == 0) ? 0 : (sg == 0 ? pm : 1 - pm);
                const zd* Z = Zall + (size_t)ma * 2 * nt * L;
                const zd* ap = AP + ((size_t)pc * 2 + pm) * L * W;
                zd acc = mk(0.0, 0.0);
                for (int l = max(m1, l0); l <= L; l++) acc = acc + Z[(pz * nt + (n - 1)) * L + (l - 1)] * ap[(l - 1) * W + (mm + nmin)];
                G[(((size_t)pc * 2 + pm) * nt + (n - 1)) * W + (mm + nmin)] = acc;
            }
        }
        __syncthreads();
        // back rotation per target degree n, phase back, LR -> TE/TM, accumulate
        for (int it = tid; it < np * nt * (nt + 2); it += PP_NT) {
            const int pc = it / (nt * (nt + 2)), ee = it - pc * (nt * (nt + 2));
            const int p = p0 + pc;
            int n = (int)sqrtf((float)(ee + 1));   // n n - 1 <= ee < (n + 1)(n + 1) - 1
            while (n * (n + 2) <= ee) n++;
            while (n * n - 1 > ee) n--;
            int k = ee - (n * n - 1) - n;   // -n..n
            int n1 = min(n, L);
            const double* Dn = D + (size_t)W * n * n;
            zd gq[2];
            for (int pm = 0; pm < 2; pm++) {
                const zd* g = G + ((size_t)pc * 2 + pm) * nt * W;
                zd acc = mk(0.0, 0.0);
                for (int m = -n1; m <= n1; m++) acc = acc + Dn[(m + nmin) * (2 * n + 1) + (k + n)] * g[(n - 1) * W + (m + nmin)];
                gq[pm] = acc * e[-k];   // phase back: e^{-i k phi}
            }
            if (dist) {
                zd* od = a.out + (size_t)p * a.ldo + a.offset[i];
                od[aidx(k, n, 0, nt)] = gq[0];
                od[aidx(k, n, 1, nt)] = gq[1];
                continue;
            }
            int s_ = aidx(k, n, 0, T);
            zd* o = a.amnp0 + (size_t)p * a.ld0;
            atomicAdd(&o[s_].x, gq[0].x + gq[1].x);
            atomicAdd(&o[s_].y, gq[0].y + gq[1].y);
            atomicAdd(&o[s_ + T * (T + 2)].x, gq[0].x - gq[1].x);
            atomicAdd(&o[s_ + T * (T + 2)].y, gq[0].y - gq[1].y);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// fosmexpansion: one CTA per (n, l).  The terms of (m, p, q) in the elements
// of degree w are a weight without w times a coupling coefficient of (m, w),
// so that each element is a matrix-vector product over m: per chunk of FO_MC
// orders m, a thread per coupling row (three kinds) fills shared memory, a warp
// forms the weights (summed over the (p, q) of one parity of p + q: that
// parity against n + l + w decides the element), then a thread per w sums
// over m.  With the lanes over m and a butterfly per (p, q, w) the kernel took
// 2.63 ms for the 350-sphere aggregate of order 9 (rows in strided global
// scratch); now 0.44 ms.
// ---------------------------------------------------------------------------
#define FO_MC 32
#define FO_NT 128
__global__ void __launch_bounds__(FO_NT) fosm_kernel(int ntot, int mc, const zd* a0, VCTab tab, double* s00, double* s02, double* sp22,
                                                     double* sm22)
{
    extern __shared__ __align__(16) double fo_smem[];
    // weights of (m, parity of p + q): on cmmpm for n + l + w of the same
    // parity (0, 1) and the other (2, 3), on cmmm2pm, cmmp2pm likewise (4..7),
    // and the four of the w >= 2 diagonal elements, both parities (8..11)
    __shared__ double wt[FO_MC][2][12];
    const int tid = threadIdx.x, VL = 2 * ntot + 2;
    double* c1[2] = {fo_smem, fo_smem + VL};   // cm1p1, cm1m1
    double* rows = fo_smem + 2 * VL;           // [kind][m][w]
    // large (n, l) first
    const int nl = ntot * ntot - 1 - (int)blockIdx.x, n = nl / ntot + 1, l = nl % ntot + 1;
    const int nb = 2 * ntot * (ntot + 2), half = ntot * (ntot + 2);
    const int wmin = abs(n - l), wmax = n + l, mm = min(n, l + 2);
    const zd fnl = sqrt((double)((n + n + 1) * (l + l + 1))) * ipow_z(l - n);
    if (tid >= 96 && tid < 98) vc_func(tab, -1, n, tid == 96 ? 1 : -1, l, c1[tid - 96]);   // independent of m
    for (int m0 = -mm; m0 <= mm; m0 += mc) {
        const int cnt = min(mc, mm - m0 + 1);
        if (tid < 96) {
            const int kind = tid / 32, j = tid % 32, m = m0 + j, k = m + (kind == 0 ? 0 : (kind == 1 ? -2 : 2));
            if (j < cnt) {
                double* v = rows + (size_t)(kind * mc + j) * VL;
                if (abs(k) <= l) vc_func(tab, -m, n, k, l, v);
                else
                    for (int w = wmin; w <= wmax; w++) v[w] = 0.0;
            }
        } else if (tid - 96 < cnt) {
            const int m = m0 + tid - 96;
            auto A = [&](int pol, int mq, int nq, int p) -> zd {
                if (mq < -nq || mq > nq) return mk(0.0, 0.0);
                return a0[(size_t)pol * nb + aidx(mq, nq, 0, ntot) + (size_t)half * p];
            };
            const double m1m = pm1(m);
            for (int c = 0; c < 2; c++) {
                double w[12];
                for (int e = 0; e < 12; e++) w[e] = 0.0;
                for (int p = 1; p <= 2; p++) {
                    const int q = c == 0 ? p : 3 - p;
                    const double m1mq = pm1(m + q), m1mnpl = pm1(m + n + p + l);
                    const zd a1n = A(0, m, n, p - 1), a2n = A(1, m, n, p - 1), a1l = A(0, m, l, q - 1), a2l = A(1, m, l, q - 1);
                    const zd a1122 = (a1n * cj(a1l) + a2n * cj(a2l)) * fnl, a2112 = (a2n * cj(a1l) - a1n * cj(a2l)) * fnl;
                    const zd a1p2 = (a1n + imul(a2n)) * cj(A(0, m - 2, l, q - 1) - imul(A(1, m - 2, l, q - 1))) * fnl;
                    const zd a1m2 = (a1n - imul(a2n)) * cj(A(0, m + 2, l, q - 1) + imul(A(1, m + 2, l, q - 1))) * fnl;
                    w[0] += -m1m * a1122.x / 2.0;       // cm1p1: s00(1,1)
                    w[1] += -m1mq * a1122.x / 2.0;      // cm1m1: s02(2,1)
                    w[2] += -m1m * a2112.y / 2.0;       // cm1p1: s00(4,4)
                    w[3] += -m1mq * a2112.x / 2.0;      // cm1m1: s02(3,4)
                    w[4] += -m1m * a1p2.x / 4.0;        // cm1p1: s02(1,2)
                    w[5] += -m1m * a1m2.x / 4.0;
                    w[6] += m1m * a1p2.y / 4.0;         // cm1p1: s02(4,3)
                    w[7] += -m1m * a1m2.y / 4.0;
                    w[8] += -m1mnpl * a1p2.x / 8.0;     // cm1m1: sm22(2,2), times (-1)^w on cmmm2pm
                    w[9] += -m1mq * a1m2.x / 8.0;
                    w[10] += -m1mq * a1p2.x / 8.0;      // cm1m1: sp22(2,2), times (-1)^w on cmmp2pm
                    w[11] += -m1mnpl * a1m2.x / 8.0;
                }
                for (int e = 0; e < 12; e++) wt[tid - 96][c][e] = w[e];
            }
        }
        __syncthreads();
        for (int w = wmin + tid; w <= wmax; w += FO_NT) {
            const int ev = (n + l + w) & 1, od = 1 - ev;
            const double m1w = pm1(w);
            double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int j = 0; j < cnt; j++) {
                const double c0 = rows[(size_t)j * VL + w], cm = rows[(size_t)(mc + j) * VL + w], cp = rows[(size_t)(2 * mc + j) * VL + w];
                const double *we = wt[j][ev], *wo = wt[j][od];
                t[0] += we[0] * c0;
                t[1] += we[1] * c0;
                t[2] += wo[2] * c0;
                t[3] += wo[3] * c0;
                t[4] += we[4] * cm + we[5] * cp;
                t[5] += wo[6] * cm + wo[7] * cp;
                t[6] += m1w * (we[8] + wo[8]) * cm + (we[9] + wo[9]) * cp;
                t[7] += (we[10] + wo[10]) * cm + m1w * (we[11] + wo[11]) * cp;
            }
            const double p1 = c1[0][w], q1 = c1[1][w];
#define SS(arr, i, j) (&arr[((i) - 1) + 4 * ((j) - 1) + 16 * w])
            atomicAdd(SS(s00, 1, 1), p1 * t[0]);
            atomicAdd(SS(s00, 4, 4), p1 * t[2]);
            if (w >= 2) {
                atomicAdd(SS(s02, 2, 1), q1 * t[1]);
                atomicAdd(SS(s02, 3, 4), q1 * t[3]);
                atomicAdd(SS(s02, 1, 2), p1 * t[4]);
                atomicAdd(SS(s02, 4, 3), p1 * t[5]);
                atomicAdd(SS(sm22, 2, 2), q1 * t[6]);
                atomicAdd(SS(sp22, 2, 2), q1 * t[7]);
            }
#undef SS
        }
        __syncthreads();
    }
}

// the sign patches and the 1/(2 m_medium) factor of fosmexpansion
// (a thread per table and degree, its 16 values in registers; in place in
// global memory, a thread per degree, it took 35 us at order 48; now 6)
__global__ void fosm_patch_kernel(int ntot, double* s00, double* s02, double* sp22, double* sm22, double scale)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x, w = e / 4, k = e % 4;
    if (w > 2 * ntot) return;
    double* S = (k == 0 ? s00 : (k == 1 ? s02 : (k == 2 ? sm22 : sp22))) + 16 * (size_t)w;
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = S[q];
#pragma unroll
    for (int i = 3; i <= 4; i++)
#pragma unroll
        for (int j = 1; j <= i; j++) v[(j - 1) + 4 * (i - 1)] = -v[(j - 1) + 4 * (i - 1)];
    if (k == 2) v[2 + 4 * 2] = -v[1 + 4 * 1];
    if (k == 3) v[2 + 4 * 2] = v[1 + 4 * 1];
#pragma unroll
    for (int q = 0; q < 16; q++) S[q] = 0.5 * v[q] / scale;
}

// fosmcalc at each angle: one CTA per angle; the functions of every degree
// (gsfrows.cuh), then the sum over w and the element patches
__global__ void __launch_bounds__(GSF_NT) fosmcalc_kernel(int ntot, int nang, const double* s00, const double* s02, const double* sp22,
                                                          const double* sm22, const double* fnr, const double* bcofd, double* smat)
{
    extern __shared__ __align__(16) double gsf_smem[];
    const int ia = blockIdx.x;
    if (ia >= nang) return;
    // polar angle as scattering_matrix_calculation forms it (input:3039-3043), pi as MSTM stores it
    double ct = cos(MSTMG_REF_PI / 180.0 * (0.0 + (180.0 - 0.0) * (double)ia / (double)(nang - 1)));
    if (ct == 1.0) ct = 0.9999999;
    if (ct == -1.0) ct = -0.9999999;
    const int nmax = 2 * ntot;
    gsf_columns(nmax, ct, fnr, bcofd, gsf_smem);
    __shared__ double red[GSF_NT / 16][16];
    __shared__ double acc[16];
    const int e = threadIdx.x % 16, part = threadIdx.x / 16;
    double v = part == 0 ? s00[e] * 1.0 : 0.0;   // degree 0: dc(0,0) = 1
    // terms: w = n uses dc(0, n(n+1)) [k=0 column]; dc(0,n(n+1)+2), dc(+-2, n(n+1)+2) [k=2]
    for (int n = 1 + part; n <= nmax; n += GSF_NT / 16) {
        const double* g = gsf_smem + GSF_ROW * n;
        v += s00[e + 16 * n] * g[GSF_D00];
        if (n >= 2) v += s02[e + 16 * n] * g[GSF_D02] + sp22[e + 16 * n] * g[GSF_D22] + sm22[e + 16 * n] * g[GSF_DM22];
    }
    red[part][e] = v;
    __syncthreads();
    if (threadIdx.x < 16) {
        double t = 0.0;
        for (int p = 0; p < GSF_NT / 16; p++) t += red[p][threadIdx.x];
        acc[threadIdx.x] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sm[16];
        for (int e = 0; e < 16; e++) sm[e] = acc[e];
#define SM(i, j) sm[((i) - 1) + 4 * ((j) - 1)]
        SM(3, 1) = -SM(3, 1);
        SM(1, 3) = -SM(1, 3);
        SM(4, 3) = -SM(4, 3);
        double temp = SM(4, 1);
        SM(4, 1) = SM(4, 2);
        SM(4, 2) = temp;
        SM(1, 2) = (SM(1, 2) + SM(2, 1)) / 2.0;
        SM(2, 1) = SM(1, 2);
        SM(3, 4) = (SM(3, 4) - SM(4, 3)) / 2.0;
        SM(4, 3) = -SM(3, 4);
#undef SM
        for (int e = 0; e < 16; e++) smat[(size_t)ia * 16 + e] = sm[e];
    }
}

// scatteringmatrix (scatprops:1498-1573) with normalize_s11 = .false. at the
// directions of scattering_matrix_calculation (input:3038-3061): one CTA per
// direction.  rotcoef(ct, 1, T) advances degree by degree in shared memory;
// per degree the threads take the orders m = -n..n, form the two tau
// functions of taufunc (modules:1324-1344) and add their terms to the four
// amplitude sums, which are reduced over the CTA at the end; thread 0 forms
// the 4x4 matrix (amplitude_to_scattering_matrix, scatprops:1410-1436).
#define PS_NT 128
__global__ void __launch_bounds__(PS_NT) planesm_kernel(PlaneSmArgs a)
{
    const int ia = blockIdx.x;
    const int i = a.ldim + ia;
    if (i > a.udim) return;
    const int T = a.T;
    __shared__ double dk0s[2 * PS_TMAX + 3], dk01s[2 * PS_TMAX + 3], dcs[3 * (2 * PS_TMAX + 1)];
    __shared__ double red[8][PS_NT / 32];
    double* dk0 = dk0s + (T + 1);
    double* dk01 = dk01s + (T + 1);
    const int W = 2 * T + 1;
#define DCR(m, k) dcs[((m) + 1) * W + ((k) + T)]
    double ct = cos(MSTMG_REF_PI / 180.0 * (a.amin + (a.amax - a.amin) * (double)(i - a.ldim) / (double)(a.udim - a.ldim)));
    if (ct == 1.0) ct = 0.9999999;
    if (ct == -1.0) ct = -0.9999999;
    const double phi = (i < 0) ? a.alpha + MSTMG_REF_PI : a.alpha;
    double cphi, sphi;
    sincos(phi, &sphi, &cphi);
    const double* fnr = a.fnr;
    double sbe = (fabs(ct) >= 1.0) ? 0.0 : sqrt(fabs((1.0 + ct) * (1.0 - ct)));
    double cbe2 = 0.5 * (1.0 + ct), sbe2 = 0.5 * (1.0 - ct);
    for (int k = threadIdx.x; k < 2 * T + 3; k += blockDim.x) { dk0s[k] = 0.0; dk01s[k] = 0.0; }
    __syncthreads();
    if (threadIdx.x == 0) dk0[0] = 1.0;
    __syncthreads();
    zd sa[4];
    for (int e = 0; e < 4; e++) sa[e] = mk(0.0, 0.0);
    const size_t ld = 2 * (size_t)T * (T + 2);
    int sgn = 1;
    double sben = 1.0;
    for (int n = 1; n <= T; n++) {
        sgn = -sgn;
        sben = sben * sbe / 2.0;
        if (sben < 1.0e-30) sben = 0.0;
        double newv[(2 * PS_TMAX + PS_NT - 1) / PS_NT];
        int cnt = 0;
        for (int k = -n + 1 + (int)threadIdx.x; k <= n - 1; k += blockDim.x)
            newv[cnt++] = (ct * (double)(n + n - 1) * dk0[k] - fnr[n - k - 1] * fnr[n + k - 1] * dk01[k]) / (fnr[n + k] * fnr[n - k]);
        __syncthreads();
        cnt = 0;
        for (int k = -n + 1 + (int)threadIdx.x; k <= n - 1; k += blockDim.x) {
            dk01[k] = dk0[k];
            dk0[k] = newv[cnt++];
        }
        if (threadIdx.x == 0) {
            dk0[n] = sgn * sben * a.bcofd[n];
            dk0[-n] = sgn * dk0[n];
            dk01[n] = 0.0;
            dk01[-n] = 0.0;
        }
        __syncthreads();
        for (int k = -n + (int)threadIdx.x; k <= n; k += blockDim.x) DCR(0, k) = dk0[k];
        __syncthreads();
        {
            const double fmn = 1.0 / fnr[n] / fnr[n + 1];
            for (int k = -n + (int)threadIdx.x; k <= n; k += blockDim.x) {
                double dkm1 = (k == -n) ? 0.0 : DCR(0, k - 1);
                double dkn1 = (k == n) ? 0.0 : DCR(0, k + 1);
                double v = (fnr[n + k] * fnr[n - k + 1] * cbe2 * dkm1 - fnr[n - k] * fnr[n + k + 1] * sbe2 * dkn1 -
                            (double)k * sbe * DCR(0, k)) * fmn;
                DCR(1, k) = v;
                DCR(-1, -k) = -v * pm1(k);
            }
        }
        __syncthreads();
        // (-i)^n
        const zd cin = (n & 3) == 0 ? mk(1.0, 0.0) : (n & 3) == 1 ? mk(0.0, -1.0) : (n & 3) == 2 ? mk(-1.0, 0.0) : mk(0.0, 1.0);
        const double fnm = sqrt((double)(n + n + 1) / 2.0) / 4.0;
        for (int m = -n + (int)threadIdx.x; m <= n; m += blockDim.x) {
            const double tau[2] = {-fnm * (-DCR(-1, m) + DCR(1, m)), -fnm * (DCR(-1, m) + DCR(1, m))};
            const int m1 = (m <= -1) ? n + 1 : m, n1 = (m <= -1) ? -m : n;
            double sm_, cm_;
            sincos((double)m * phi, &sm_, &cm_);
            const zd ce = cin * mk(cm_, sm_);
            for (int p = 0; p < 2; p++) {
                const size_t ix = (size_t)aidx(m1, n1, p, T);
                const zd a1 = a.a0[ix], a2 = a.a0[ix + ld];
                zd av, bv;
                if (a.rotate) {
                    av = cphi * a1 + sphi * a2;
                    bv = sphi * a1 - cphi * a2;
                } else {
                    av = a1;
                    bv = -a2;
                }
                const zd tb = ce * bv, ta = ce * av;
                sa[0] = sa[0] + tau[1 - p] * tb;
                sa[1] = sa[1] + tau[p] * imul(ta);
                sa[2] = sa[2] + tau[p] * imul(tb);
                sa[3] = sa[3] + tau[1 - p] * ta;
            }
        }
        __syncthreads();
    }
#undef DCR
    // CTA reduction of the 8 doubles
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double v8[8] = {sa[0].x, sa[0].y, sa[1].x, sa[1].y, sa[2].x, sa[2].y, sa[3].x, sa[3].y};
    for (int e = 0; e < 8; e++) {
        double v = v8[e];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[e][wid] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        zd s[4];
        for (int e = 0; e < 4; e++) {
            double re = 0.0, im = 0.0;
            for (int w = 0; w < PS_NT / 32; w++) { re += red[2 * e][w]; im += red[2 * e + 1][w]; }
            s[e] = (4.0 / sqrt(2.0 * (1.0 / MSTMG_REF_PI))) * mk(re, im);
        }
        zd sp[4][4];
        for (int r = 0; r < 4; r++)
            for (int q = 0; q < 4; q++) sp[r][q] = s[r] * cj(s[q]);
        double sm[16];
#define SP(r, q) sp[(r) - 1][(q) - 1]
#define SM(r, q) sm[((r) - 1) + 4 * ((q) - 1)]
        SM(1, 1) = (SP(1, 1) + SP(2, 2) + SP(3, 3) + SP(4, 4)).x;
        SM(1, 2) = (-SP(1, 1) + SP(2, 2) - SP(3, 3) + SP(4, 4)).x;
        SM(2, 1) = (-SP(1, 1) + SP(2, 2) + SP(3, 3) - SP(4, 4)).x;
        SM(2, 2) = (SP(1, 1) + SP(2, 2) - SP(3, 3) - SP(4, 4)).x;
        SM(3, 3) = 2.0 * (SP(1, 2) + SP(3, 4)).x;
        SM(3, 4) = 2.0 * (SP(2, 1) + SP(4, 3)).y;
        SM(4, 3) = 2.0 * (SP(1, 2) - SP(3, 4)).y;
        SM(4, 4) = 2.0 * (SP(1, 2) - SP(3, 4)).x;
        SM(1, 3) = 2.0 * (SP(2, 3) + SP(1, 4)).x;
        SM(3, 1) = 2.0 * (SP(2, 4) + SP(1, 3)).x;
        SM(1, 4) = -2.0 * (SP(2, 3) - SP(1, 4)).y;
        SM(4, 1) = -2.0 * (SP(4, 2) + SP(1, 3)).y;
        SM(2, 3) = -2.0 * (SP(2, 3) - SP(1, 4)).x;
        SM(3, 2) = -2.0 * (SP(2, 4) - SP(1, 3)).x;
        SM(2, 4) = -2.0 * (SP(2, 3) + SP(1, 4)).y;
        SM(4, 2) = -2.0 * (SP(4, 2) - SP(1, 3)).y;
#undef SP
#undef SM
        for (int e = 0; e < 16; e++) a.smat[(size_t)ia * 16 + e] = sm[e] / (4.0 * MSTMG_REF_PI) / a.rimed_re;
    }
}

void launch_tranorder(int nsph, const double* pos, const int* order, const double* origin, double rire, double eps, int maxt,
                      const double* bcof, const double* fnr, int nbc, int* tord, int nsm, cudaStream_t st)
{
    VCTab t{bcof, fnr, nbc};
    // a warp per sphere, three to an SM (72 KB of shared memory each)
    const int smem = (int)(sizeof(zd) * 2 * TRANORDER_ROW + sizeof(double) * 32 * TRANORDER_ROW);
    allow_smem(tranorder_kernel, smem);
    tranorder_kernel<<<std::max(1, std::min(nsph, 3 * nsm)), 32, smem, st>>>(nsph, pos, order, origin[0], origin[1], origin[2], rire, eps, maxt,
                                                                             t, tord);
    launch_counter() += 1;
}

void launch_regular_couplings(int Tt, int Ls, const double* bcof, const double* fnr, int nbc, double* vcc, cudaStream_t st)
{
    VCTab t{bcof, fnr, nbc};
    const int smem = (int)sizeof(double) * (2 * std::min(Tt, Ls) + 2) * (Tt + Ls + 1);
    allow_smem(regular_couplings_kernel, smem);
    regular_couplings_kernel<<<dim3(Tt, Ls), RC_NT, smem, st>>>(Tt, Ls, t, vcc);
    launch_counter() += 1;
}

size_t merge_scratch_per_cta(int T, int L, int npol)
{
    const size_t nmin = std::min(T, L), nmax = std::max(T, L), W = 2 * nmin + 1, np = std::min(npol, MERGE_PC);
    const size_t z = (nmax + L + 4) * 3 + (2 * nmax + 1);               // xi + Bessel scratch + e^{i m phi}
    const size_t dbl = (W * (nmax + 1) * (nmax + 1) + 1) / 2 * 2;       // D
    const size_t zz = (nmin + 1) * 2 * T * L + np * (2 * (size_t)L * W + 2 * (size_t)T * W + 2 * (size_t)L * (L + 2));
    return z + dbl / 2 + zz + 8;                                        // in zd units
}
int merge_chunks(int npol) { return (npol + MERGE_PC - 1) / MERGE_PC; }

void launch_merge(const MergeArgs& a, int grid, cudaStream_t st)
{
    // two rows of the Wigner recurrence a warp; orders reach MSTMG_LMAX and T
    const int nmax = std::max(a.T, MSTMG_LMAX), smem = (int)sizeof(double) * (PP_NT / 32) * 2 * (2 * nmax + 3);
    allow_smem(merge_kernel, smem);
    merge_kernel<<<dim3(grid, merge_chunks(a.npol)), PP_NT, smem, st>>>(a);
    launch_counter() += 1;
}

void launch_fosm(int ntot, const zd* a0, const double* bcof, const double* fnr, int nbc, double* s00, double* s02, double* sp22,
                 double* sm22, cudaStream_t st)
{
    VCTab t{bcof, fnr, nbc};
    // FO_MC orders m a chunk while three rows of each fit 200 KB (order 128)
    const int row = (int)sizeof(double) * (2 * ntot + 2), mc = std::max(1, std::min(FO_MC, (200 * 1024 - 2 * row) / (3 * row)));
    const int smem = row * (2 + 3 * mc);
    allow_smem(fosm_kernel, smem);
    fosm_kernel<<<ntot * ntot, FO_NT, smem, st>>>(ntot, mc, a0, t, s00, s02, sp22, sm22);
    fosm_patch_kernel<<<(4 * (2 * ntot + 1) + 63) / 64, 64, 0, st>>>(ntot, s00, s02, sp22, sm22, 1.0);
    launch_counter() += 2;
}

void launch_fosmcalc(int ntot, int nang, const double* s00, const double* s02, const double* sp22, const double* sm22,
                     const double* fnr, const double* bcofd, double* smat, cudaStream_t st)
{
    fosmcalc_kernel<<<nang, GSF_NT, gsf_smem_bytes(2 * ntot), st>>>(ntot, nang, s00, s02, sp22, sm22, fnr, bcofd, smat);
    launch_counter() += 1;
}

void launch_planesm(const PlaneSmArgs& a, cudaStream_t st)
{
    planesm_kernel<<<a.udim - a.ldim + 1, PS_NT, 0, st>>>(a);
    launch_counter() += 1;
}
