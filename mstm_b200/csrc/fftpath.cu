// fftpath.cu -- MSTM's FFT translation for large clusters
// (fft_translation-5.f90): near pairs go through the pair kernels; the rest
// travels sphere -> cell node (regular translation), node -> node (outgoing
// translation as a convolution on the zero-padded cell grid, evaluated with
// FFTs), node -> sphere (regular translation).
//
//   fft_j_kernel       per sphere, the dense regular translations to and from
//                      its node (gentranmatrix, vswf_type 1; the identity
//                      for translations shorter than 1e-3, the reference's
//                      zero_translation)                         fft:482-652
//   fft_hbuild_kernel  per slot of the (2 cell_dim)^3 grid, the outgoing
//                      translation matrices of the node offsets that map to
//                      it, summed in single precision in the reference's
//                      octant order (fft:901-974); a batched double FFT then
//                      gives the stored single-precision spectra
//   fft_s2n_kernel     x (shifted for conjugate-transpose columns) -> node
//                      coefficients on the padded grid (atomic adds: a cell
//                      holds several spheres)
//   fft_mul_kernel     per frequency: g(l) = sum_n H(l, n) a(n), both modes,
//                      all columns                                 fft:827-899
//   fft_n2s_kernel     node coefficients -> sphere (1/N of the inverse FFT
//                      folded in), shifted back, added to y
#include <type_traits>
#include "common.cuh"
#include "gentran.cuh"
#include "fftpath.cuh"
#include "tables.h"
#include <algorithm>
#include <cmath>

void gentran_constants(int nmax, std::vector<double>& tc)
{
    mstmg::Tables tb(6 * nmax + 6);
    const int nd = nmax * (nmax + 2);
    tc.assign((size_t)nd * nd * (2 * nmax + 1), 0.0);
    std::vector<double> vc1(2 * nmax + 2), vc2(2 * nmax + 2);
    for (int l = 1; l <= nmax; l++)
        for (int n = 1; n <= nmax; n++) {
            const int wmax = n + l;
            tb.vcfunc(-1, n, 1, l, vc2.data());
            // c = -i^(n-l) sqrt(2n+1) sqrt(2l+1)
            int e0 = ((n - l) % 4 + 4) % 4;
            double ire = (e0 == 0) ? 1.0 : (e0 == 2 ? -1.0 : 0.0), iim = (e0 == 1) ? 1.0 : (e0 == 3 ? -1.0 : 0.0);
            double cre = (-ire * tb.fnr[n + n + 1]) * tb.fnr[l + l + 1], cim = (-iim * tb.fnr[n + n + 1]) * tb.fnr[l + l + 1];
            for (int k = -l; k <= l; k++) {
                const int kl = l * (l + 1) + k;
                for (int m = -n; m <= n; m++) {
                    const int mn = n * (n + 1) + m;
                    const double m1m = (m & 1) ? -1.0 : 1.0;
                    const int v = k - m;
                    tb.vcfunc(-m, n, k, l, vc1.data());
                    const int wmin = std::max(std::abs(v), std::abs(n - l));
                    for (int w = wmax; w >= wmin; w--) {
                        // i^w c exactly, then times (-1)^m, vc1(w), vc2(w) in the reference's order
                        int e = w % 4;
                        double are, aim;
                        if (e == 0) { are = cre; aim = cim; }
                        else if (e == 1) { are = -cim; aim = cre; }
                        else if (e == 2) { are = -cre; aim = -cim; }
                        else { are = cim; aim = -cre; }
                        are = ((are * m1m) * vc1[w]) * vc2[w];
                        aim = ((aim * m1m) * vc1[w]) * vc2[w];
                        tc[(size_t)(mn - 1) + (size_t)nd * ((size_t)(kl - 1) + (size_t)nd * w)] = ((wmax - w) % 2 == 0) ? are : aim;
                    }
                }
            }
        }
}

// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(FFT_NT) fft_j_kernel(FftJArgs a)
{
    __shared__ GtShared gs;
    const int i = blockIdx.x;
    if (i >= a.nsph) return;
    const int L = a.order[i], nb = L * (L + 2), No = a.No, nbN = No * (No + 2);
    double rv[3], r2 = 0.0;
    for (int m = 0; m < 3; m++) {
        int nd = a.snode[3 * i + m];   // 1-based cell
        rv[m] = a.dcell * ((double)nd - 0.5) - a.pos[3 * i + m] + a.cb[m];
        r2 += rv[m] * rv[m];
    }
    const bool ident = r2 < 1.0e-6;   // the reference's zero_translation
    zd* Jsn = a.Jsn + a.joff[i];       // nbN x nb x 2 (target node, source sphere)
    zd* Jns = a.Jns + a.joff[i];       // nb x nbN x 2
    const zd ri = mk(a.rimed_re, a.rimed_im);
    for (int pass = 0; pass < 2; pass++) {
        const int ns = pass == 0 ? L : No, nt = pass == 0 ? No : L;
        const int nbs = ns * (ns + 2), nbt = nt * (nt + 2);
        zd* out = pass == 0 ? Jsn : Jns;
        if (ident) {
            for (int e = threadIdx.x; e < nbt * nbs; e += FFT_NT) {
                int t = e % nbt, s = e / nbt;
                zd v = (t == s) ? mk(1.0, 0.0) : mk(0.0, 0.0);
                out[e] = v;
                out[e + (size_t)nbt * nbs] = v;
            }
            continue;
        }
        double xp[3] = {pass == 0 ? rv[0] : -rv[0], pass == 0 ? rv[1] : -rv[1], pass == 0 ? rv[2] : -rv[2]};
        const int wmaxt = ns + nt;
        gt_prepare(gs, a.g, xp, 1, ri, wmaxt);
        for (int e = threadIdx.x; e < nbt * nbs; e += FFT_NT) {
            int t = e % nbt, s = e / nbt;
            int m, n, k, l;
            gt_mn(s, ns, m, n);
            gt_mn(t, nt, k, l);
            zd e1, e2;
            gt_element(gs, a.g, 1, wmaxt, n, m, l, k, e1, e2);
            out[e] = e1;
            out[e + (size_t)nbt * nbs] = e2;
        }
        __syncthreads();
    }
    (void)nb;
    (void)nbN;
}

// One CTA per slot of the padded grid: the node offset that maps to the slot
// and the octants that reach it (fft_translation_initialization's loops),
// each octant's H(xp) added in single precision in octant order.
__global__ void __launch_bounds__(FFT_NT) fft_hbuild_kernel(FftHArgs a)
{
    __shared__ GtShared gs;
    const int N0 = 2 * a.cd[0], N1 = 2 * a.cd[1], N2 = 2 * a.cd[2];
    const int nslot = N0 * N1 * N2, No = a.No, nbN = No * (No + 2);
    const zd ri = mk(a.rimed_re, a.rimed_im);
    for (int slot = blockIdx.x; slot < nslot; slot += gridDim.x) {
        const int j0 = slot % N0, j1 = (slot / N0) % N1, j2 = slot / (N0 * N1);
        const int jj[3] = {j0, j1, j2};
        int off[3];
        bool okp[3], okm[3];
        for (int d = 0; d < 3; d++) {
            const int cd = a.cd[d];
            okp[d] = jj[d] <= cd;                     // is = +1: slot = offset
            okm[d] = jj[d] >= cd && jj[d] < 2 * cd;    // is = -1: slot = 2 cd - offset (offset >= 1)
            off[d] = jj[d] <= cd ? jj[d] : 2 * cd - jj[d];
        }
        // the neighbour stencil is a hole in the kernel
        bool hole = false;
        for (int q = 0; q < a.nnb; q++)
            if (off[0] == a.nbv[3 * q] && off[1] == a.nbv[3 * q + 1] && off[2] == a.nbv[3 * q + 2]) hole = true;
        // element (p, target t, source s) of this slot at ((p nbN + t) nbN + s) nslot + slot
        const int nel = 2 * nbN * nbN;
        for (int e = threadIdx.x; e < nel; e += FFT_NT) a.hr[(size_t)e * nslot + slot] = mk(0.0, 0.0);
        __syncthreads();
        if (hole) continue;
        for (int is = 0; is < 8; is++) {
            const int sx = (is & 1) ? -1 : 1, sy = (is & 2) ? -1 : 1, sz = (is & 4) ? -1 : 1;
            if ((sx > 0 ? !okp[0] : !okm[0]) || (sy > 0 ? !okp[1] : !okm[1]) || (sz > 0 ? !okp[2] : !okm[2])) continue;
            double xp[3] = {sx * a.dcell * (double)off[0], sy * a.dcell * (double)off[1], sz * a.dcell * (double)off[2]};
            gt_prepare(gs, a.g, xp, 3, ri, 2 * No);
            for (int e = threadIdx.x; e < nbN * nbN; e += FFT_NT) {
                int t = e % nbN, s = e / nbN;   // target (row l), source (column n)
                int m, n, k, l;
                gt_mn(s, No, m, n);
                gt_mn(t, No, k, l);
                zd e1, e2;
                gt_element(gs, a.g, 3, 2 * No, n, m, l, k, e1, e2);
                // complex(4) accumulation: (float)(acc + h)
                zd* h1 = &a.hr[((size_t)(0 * nbN + t) * nbN + s) * nslot + slot];
                zd* h2 = &a.hr[((size_t)(1 * nbN + t) * nbN + s) * nslot + slot];
                *h1 = mk((double)(float)(h1->x + e1.x), (double)(float)(h1->y + e1.y));
                *h2 = mk((double)(float)(h2->x + e2.x), (double)(float)(h2->y + e2.y));
            }
            __syncthreads();
        }
    }
}

__global__ void fft_round_kernel(size_t n, const zd* in, float2* out)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
        out[e] = make_float2((float)in[e].x, (float)in[e].y);
}

// 8 or 16 bytes in one load
__device__ __forceinline__ zf ldc(const zf* p)
{
    const float2 v = *reinterpret_cast<const float2*>(p);
    return mk(v.x, v.y);
}
__device__ __forceinline__ zd ldc(const zd* p)
{
    const double2 v = *reinterpret_cast<const double2*>(p);
    return mk(v.x, v.y);
}

#define FFT_MB 8   // J records of a thread in flight, the last few of a share included

// The three kernels below are bound by the J records (read once a pass), the
// kernel spectra H (likewise) and the caches: a fixed number of columns NC
// keeps the sums in registers (a runtime count kept them in local memory).
// For 2500 spheres of order 7 and two FP32 columns they took 75 (s2n), 154
// (mul) and 41 us (n2s); now 24, 49 and 28.

// sphere -> node: A[col][p][k][slot_i] += sum_m Jsn_i(k, m, p) (S x_i)(m, p).
// One CTA a sphere; a thread has an element (p, k) and one of the shares the
// sum over m is cut into so that every thread works.
template <typename T, int NC>
__global__ void __launch_bounds__(FFT_MT) fft_s2n_kernel(FftMArgs a, const cpx<T>* J, const cpx<T>* x, int ld, unsigned contran, cpx<T>* A)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    cpx<T>* xs = reinterpret_cast<cpx<T>*>(smraw);   // NC x 2 nbmax
    const int i = blockIdx.x;
    const int L = a.order[i], nb = L * (L + 2), No = a.No, nbN = No * (No + 2);
    cpx<T>* ps = xs + NC * 2 * a.nbmax;              // NC x FFT_MT partial sums
    const size_t N8 = a.N8;
    for (int e = threadIdx.x; e < NC * 2 * nb; e += FFT_MT) {
        int c = e / (2 * nb), el = e % (2 * nb);
        int p = el / nb, idx = el % nb;
        cpx<T> v = x[(size_t)c * ld + a.offset[i] + el];
        if ((contran >> c) & 1u) {
            // shiftcoefficient(-1, -1): a'(+-m, n) = (-1)^m a(-+m, n)
            int m, n;
            gt_mn(idx, L, m, n);
            int src = (m == 0) ? idx : aidx(-m, n, 0, L);
            v = x[(size_t)c * ld + a.offset[i] + p * nb + src];
            if (m & 1) v = mk(-v.x, -v.y);
        }
        xs[e] = v;
    }
    __syncthreads();
    const cpx<T>* Ji = J + a.joff[i];
    const int slot = a.slot[i], items = 2 * nbN;
    const int nsh = max(1, FFT_MT / items), mper = (nb + nsh - 1) / nsh;
    for (int e0 = 0; e0 < items; e0 += FFT_MT) {
        const int cnt = min(items - e0, FFT_MT), sh = threadIdx.x / cnt, e = e0 + threadIdx.x % cnt;
        const int p = e / nbN, k = e % nbN;
        cpx<T> acc[NC];
        for (int c = 0; c < NC; c++) acc[c] = mk((T)0, (T)0);
        if (sh < nsh) {
            const cpx<T>* Jp = Ji + k + (size_t)nbN * nb * p;
            const cpx<T>* xp = xs + p * nb;
            const int m1 = min(nb, (sh + 1) * mper);
            for (int m = sh * mper; m < m1; m += FFT_MB) {
                cpx<T> j[FFT_MB];
#pragma unroll
                for (int u = 0; u < FFT_MB; u++) j[u] = m + u < m1 ? ldc(Jp + (size_t)nbN * (m + u)) : mk((T)0, (T)0);
#pragma unroll
                for (int u = 0; u < FFT_MB; u++)
                    if (m + u < m1)
#pragma unroll
                        for (int c = 0; c < NC; c++) acc[c] = acc[c] + j[u] * xp[c * 2 * nb + m + u];
            }
        }
        if (nsh > 1) {
            for (int c = 0; c < NC; c++) ps[c * FFT_MT + threadIdx.x] = acc[c];
            __syncthreads();
            if (sh == 0)
                for (int c = 0; c < NC; c++)
                    for (int q = 1; q < nsh; q++) acc[c] = acc[c] + ps[c * FFT_MT + threadIdx.x + q * cnt];
        }
        if (sh == 0)
            for (int c = 0; c < NC; c++) {
                cpx<T>* dst = A + ((size_t)(c * 2 + p) * nbN + k) * N8 + slot;
                atomicAdd(&dst->x, acc[c].x);
                atomicAdd(&dst->y, acc[c].y);
            }
    }
}

// per frequency f: G[col][p][l][f] = sum_n H[p][l][n][f] A[col][p][n][f].
// A thread has one f and R rows l of one p (blockIdx.y): every H element is
// read once, coalesced along f, and each A value serves R rows from a register.
template <typename T, int NC, int R>
__global__ void __launch_bounds__(FFT_NT) fft_mul_kernel(int nbN, size_t N8, const float2* H, const cpx<T>* A, cpx<T>* G)
{
    const int ng = (nbN + R - 1) / R, p = blockIdx.y / ng, l0 = (blockIdx.y - p * ng) * R, nr = min(R, nbN - l0);
    const size_t f = blockIdx.x * (size_t)FFT_NT + threadIdx.x;
    if (f >= N8) return;
    const float2* h = H + ((size_t)(p * nbN + l0) * nbN) * N8 + f;
    const cpx<T>* Ap = A + (size_t)p * nbN * N8 + f;
    const size_t cs = (size_t)2 * nbN * N8;   // a column
    cpx<T> acc[R][NC];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < NC; c++) acc[r][c] = mk((T)0, (T)0);
    auto rows = [&](auto full) {
#pragma unroll 2
        for (int n = 0; n < nbN; n++) {
            cpx<T> av[NC];
            float2 hv[R];
#pragma unroll
            for (int r = 0; r < R; r++)
                if (full || r < nr) hv[r] = __ldcs(&h[((size_t)r * nbN + n) * N8]);
#pragma unroll
            for (int c = 0; c < NC; c++) av[c] = ldc(Ap + c * cs + (size_t)n * N8);
#pragma unroll
            for (int r = 0; r < R; r++)
                if (full || r < nr)
#pragma unroll
                    for (int c = 0; c < NC; c++) acc[r][c] = acc[r][c] + mk((T)hv[r].x, (T)hv[r].y) * av[c];
        }
    };
    if (nr == R) rows(std::true_type());
    else rows(std::false_type());
#pragma unroll
    for (int r = 0; r < R; r++)
        if (r < nr)
#pragma unroll
            for (int c = 0; c < NC; c++) G[c * cs + (size_t)(p * nbN + l0 + r) * N8 + f] = acc[r][c];
}

// node -> sphere: y_i += S (Jns_i g_node / N8); the sum over k in shares as in s2n
template <typename T, int NC>
__global__ void __launch_bounds__(FFT_MT) fft_n2s_kernel(FftMArgs a, const cpx<T>* J, const cpx<T>* G, unsigned contran, cpx<T>* y, int ld)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int i = blockIdx.x;
    const int L = a.order[i], nb = L * (L + 2), No = a.No, nbN = No * (No + 2);
    cpx<T>* gs = reinterpret_cast<cpx<T>*>(smraw);   // NC x 2 nbN
    cpx<T>* ys = gs + NC * 2 * nbN;                   // NC x 2 nbmax
    cpx<T>* ps = ys + NC * 2 * a.nbmax;               // NC x FFT_MT partial sums
    const size_t N8 = a.N8;
    const int slot = a.slot[i];
    const T inv = (T)(1.0 / (double)N8);
    for (int e = threadIdx.x; e < NC * 2 * nbN; e += FFT_MT) {
        const cpx<T> v = ldc(G + (size_t)e * N8 + slot);
        gs[e] = mk(v.x * inv, v.y * inv);
    }
    __syncthreads();
    const cpx<T>* Ji = J + a.joff[i];
    const int items = 2 * nb, nsh = max(1, FFT_MT / items), kper = (nbN + nsh - 1) / nsh;
    for (int e0 = 0; e0 < items; e0 += FFT_MT) {
        const int cnt = min(items - e0, FFT_MT), sh = threadIdx.x / cnt, e = e0 + threadIdx.x % cnt;
        const int p = e / nb, m = e % nb;
        cpx<T> acc[NC];
        for (int c = 0; c < NC; c++) acc[c] = mk((T)0, (T)0);
        if (sh < nsh) {
            const cpx<T>* Jp = Ji + m + (size_t)nb * nbN * p;
            const cpx<T>* gp = gs + p * nbN;
            const int k1 = min(nbN, (sh + 1) * kper);
            for (int k = sh * kper; k < k1; k += FFT_MB) {
                cpx<T> j[FFT_MB];
#pragma unroll
                for (int u = 0; u < FFT_MB; u++) j[u] = k + u < k1 ? ldc(Jp + (size_t)nb * (k + u)) : mk((T)0, (T)0);
#pragma unroll
                for (int u = 0; u < FFT_MB; u++)
                    if (k + u < k1)
#pragma unroll
                        for (int c = 0; c < NC; c++) acc[c] = acc[c] + j[u] * gp[c * 2 * nbN + k + u];
            }
        }
        if (nsh > 1) {
            for (int c = 0; c < NC; c++) ps[c * FFT_MT + threadIdx.x] = acc[c];
            __syncthreads();
            if (sh == 0)
                for (int c = 0; c < NC; c++)
                    for (int q = 1; q < nsh; q++) acc[c] = acc[c] + ps[c * FFT_MT + threadIdx.x + q * cnt];
        }
        if (sh == 0)
            for (int c = 0; c < NC; c++) ys[c * 2 * nb + e] = acc[c];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < NC * 2 * nb; e += FFT_MT) {
        int c = e / (2 * nb), el = e % (2 * nb);
        int p = el / nb, idx = el % nb;
        cpx<T> v = ys[e];
        if ((contran >> c) & 1u) {
            int m, n;
            gt_mn(idx, L, m, n);
            int src = (m == 0) ? idx : aidx(-m, n, 0, L);
            v = ys[c * 2 * nb + p * nb + src];
            if (m & 1) v = mk(-v.x, -v.y);
        }
        cpx<T>* dst = y + (size_t)c * ld + a.offset[i] + el;
        *dst = *dst + v;
    }
}

// ---------------------------------------------------------------------------

void launch_fft_j(const FftJArgs& a, cudaStream_t st)
{
    fft_j_kernel<<<a.nsph, FFT_NT, 0, st>>>(a);
    launch_counter() += 1;
}
void launch_fft_hbuild(const FftHArgs& a, int nsm, cudaStream_t st)
{
    int nslot = 8 * a.cd[0] * a.cd[1] * a.cd[2];
    fft_hbuild_kernel<<<std::min(nslot, nsm * 8), FFT_NT, 0, st>>>(a);
    launch_counter() += 1;
}
void launch_fft_round(size_t n, const zd* in, float2* out, cudaStream_t st)
{
    fft_round_kernel<<<(int)std::min<size_t>((n + 255) / 256, 148 * 32), 256, 0, st>>>(n, in, out);
    launch_counter() += 1;
}
// f(number of columns as a constant), 1 .. 4
template <typename F> static void with_columns(int ncol, F f)
{
    switch (ncol) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    default: f(std::integral_constant<int, 4>()); break;
    }
}
template <typename T>
void launch_fft_s2n(const FftMArgs& a, const cpx<T>* J, const cpx<T>* x, int ld, int ncol, unsigned contran, cpx<T>* A, cudaStream_t st)
{
    const int smem = (int)sizeof(cpx<T>) * ncol * (2 * a.nbmax + FFT_MT);
    with_columns(ncol, [&](auto nc) {
        auto k = fft_s2n_kernel<T, decltype(nc)::value>;
        allow_smem(k, smem);
        k<<<a.nsph, FFT_MT, smem, st>>>(a, J, x, ld, contran, A);
    });
    launch_counter() += 1;
}
template <typename T> void launch_fft_mul(int nbN, size_t N8, int ncol, const float2* H, const cpx<T>* A, cpx<T>* G, cudaStream_t st)
{
    // rows a thread: as many as leave two CTAs' registers to an SM
    constexpr int R = sizeof(T) == 4 ? 8 : 4;
    const dim3 g((unsigned)((N8 + FFT_NT - 1) / FFT_NT), 2 * ((nbN + R - 1) / R));
    with_columns(ncol, [&](auto nc) { fft_mul_kernel<T, decltype(nc)::value, R><<<g, FFT_NT, 0, st>>>(nbN, N8, H, A, G); });
    launch_counter() += 1;
}
template <typename T>
void launch_fft_n2s(const FftMArgs& a, const cpx<T>* J, const cpx<T>* G, int ncol, unsigned contran, cpx<T>* y, int ld, cudaStream_t st)
{
    const int nbN = a.No * (a.No + 2), smem = (int)sizeof(cpx<T>) * ncol * (2 * nbN + 2 * a.nbmax + FFT_MT);
    with_columns(ncol, [&](auto nc) {
        auto k = fft_n2s_kernel<T, decltype(nc)::value>;
        allow_smem(k, smem);
        k<<<a.nsph, FFT_MT, smem, st>>>(a, J, G, contran, y, ld);
    });
    launch_counter() += 1;
}

template void launch_fft_s2n<double>(const FftMArgs&, const zd*, const zd*, int, int, unsigned, zd*, cudaStream_t);
template void launch_fft_s2n<float>(const FftMArgs&, const zf*, const zf*, int, int, unsigned, zf*, cudaStream_t);
template void launch_fft_mul<double>(int, size_t, int, const float2*, const zd*, zd*, cudaStream_t);
template void launch_fft_mul<float>(int, size_t, int, const float2*, const zf*, zf*, cudaStream_t);
template void launch_fft_n2s<double>(const FftMArgs&, const zd*, const zd*, int, unsigned, zd*, int, cudaStream_t);
template void launch_fft_n2s<float>(const FftMArgs&, const zf*, const zf*, int, unsigned, zf*, int, cudaStream_t);
