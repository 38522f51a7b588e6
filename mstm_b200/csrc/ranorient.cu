// ranorient.cu -- orientation-averaged scattering matrix from the cluster T
// matrix (ranorientscatmatrix, december2023/mstm-scatprops-26.f90:1963-2530,
// and ranorienscatmatrixcalc, :2538-2592), FP64 sums over the single-precision
// T matrix exactly as the reference keeps it after reading the T-matrix file.
//
//   ro_prep_kernel   complex(4) copy of T with the symmetric rows filled and
//                    the (beam-free) GB modification applied; per-order traces
//   ro_vc_kernel     vector-coupling rows of the bm contraction, one thread a row
//   ro_bm_kernel     one CTA per (w, v, n): the am / bm contractions in shared
//                    memory, bm(k, n(n+1)+m, p) to global memory
//   ro_dm_kernel     dm(u,ku,n,p,n1,p1) += sum over (w, v) of bm bm*, a batch of
//                    complex products over the items (w, v)
//   ro_coef_kernel   one CTA per (GSF degree w, n): fm, then the terms of n in
//                    aw/bw/cw/dw; ro_sum_kernel: the sums over n and the 16
//                    expansion coefficients sm(:,:,w), smcf(:,:,w)
//   ro_calc_kernel   one CTA per polar angle: generalised spherical functions
//                    by the rotcoef recurrence (kmax = 2) and the 16 elements
#include "common.cuh"
#include "ranorient.cuh"
#include "vcoupling.cuh"
#include "gsfrows.cuh"

namespace {

__device__ __forceinline__ zd ipw(int k)
{
    int e = ((k % 4) + 4) % 4;
    return (e == 0) ? mk(1.0, 0.0) : (e == 1 ? mk(0.0, 1.0) : (e == 2 ? mk(-1.0, 0.0) : mk(0.0, -1.0)));
}
__device__ __forceinline__ void atomic_addz(zd* p, zd v)
{
    atomicAdd(&p->x, v.x);
    atomicAdd(&p->y, v.y);
}
__device__ __forceinline__ zd up2(float2 a) { return mk((double)a.x, (double)a.y); }

}  // namespace

// tc(p,mn,q,kl) at ((2(mn-1)+p-1) + nblkt (2(kl-1)+q-1)), as float2
__global__ void ro_prep_kernel(int nodr, const zd* tmat, float2* tc)
{
    const int nblk = nodr * (nodr + 2), nblkt = 2 * nblk;
    // one thread per (p, mn, kl): the q = 1, 2 pair of the GB modification
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)2 * nblk * nblk; e += (size_t)gridDim.x * blockDim.x) {
        int row = (int)(e % nblkt), kl = (int)(e / nblkt) + 1;
        int mn = row / 2 + 1, p = row % 2 + 1;
        int n = 1;
        while (n * (n + 2) < mn) n++;
        int l = 1;
        while (l * (l + 2) < kl) l++;
        float2 v[2];
        for (int q = 1; q <= 2; q++) {
            zd t;
            if (n <= l) {
                t = tmat[(size_t)row + (size_t)nblkt * (2 * (kl - 1) + q - 1)];
            } else {
                int m = mn - n * (n + 1), k = kl - l * (l + 1);
                int srow = 2 * (l * (l + 1) - k - 1) + (q - 1), scol = 2 * (n * (n + 1) - m - 1) + (p - 1);
                zd s = tmat[(size_t)srow + (size_t)nblkt * scol];
                // the file reader copies the single-precision value times (-1)^(m+k)
                float sg = (float)pm1(m + k);
                t = mk((double)((float)s.x * sg), (double)((float)s.y * sg));
            }
            v[q - 1] = make_float2((float)t.x, (float)t.y);
        }
        // GB-modified T matrix without a beam: pp(l,1,1) = -i^(l+1) sqrt(2l+1)/2,
        // pp(l,2,1) = pp(l,1,2) = pp(l,2,2) = -pp(l,1,1); results stored in single precision
        zd pp11 = (-0.5 * sqrt((double)(l + l + 1))) * ipw(l + 1);
        zd pp21 = -pp11, pp12 = -pp11, pp22 = pp21;
        zd a = up2(v[0]);
        zd t1 = a * pp11 + up2(v[1]) * pp12;
        float2 n1 = make_float2((float)t1.x, (float)t1.y);
        zd t2 = a * pp21 + up2(v[1]) * pp22;
        float2 n2 = make_float2((float)t2.x, (float)t2.y);
        tc[(size_t)row + (size_t)nblkt * (2 * (kl - 1))] = n1;
        tc[(size_t)row + (size_t)nblkt * (2 * (kl - 1) + 1)] = n2;
    }
}

// trace(p,k,n) = sum_kt tc(p, n(n+1)+kt, k, n(n+1)+kt) in double (the coherent part)
__global__ void ro_trace_kernel(int nodr, const float2* tc, zd* trace)
{
    const int nblkt = 2 * nodr * (nodr + 2);
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 4 * nodr) return;
    int n = e / 4 + 1, k = (e / 2) % 2 + 1, p = e % 2 + 1;
    int nn1 = n * (n + 1);
    zd s = mk(0.0, 0.0);
    for (int kt = -n; kt <= n; kt++) {
        int mn = nn1 + kt;
        s = s + up2(tc[(size_t)(2 * (mn - 1) + p - 1) + (size_t)nblkt * (2 * (mn - 1) + k - 1)]);
    }
    trace[e] = s;
}

// The big loop of ranorientscatmatrix runs over items (w, v), item = w w + w + v,
// in chunks [i0, i1) whose bm fit the buffer a.bg:
//   bg[ik][u + nodr + 1][item - i0][2 (n-1) + p - 1],   m = u -+ 1 for ik = 0, 1
// (zero where |m| > n); the coherent part, v = 0 only, in bcf with w as the item.
__device__ __forceinline__ int item_w(int item)
{
    int w = (int)sqrtf((float)item);
    while (w * w > item) w--;
    while ((w + 1) * (w + 1) <= item) w++;
    return w;
}

// vcfunc(-u,w,m,n)(0 .. w+n), u = m -+ 1, for w = w0 .. w0 + nw - 1, |m| <= n
// <= nodr: they do not depend on v, which the CTAs of (w, v, n) share them over
__global__ void __launch_bounds__(64) ro_vc_kernel(RoArgs a, int w0, int nw)
{
    const int nodr = a.nodr, nm = 2 * nodr + 1, VL = 3 * nodr + 2;
    const int e = blockIdx.x * 64 + threadIdx.x;
    if (e >= nw * nodr * nm * 2) return;
    const int k = e % 2, m = (e / 2) % nm - nodr, n = (e / (2 * nm)) % nodr + 1, w = w0 + e / (2 * nm * nodr);
    const int u = m - (2 * k - 1);
    if (m < -n || m > n || u < -w || u > w) return;
    vc_func(VCTab{a.bcof, a.fnr, a.nbc}, -u, w, m, n, a.vtab + (size_t)e * VL);
}

__global__ void __launch_bounds__(RO_NT) ro_bm_kernel(RoArgs a, int i0, int ni)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nodr = a.nodr, nblkt = 2 * nodr * (nodr + 2), nm = 2 * nodr + 1, VL = 3 * nodr + 2, tid = threadIdx.x;
    zd* am = reinterpret_cast<zd*>(smraw);                       // am(k,l,p): 2 x nodr x 2
    zd* amcf = am + 4 * nodr;                                    // amcf(k,n,p): 2 x 2
    double* vct = reinterpret_cast<double*>(amcf + 4);           // rows of vcfunc(v,w,-t,n)
    // the longest n first: they share the grid's last wave with short ones
    const int n = nodr - (int)(blockIdx.x / ni), it = blockIdx.x % ni, item = i0 + it;
    const int W = item_w(item), v = item - W * W - W, nn1 = n * (n + 1);
    const int lmin = max(1, abs(W - n)), lmax = min(nodr, W + n);
#define TCG(p, mn, q, kl) up2(a.tc[(size_t)(2 * ((mn) - 1) + (p) - 1) + (size_t)nblkt * (2 * ((kl) - 1) + (q) - 1)])
    if (lmin <= lmax) {
        for (int t = -n + tid; t <= n; t += RO_NT) vc_func(VCTab{a.bcof, a.fnr, a.nbc}, v, W, -t, n, vct + (size_t)(t + n) * VL);
        __syncthreads();
        // am(k,l,p) = sum_t vc(l) tc(p, n(n+1)+t, k, l(l+1)+t-v)
        for (int e = tid; e < 4 * (lmax - lmin + 1); e += RO_NT) {
            const int p = e % 2 + 1, k = (e / 2) % 2 + 1, l = lmin + e / 4;
            zd s = mk(0.0, 0.0);
#pragma unroll 4
            for (int t = max(-n, v - l); t <= min(n, v + l); t++) {
                const double vcl = vct[(size_t)(t + n) * VL + l];
                s = s + vcl * TCG(p, nn1 + t, k, l * (l + 1) + t - v);
            }
            am[(k - 1) + 2 * ((p - 1) + 2 * (l - 1))] = s;
        }
        if (v == 0 && tid < 4) {
            zd sc = mk(0.0, 0.0);
            const int k = tid / 2, p = tid % 2;
            if (n >= lmin && n <= lmax)
                for (int t = -n; t <= n; t++) {
                    const zd tv = vct[(size_t)(t + n) * VL + n] * a.trace[4 * (n - 1) + 2 * k + p];
                    sc = sc + mk(tv.x / (double)(n + n + 1), tv.y / (double)(n + n + 1));
                }
            amcf[k + 2 * p] = sc;
        }
        __syncthreads();
    }
#undef TCG
    // bm(k, n(n+1)+m, p) = sum_l am(k,l,p) fl(l), fl = -(-1)^l vcfunc(-u,w,m,n)(l)/(2l+1)
    const int umax = min(W, nodr + 1), nu = 2 * umax + 1;
    const double* vt = a.vtab + (size_t)(W - a.vw0) * nodr * nm * 2 * VL;
    for (int e = tid; e < 4 * nu; e += RO_NT) {
        const int p = e % 2, k = (e / 2) % 2, u = e / 4 - umax, m = u + 2 * k - 1;
        zd s = mk(0.0, 0.0), sc = mk(0.0, 0.0);
        if (m >= -n && m <= n && lmin <= lmax) {
            const double* vr = vt + (size_t)(((n - 1) * nm + m + nodr) * 2 + k) * VL;
            for (int l = lmin; l <= lmax; l++) {
                const double fl = -pm1(l) * vr[l] / (double)(l + l + 1);
                s = s + am[k + 2 * (p + 2 * (l - 1))] * fl;
            }
            if (v == 0 && n >= lmin && n <= lmax) sc = amcf[k + 2 * p] * (-pm1(n) * vr[n] / (double)(n + n + 1));
        }
        const size_t row = (size_t)k * (2 * nodr + 3) + u + nodr + 1;
        a.bg[(row * a.bgi + it) * (2 * nodr) + 2 * (n - 1) + p] = s;
        if (v == 0) a.bcf[(row * (2 * nodr + 1) + W) * (2 * nodr) + 2 * (n - 1) + p] = sc;
    }
}

// dm(u,ku,n,p,n1,p1) += sum_items (2w+1) bm(ik,nu,p) i^(n-n1) fl conj(bm(ik1,nu1,p1)):
// per (u, ku) one complex product of 2 nodr x 2 nodr over the items with
// w >= |u|, in tiles of RO_TILE x RO_TILE, RO_KC items of a tile in shared
// memory at a time, a share of the items (blockIdx.z) a CTA and its sums added
// with FP64 atomics.  FP64-rate bound: 16 multiply-adds for every four 16-byte
// shared loads of a thread (2 x 2 outputs).  With a CTA per item adding every
// product to dm by its own atomics the loop took 32.6 ms for order 28; now 3.8
// ms, 2.4 of them the contractions of ro_bm_kernel.
#define RO_TILE 32
#define RO_KC 16
template <bool COH>
__global__ void __launch_bounds__(256) ro_dm_kernel(RoArgs a, int i0, int ni)
{
    __shared__ zd sa[RO_KC][RO_TILE], sb[RO_KC][RO_TILE];
    const int nodr = a.nodr, M = 2 * nodr, tid = threadIdx.x;
    const int u = (int)blockIdx.x / 3 - (nodr + 1), ku = blockIdx.x % 3;
    const int k = (ku == 0) ? 0 : 1, k1 = (ku == 1) ? 1 : 0;   // ik, ik1 less one
    const int nt = (M + RO_TILE - 1) / RO_TILE, r0 = (blockIdx.y / nt) * RO_TILE, c0 = (blockIdx.y % nt) * RO_TILE;
    const int stride = COH ? 2 * nodr + 1 : a.bgi;
    const zd* src = COH ? a.bcf : a.bg;
    const zd* A = src + ((size_t)k * (2 * nodr + 3) + u + nodr + 1) * stride * M;
    const zd* B = src + ((size_t)k1 * (2 * nodr + 3) + u + nodr + 1) * stride * M;
    // items of this chunk with w >= |u|, this CTA's share
    const int au = abs(u);
    const int first = max(0, (COH ? au : au * au) - i0);
    const int per = ((ni - first + (int)gridDim.z - 1) / (int)gridDim.z + RO_KC - 1) / RO_KC * RO_KC;
    const int ib = first + (int)blockIdx.z * per, ie = min(ni, ib + per);
    if (ib >= ie) return;
    zd acc[2][2];
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++) acc[i][j] = mk(0.0, 0.0);
    const int tr = tid / 16, tc = tid % 16;
    for (int i = ib; i < ie; i += RO_KC) {
        for (int e = tid; e < RO_KC * RO_TILE; e += 256) {
            const int kk = e / RO_TILE, x = e % RO_TILE;
            zd va = mk(0.0, 0.0), vb = mk(0.0, 0.0);
            if (i + kk < ie) {
                const int w = COH ? i + kk + i0 : item_w(i + kk + i0);
                if (r0 + x < M) va = (double)(w + w + 1) * A[(size_t)(i + kk) * M + r0 + x];
                if (c0 + x < M) vb = B[(size_t)(i + kk) * M + c0 + x];
            }
            sa[kk][x] = va;
            sb[kk][x] = vb;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < RO_KC; kk++) {
            const zd a0 = sa[kk][tr], a1 = sa[kk][tr + 16], b0 = cj(sb[kk][tc]), b1 = cj(sb[kk][tc + 16]);
            acc[0][0] = acc[0][0] + a0 * b0;
            acc[0][1] = acc[0][1] + a0 * b1;
            acc[1][0] = acc[1][0] + a1 * b0;
            acc[1][1] = acc[1][1] + a1 * b1;
        }
        __syncthreads();
    }
    zd* dm = (COH ? a.dmcf : a.dm) + (size_t)blockIdx.x * M * M;
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++) {
            const int r = r0 + tr + 16 * i, c = c0 + tc + 16 * j;
            if (r >= M || c >= M) continue;
            const int n = r / 2 + 1, n1 = c / 2 + 1;
            const double fl = -a.fnr[n + n + 1] * a.fnr[n1 + n1 + 1];
            atomic_addz(&dm[(size_t)r * M + c], ipw(n - n1) * (acc[i][j] * fl));
        }
}

// The terms of degree n in the expansion coefficients of degree w, one CTA per
// (w, n).  fm(ik,n,p,n1,p1) = sum_u dm fl by a thread per (ik, p, n1, p1) and
// part (0: all, 1: coherent), the vcfunc(m,n,0,w) and (m,n,-2,w) rows once in
// shared memory for every u and n1; then the 12 sums of fm that the
// coefficients take, a warp each, to a.part[part][w][n][12] in the order
//   aw(0,-1) aw(0,1) bw(0,-1) bw(0,1) aw(2,0) bw(2,0) aw(2,-1) aw(2,1) bw(2,-1) bw(2,1) cw dw
// One CTA per w with a vcfunc per (ik, n, n1, u) and the sums on one thread
// took 26.4 ms for order 28; now below 0.7 ms.
#define RO_CT 256
__global__ void __launch_bounds__(RO_CT) ro_coef_kernel(RoArgs a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nodr = a.nodr, M = 2 * nodr, tid = threadIdx.x, VL = 3 * nodr + 2;
    const int n = nodr - (int)blockIdx.x, w = 2 * nodr - (int)blockIdx.y;
    const int n1s = max(1, abs(n - w)), n1e = min(nodr, n + w);
    zd* part = a.part + ((size_t)w * nodr + n - 1) * 24;
    if (n1s > n1e) {
        if (tid < 24) part[tid] = mk(0.0, 0.0);
        return;
    }
    const int nf = 6 * M;                                   // (ik, p, n1, p1) of one part
    zd* f = reinterpret_cast<zd*>(smraw);                   // nf
    double* vc = reinterpret_cast<double*>(f + nf);         // [type][m + n][0 .. n + w]
    for (int e = tid; e < 2 * (2 * n + 1); e += RO_CT) {
        const int m = e % (2 * n + 1) - n, type = e / (2 * n + 1);
        if (type == 0 || w >= 2) vc_func(VCTab{a.bcof, a.fnr, a.nbc}, m, n, -2 * type, w, vc + (size_t)e * VL);
    }
    const double* vc1[2] = {vc + (size_t)(n + 1) * VL, vc + (size_t)(2 * n + 1 + n + 1) * VL};   // m = 1
    const int lane = tid & 31, warp = tid >> 5;
    for (int pt = 0; pt < 2; pt++) {
        const zd* dm = pt ? a.dmcf : a.dm;
        __syncthreads();
        for (int e = tid; e < nf; e += RO_CT) {
            const int c = e % M, p = (e / M) % 2, ik = e / (2 * M), n1 = c / 2 + 1;
            zd s = mk(0.0, 0.0);
            if (n1 >= n1s && n1 <= n1e && (ik < 2 || w >= 2)) {
                // m = u -+ 1 (ik 0, 1); m = u + 1 and m1 = u - 1 (ik 2)
                const int lim = min(n, n1);
                int ulo, uhi;
                if (ik < 2) {
                    ulo = -lim - (2 * ik - 1);
                    uhi = lim - (2 * ik - 1);
                } else {
                    ulo = max(-n - 1, -n1 + 1);
                    uhi = min(n - 1, n1 + 1);
                }
                const double* vr = vc + (ik < 2 ? (size_t)(n + 2 * ik - 1) * VL : (size_t)(2 * n + 1 + n + 1) * VL) + n1;
                const zd* d = dm + ((size_t)(nodr + 1) * 3 + ik) * M * M + (size_t)(2 * (n - 1) + p) * M + c;
#pragma unroll 4
                for (int u = ulo; u <= uhi; u++) s = s + d[(long long)u * 3 * M * M] * vr[u * VL];
                s = s * (-pm1(n) * a.fnr[w + w + 1] / a.fnr[n1 + n1 + 1]);
            }
            f[e] = s;
        }
        __syncthreads();
        for (int o = warp; o < 12; o += RO_CT / 32) {
            // which (ik, same-or-other p1, vcfunc type) this sum takes
            static const signed char ikof[12] = {0, 1, 0, 1, 2, 2, 0, 1, 0, 1, 2, 2};
            static const signed char oth[12] = {0, 0, 1, 1, 0, 1, 0, 0, 1, 1, -1, -1};
            const int ik = ikof[o], ot = oth[o], type = o >= 6;
            zd s = mk(0.0, 0.0);
            if (type == 0 || w >= 2)
                for (int e = lane; e < 2 * M; e += 32) {
                    const int c = e % M, p = e / M + 1, n1 = c / 2 + 1, p1 = c % 2 + 1;
                    if (n1 < n1s || n1 > n1e) continue;
                    const int same = ((n + n1 - w) % 2 == 0) == (p1 == p);   // p1 is the partner of p
                    if (ot >= 0 && same == ot) continue;
                    const double v = vc1[type][n1];
                    double fl = 2.0 * (o == 11 ? pm1(n1 + w) : pm1(n)) * v * a.fnr[w + w + 1] / a.fnr[n1 + n1 + 1];
                    if (type) fl = fl * (o == 11 ? pm1(p) : pm1(p1));
                    s = s + f[(size_t)ik * 2 * M + e] * fl;
                }
            for (int x = 16; x > 0; x >>= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, x);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, x);
            }
            if (lane == 0) part[12 * pt + o] = s;
        }
    }
}

// expansion coefficients of degree w: the sums over n, one CTA of 32 threads per w
__global__ void ro_sum_kernel(RoArgs a)
{
    __shared__ zd t[24];
    const int nodr = a.nodr, w = blockIdx.x;
    if (threadIdx.x < 24) {
        zd s = mk(0.0, 0.0);
        for (int n = 1; n <= nodr; n++) s = s + a.part[((size_t)w * nodr + n - 1) * 24 + threadIdx.x];
        t[threadIdx.x] = s;
    }
    __syncwarp();
    if (threadIdx.x >= 2) return;
    const int c = threadIdx.x;
    const zd* q = t + 12 * c;
    const zd a0m = q[0], a0p = q[1], b0m = q[2], b0p = q[3], a20 = q[4], b20 = q[5], a2m = q[6], a2p = q[7], b2m = q[8], b2p = q[9],
             cw = q[10], dw = q[11];
    double* o = (c ? a.smcf : a.sm) + 16 * w;
#define SMO(i, j) o[((i) - 1) + 4 * ((j) - 1)]
    for (int e = 0; e < 16; e++) o[e] = 0.0;
    SMO(1, 1) = (a0m + a0p).x;
    SMO(1, 2) = (a2m + a2p).x;
    SMO(1, 3) = 2.0 * a20.y;
    SMO(1, 4) = (a0p - a0m).x;
    SMO(2, 2) = dw.x;
    SMO(2, 3) = dw.y;
    SMO(2, 4) = (a2p - a2m).x;
    SMO(3, 1) = -(b2m + b2p).y;
    SMO(3, 2) = cw.y;
    SMO(3, 3) = cw.x;
    SMO(3, 4) = (b2m - b2p).y;
    SMO(4, 1) = (b0m + b0p).x;
    SMO(4, 2) = 2.0 * b20.x;
    SMO(4, 4) = (b0p - b0m).x;
    for (int e = 0; e < 16; e++) o[e] = o[e] / a.rimed_re / 2.0;
#undef SMO
}

// ranorienscatmatrixcalc at theta_i = i pi/(nang-1) (pi as the reference stores it)
__global__ void __launch_bounds__(GSF_NT) ro_calc_kernel(int nmax, int nang, const double* smc, const double* fnr, const double* bcofd,
                                                         double* smat)
{
    extern __shared__ __align__(16) double gsf_smem[];
    const int ia = blockIdx.x;
    if (ia >= nang) return;
    const double ct = cos((double)ia * MSTMG_REF_PI / (double)(nang - 1));
    gsf_columns(nmax, ct, fnr, bcofd, gsf_smem);
    // a warp per element of the upper set, lanes over the degrees
    __shared__ double so[16];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#define SC(i, j, n) smc[((i) - 1) + 4 * ((j) - 1) + 16 * (n)]
    for (int el = warp; el < 16; el += GSF_NT / 32) {
        const int i = el % 4 + 1, j = el / 4 + 1;
        double v = 0.0;
        for (int n = lane; n <= nmax; n += 32) {
            const double* g = gsf_smem + GSF_ROW * n;
            const double d00 = n ? g[GSF_D00] : 1.0;   // degree 0: dc(0,0) = 1
            if ((i == 1 || i == 4) && (j == 1 || j == 4)) v += d00 * SC(i, j, n);
            if (n < 2) continue;
            // dc(k, n(n+1)+m) of rotcoef(ct, 2, nodrexp) is the table's (k, m)
            const double d20 = g[GSF_D20], d2m = g[GSF_D2M], d2p = g[GSF_D22];
            if ((i == 1 && (j == 2 || j == 3)) || (i == 2 && j == 4) || (i == 3 && j == 4) || (i == 4 && j == 2)) v += d20 * SC(i, j, n);
            if (i == 2 && j == 2) v += d2m * SC(2, 2, n) + d2p * SC(3, 3, n);
            if (i == 2 && j == 3) v += d2p * SC(2, 3, n) + d2p * SC(3, 2, n);
            if (i == 3 && j == 3) v += -d2m * SC(2, 2, n) + d2p * SC(3, 3, n);
            if (i == 3 && j == 2) v += d2p * SC(2, 3, n) - d2p * SC(3, 2, n);
        }
        for (int x = 16; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
        if (lane == 0) so[el] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#define SO(i, j) so[((i) - 1) + 4 * ((j) - 1)]
        // as the reference writes it: each degree starts from the new (1,3)
        SO(3, 1) = nmax >= 2 ? SO(1, 3) + gsf_smem[GSF_ROW * nmax + GSF_D20] * SC(3, 1, nmax) : 0.0;
        SO(2, 1) = SO(1, 2);
        SO(4, 3) = -SO(3, 4);
#undef SO
        for (int e = 0; e < 16; e++) smat[16 * (size_t)ia + e] = so[e];
    }
#undef SC
}

// items from i0 on whose bm and vector-coupling rows fit the buffers; nodr
// bounds both so that a handful of launches cover the loop and the buffers
// stay near the size of L2
static int ro_chunk_end(int nodr, int i0)
{
    const int nitems = (2 * nodr + 1) * (2 * nodr + 1);
    const size_t bgb = sizeof(zd) * 2 * (2 * (size_t)nodr + 3) * 2 * nodr, vcb = ro_vtab_w(nodr) * sizeof(double);
    int w0 = 0;
    while ((w0 + 1) * (w0 + 1) <= i0) w0++;
    const int nw = (int)std::max<size_t>(1, ((size_t)32 << 20) / vcb);
    const long long wend = (long long)(w0 + nw) * (w0 + nw);
    return (int)std::min<long long>({(long long)nitems, wend, i0 + std::max<long long>(1, ((64LL << 20) / (long long)bgb))});
}
size_t ro_vtab_w(int nodr) { return (size_t)nodr * (2 * nodr + 1) * 2 * (3 * nodr + 2); }
RoSizes ro_sizes(int nodr)
{
    RoSizes z{0, 0, 0, 0, 0};
    const int nitems = (2 * nodr + 1) * (2 * nodr + 1);
    for (int i0 = 0; i0 < nitems;) {
        const int i1 = ro_chunk_end(nodr, i0);
        int w0 = 0, w1 = 0;
        while ((w0 + 1) * (w0 + 1) <= i0) w0++;
        while ((w1 + 1) * (w1 + 1) <= i1 - 1) w1++;
        z.bgi = std::max(z.bgi, i1 - i0);
        z.vtab = std::max(z.vtab, ro_vtab_w(nodr) * (w1 - w0 + 1));
        i0 = i1;
    }
    z.bg = 2 * (2 * (size_t)nodr + 3) * z.bgi * 2 * nodr;
    z.bcf = 2 * (2 * (size_t)nodr + 3) * (2 * nodr + 1) * 2 * nodr;
    z.part = 24 * (size_t)nodr * (2 * nodr + 1);
    return z;
}
size_t ro_dm_elems(int nodr) { return (size_t)(2 * nodr + 3) * 3 * nodr * 2 * nodr * 2; }

int launch_ranorient(const RoArgs& args, const zd* tmat, int nang, const double* bcofd, double* smat, int nsm, cudaStream_t st)
{
    RoArgs a = args;
    const int nodr = a.nodr;
    if (nodr > RO_ORDER_MAX) return -1;
    size_t nblk = (size_t)nodr * (nodr + 2);
    int g = (int)std::min<size_t>((2 * nblk * nblk + 255) / 256, (size_t)nsm * 16);
    ro_prep_kernel<<<g, 256, 0, st>>>(nodr, tmat, a.tc);
    ro_trace_kernel<<<(4 * nodr + 63) / 64, 64, 0, st>>>(nodr, a.tc, a.trace);
    launch_counter() += 2;
    const int VL = 3 * nodr + 2, nitems = (2 * nodr + 1) * (2 * nodr + 1), nt = (2 * nodr + RO_TILE - 1) / RO_TILE;
    const int nu3 = 3 * (2 * nodr + 3);
    const size_t sm_bm = sizeof(zd) * (4 * nodr + 4) + sizeof(double) * (2 * nodr + 1) * VL;
    const size_t sm_co = sizeof(zd) * 12 * nodr + sizeof(double) * 2 * (2 * nodr + 1) * VL;
    allow_smem(ro_bm_kernel, sm_bm);
    allow_smem(ro_coef_kernel, sm_co);
    for (int i0 = 0; i0 < nitems;) {
        const int i1 = ro_chunk_end(nodr, i0), ni = i1 - i0;
        int w0 = 0, w1 = 0;
        while ((w0 + 1) * (w0 + 1) <= i0) w0++;
        while ((w1 + 1) * (w1 + 1) <= i1 - 1) w1++;
        a.vw0 = w0;
        const int rows = (w1 - w0 + 1) * nodr * (2 * nodr + 1) * 2;
        ro_vc_kernel<<<(rows + 63) / 64, 64, 0, st>>>(a, w0, w1 - w0 + 1);
        ro_bm_kernel<<<nodr * ni, RO_NT, sm_bm, st>>>(a, i0, ni);
        // two waves of CTAs where the items allow it
        const int z = std::max(1, std::min(ni / (4 * RO_KC), (8 * nsm + nu3 * nt * nt - 1) / (nu3 * nt * nt)));
        ro_dm_kernel<false><<<dim3(nu3, nt * nt, z), 256, 0, st>>>(a, i0, ni);
        launch_counter() += 3;
        i0 = i1;
    }
    ro_dm_kernel<true><<<dim3(nu3, nt * nt, 1), 256, 0, st>>>(a, 0, 2 * nodr + 1);
    ro_coef_kernel<<<dim3(nodr, 2 * nodr + 1), RO_CT, sm_co, st>>>(a);
    ro_sum_kernel<<<2 * nodr + 1, 32, 0, st>>>(a);
    if (nang > 1) ro_calc_kernel<<<nang, GSF_NT, gsf_smem_bytes(2 * nodr), st>>>(2 * nodr, nang, a.sm, a.fnr, bcofd, smat);
    launch_counter() += (nang > 1) ? 4 : 3;
    return 0;
}
