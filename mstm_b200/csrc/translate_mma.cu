// translate_mma.cu -- the pair translation pass (MSTM's
// external_to_external_expansion, december2023/mstm-modules-33.f90:6390-6525,
// applying coefficient_translation, modules:6610-6787, in both directions of
// every pair) on the FP64 tensor cores, for spheres of any orders.
//
// Per pair and direction: shift and phase e^{i m phi}, rotation of every
// degree n by the folded Wigner blocks E_n, O_n, axial translation of every
// degree m by Z_m, rotation back, phase and shift.  The products are small
// dense blocks applied to 8 complex columns (direction x mode x right-hand
// side), i.e. to an MMA's 8 columns of real parts and 8 of imaginary parts:
//   A+B  [P; Q](k) = [E_n s; O_n t](k), s and t formed from the sources in
//        registers as the B operand; a'(k) = P + Q, a'(-k) = (-1)^k (P - Q)
//   C    g = Z_m a' (Z_m^T for i -> j), columns (re, im) of 4 complex ones,
//        both modes' blocks in one unit, which leaves g(m) and g(-m) of a
//        column in one lane: s' = g(m) + (-1)^m g(-m), t' = g(m) - (-1)^m g(-m)
//   D    the rotation back, E_n^T s' and O_n^T t', phase, shift, added to
//        the tile's outputs in shared memory
// with m8n8k4 FP64 MMAs: one instruction does 256 multiply-adds where the
// scalar kernels issued one per lane.  Blocks of 1 or 2 x 8 rows and 4-deep
// products pad the work about twofold (352 MMAs a pair at order 9).
//
// What bounds it: the latency of a pair's chain of dependent phases.  Of the
// 2.7k cycles a pair takes an SM at order 9 the FP64 tensor pipe is busy 50 %,
// the scalar FP64 pipe 12 %, shared memory 68 %; HBM (17 KB of operators a
// pair) gives 1.7 TB/s.  Choices that measured (500 spheres of order 9, 2
// columns, FP64, each against the kernel of its day):
//   * straight code per warp over units dealt at compile time, few warps a
//     CTA and several CTAs per SM, against unit loops with index arithmetic
//     at run time: 6.2k -> 4.2k instructions a pair;
//   * a copying warp that issues the copies and adds finished tiles to y by
//     bulk reductions (cp.reduce.async.bulk), against thread 0 of a computing
//     warp and atomics by all threads: 1603 -> 1363 us;
//   * tiles of one pair of spheres at order 9 and above (2 x 2 spheres up to
//     8, 4 x 4 up to 4): the outputs of a 4 x 4 tile in shared memory would
//     halve the resident CTAs: 1358 -> 1172 us.
// The scalar kernels it replaced took 2920 us (FP64) and 1385 us (FP32).
//
// A CTA works through whole tiles: the pairs between two groups of up to 4
// spheres (host: TileSet).  Operators and sources stream in one pair ahead
// (cp.async.bulk, mbarriers, bounded waits), each part into the place its
// predecessor has left; outputs of the tile's spheres accumulate in shared
// memory and are added to y once per tile.  Two work buffers alternate:
// sources / a' / (s', t') of a pair use buffers b, 1 - b, b, and the next
// pair's sources go to 1 - b once C is done.  Rows of a' and of (s', t') are 8
// columns of 16 bytes, their columns XORed by functions of degree and order
// so that the 8 lanes of an access phase fall on different banks.
//
// FP32 passes run the same kernel, their columns widened before and rounded
// after: FP64 records, products and sums.
//
// A wait that runs out ends the whole CTA: the warp, which waits as one, leaves
// a word in shared memory and returns; the copying warp looks for it behind
// phase B's barrier, before it arms that phase's barriers again, and before it
// adds a tile to y; it then issues no more copies, makes the step the last one,
// waits (bounded) for the copies in flight, sets *err to MSTMG_ERR_CUDA and
// leaves the tile out of y.  (500 spheres of order 9, 2 columns: 1174 -> 1202
// us, up to 2 % of a pass at other orders; a vote of the CTA in its barriers
// took 5 %, waits by the copying warp alone 6 %.)
//
// Clusters of one order (3 .. 10) have instances with that order and the
// units of every warp at compile time; other tiles (mixed or larger orders)
// run the instances with orders at run time (LC = 0).
#include "common.cuh"
#include "kernels.cuh"
#include "oplayout.cuh"
#include "pairpipe.cuh"
#include "translate_mma.cuh"
#include <algorithm>
#include <type_traits>
#include <utility>
#include <vector>

using namespace pairpipe;

namespace {

constexpr int MMA_PAD = 4;      // zero values after the records: what the last row of a block may read past it
constexpr int MMA_HEAD = 384;   // bytes of barriers, step ring, offset tables and a zero value

__device__ __forceinline__ void mma884(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
// with first: c = a b
__device__ __forceinline__ void mma884(double (&c)[2], double a, double b, bool first)
{
    if (first)
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};" : "=d"(c[0]), "=d"(c[1]) : "d"(a), "d"(b), "d"(0.0));
    else
        mma884(c, a, b);
}
// v or -v by the lowest bit of s, off the FP64 pipe
__device__ __forceinline__ double flip(double v, int s)
{
    return __hiloint2double(__double2hiint(v) ^ (s << 31), __double2loint(v));
}
__device__ __forceinline__ zd ldx(const zd* p)
{
    const double2 v = *reinterpret_cast<const double2*>(p);
    return mk(v.x, v.y);
}
__device__ __forceinline__ void sto(unsigned char* sm, int off, zd v) { *reinterpret_cast<double2*>(sm + off) = make_double2(v.x, v.y); }
__device__ __forceinline__ void stx(zd* p, zd v) { *reinterpret_cast<double2*>(p) = make_double2(v.x, v.y); }

// Rows of a' (order k, degree n; the degrees of one order consecutive) start
// at abase(k) + n; rows of s', t' (degree n, order m; the orders of one
// degree consecutive), t' after s'.  abase: k = 0, then 1, -1, 2, -2, ...
__host__ __device__ constexpr int abase(int k, int L)
{
    const int m = k < 0 ? -k : k;
    return m ? L + (m - 1) * (2 * L + 2 - m) + (k < 0 ? L + 1 - m : 0) - m : -1;
}
__device__ __forceinline__ int acol(int n, int k, int col) { return col ^ (n & 3) ^ ((k & 1) << 2); }
__host__ __device__ constexpr int srow(int n, int m) { return (n - 1) * (n + 2) / 2 + m; }
__host__ __device__ constexpr int trow(int n, int m) { return (n - 1) * n / 2 + m - 1; }
__device__ __forceinline__ int scol(int n, int m, int col) { return col ^ (m & 3) ^ ((n & 1) << 2); }

// barrier of the CTA, from the copying warp's code and the others'
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 0;" ::: "memory"); }
// bounded wait of a whole warp.  With the first poll before the loop the
// compiler orders what follows it otherwise: passes of orders up to 6 and of
// mixed orders are 1 to 5 % faster, those of orders 7 to 10 2 to 4 % slower.
template <int LC> __device__ __forceinline__ bool mb_wait_warp(uint64_t* bar, uint32_t parity)
{
    if constexpr (LC < 7) {
        bool in = __all_sync(0xffffffffu, mb_try(bar, parity));
        for (int it = 1; !in && it < WAIT_POLLS; ++it) in = __all_sync(0xffffffffu, mb_try(bar, parity));
        return in;
    } else {
        for (int it = 0; it < WAIT_POLLS; ++it)
            if (__all_sync(0xffffffffu, mb_try(bar, parity))) return true;
        return false;
    }
}
// y[] += shared values, `bytes` long, by one bulk reduction
__device__ __forceinline__ void bulk_add(void* dst, const void* src, uint32_t bytes)
{
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst), "r"(su32(src)), "r"(bytes) : "memory");
}

template <int V> struct IntC { static constexpr int value = V; };

// The units of a pair of one order L, dealt to NW warps at compile time (each
// warp runs straight code over its own units): the rotation of a degree n, the
// axial translation of an order m (both directions), in descending order of
// MMAs, each to the warp with the least so far.
template <int L, int NW> struct Deal {
    int nrot[NW] = {}, rot[NW][8] = {}, nax[NW] = {}, ax[NW][8] = {};
    int ofs[NW][8] = {}, steps = 0;   // a rotation unit's first step of 4 orders among its warp's; the most of a warp
    constexpr Deal()
    {
        int cost[64] = {}, code[64] = {}, k = 0, load[NW] = {};
        for (int n = 1; n <= L; n++) {
            cost[k] = (4 * (n / 4 + 1) + 6) * (n / 8 + 1);
            code[k++] = n;
        }
        give(k, cost, code, load, nrot, rot);
        for (int w = 0; w < NW; w++) {
            load[w] = 0;
            int o = 0;
            for (int i = 0; i < nrot[w]; i++) {
                ofs[w][i] = o;
                o += (rot[w][i] / 4 + 1) * (rot[w][i] / 8 + 1);
            }
            if (o > steps) steps = o;
        }
        k = 0;
        for (int m = 0; m <= L; m++) {
            const int j = L - (m ? m : 1) + 1;
            cost[k] = ((m ? 8 : 4) * ((j + 3) / 4) + 6) * ((j + 7) / 8);
            code[k++] = m;
        }
        give(k, cost, code, load, nax, ax);
    }
    static constexpr void give(int k, int* cost, int* code, int* load, int* num, int (*out)[8])
    {
        for (int q = 0; q < k; q++) {
            int b = 0, w = 0;
            for (int i = 1; i < k; i++)
                if (cost[i] > cost[b]) b = i;
            for (int i = 1; i < NW; i++)
                if (load[i] < load[w]) w = i;
            out[w][num[w]++] = code[b];
            load[w] += cost[b];
            cost[b] = -1;
        }
    }
};
template <int L, int NW> constexpr Deal<L, NW> kDeal{};

// f(IntC<u>) for the rotation (axial) units u of warp w
template <int L, int NW, int W, typename F, size_t... I> __device__ __forceinline__ void rot_units(F&& f, std::index_sequence<I...>)
{
    (f(IntC<kDeal<L, NW>.rot[W][I]>{}, IntC<kDeal<L, NW>.ofs[W][I]>{}), ...);
}
template <int L, int NW, int W, typename F, size_t... I> __device__ __forceinline__ void ax_units(F&& f, std::index_sequence<I...>)
{
    (f(IntC<kDeal<L, NW>.ax[W][I]>{}), ...);
}
template <int L, int NW, bool AX, int W = 0, typename F> __device__ __forceinline__ void warp_units(int warp, F&& f)
{
    if constexpr (W < NW) {
        if (warp == W) {
            if constexpr (AX) ax_units<L, NW, W>(f, std::make_index_sequence<kDeal<L, NW>.nax[W]>{});
            else rot_units<L, NW, W>(f, std::make_index_sequence<kDeal<L, NW>.nrot[W]>{});
        } else {
            warp_units<L, NW, AX, W + 1>(warp, f);
        }
    }
}


struct Step {
    int offi, offj;
    unsigned lls;   // 0: no step
    unsigned rec4;
    int row, chunk, cols, last;
};

}  // namespace

// LC: the order of every pair, or 0: orders by pair
template <int LC, int NW, int MINB> __global__ void __launch_bounds__((NW + 1) * 32, MINB) translate_mma_kernel(const __grid_constant__ MmaArgs a)
{
    extern __shared__ __align__(128) unsigned char sm[];
    // uniform orders: [0] rotation blocks, [1], [2] axial blocks of even and odd
    // steps, [SRC] sources; else [0], [1] operators, [2] sources.  Up to order 7
    // rotation blocks and sources share [0] (one wait a pair less: 1 to 2 % of
    // a pass at orders 5 to 7, but 2 % more at 8 and 9).
    constexpr int SRC = LC == 0 ? 2 : LC < 8 ? 0 : 3;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm);
    volatile int* gave_up = reinterpret_cast<int*>(sm + 32);      // a wait ran out
    Step* ring = reinterpret_cast<Step*>(sm + 48);                // 4 steps
    int* roff = reinterpret_cast<int*>(sm + 48 + 4 * sizeof(Step));   // per degree: E_n in the record
    int* zoff = roff + MSTMG_LMAX + 2;                            // per order: Z_m in the record
    double* recb = reinterpret_cast<double*>(sm + MMA_HEAD);      // the 16 bytes before are zero
    const int boff = (MMA_HEAD + (LC ? a.maxrec + op_head(LC) : a.recs * a.maxrec) * 8 + 16 * MMA_PAD + 127) & ~127;   // rows of the work buffers are 128-byte aligned
    zd* buf0 = reinterpret_cast<zd*>(sm + boff);
    zd* buf1 = buf0 + a.bufc;
    zd* ACC = buf1 + a.bufc;                                      // slots x 2 columns x 2 modes, acs apart

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kr = lane >> 2, kq = lane & 3;                      // row of A and C; depth of A and B, column pair of C
    const int acs = a.acs;
    const int G = gridDim.x, NI = a.ntiles * a.nchunk;
    if ((int)blockIdx.x >= NI) return;
    if (a.skip && (a.skip[0] | a.skip[1])) return;
    // everything a product may read past a block's end has to be finite
    for (zd* e = reinterpret_cast<zd*>(recb) - 1 + tid; e < ACC + a.slots * 4 * acs; e += (NW + 1) * 32) *e = mk(0.0, 0.0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (tid == 0) {
        for (int k = 0; k < 4; k++) mb_init(&bar[k], SRC == 0 && k == 0 ? 2 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *gave_up = a.give_up_at == 0;
    }

    // thread 0: the steps in order, fetched two ahead (the next tile's
    // descriptor one tile ahead)
    int f_it = blockIdx.x, f_q = 0, f_end = 0, f_row = 0, f_chunk = 0, f_cols = 0;
    int4 f_next = make_int4(0, 0, 0, 0);
    bool f_ok = false;
    auto enter = [&](int4 t) {
        f_q = t.x;
        f_end = t.x + t.y;
        f_row = t.z;
        f_chunk = f_it % a.nchunk;
        const int c0 = 2 * f_chunk;
        f_cols = (a.ncols - c0 < 2 ? 1 : 2) << 2 | ((a.contran >> (c0 % a.period)) & 1u) | ((a.contran >> ((c0 + 1) % a.period)) & 1u) << 1;
        if (f_it + G < NI) f_next = a.tiles[(f_it + G) / a.nchunk];
    };
    auto fetch = [&](Step& s) -> bool {   // the next step, if there is one
        if (!f_ok) return false;
        const int4 p = *reinterpret_cast<const int4*>(a.pairs + f_q);
        s.offi = p.x;
        s.offj = p.y;
        s.lls = (unsigned)p.z;
        s.rec4 = (unsigned)p.w;
        s.row = f_row;
        s.chunk = f_chunk;
        s.cols = f_cols;
        s.last = ++f_q == f_end;
        if (s.last) {
            f_it += G;
            if (f_it < NI) enter(f_next);
            else f_ok = false;
        }
        return true;
    };
    // uniform orders: header and rotation blocks, then the axial blocks, apart
    // (the body's single copy is free for the next pair's once read)
    double* const body = recb + op_head(LC);   // body[op_head ..]: rotation and axial blocks
    auto load_rot = [&](const Step& s, int b) {
        constexpr uint32_t h = op_head(LC) * 8u, r = (op_z_base(LC, LC) - op_head(LC)) * 8u;
        const double* g = a.ops + (size_t)s.rec4 * 4;
        mb_expect(&bar[0], h + r);
        bulk_copy(recb + b * op_head(LC), g, h, &bar[0]);
        bulk_copy(body + op_head(LC), g + op_head(LC), r, &bar[0]);
    };
    auto load_ax = [&](const Step& s, int b) {
        constexpr uint32_t z = (op_record_units(LC, LC) - op_z_base(LC, LC)) * 8u;
        mb_expect(&bar[1 + b], z);
        bulk_copy(body + op_z_base(LC, LC), a.ops + (size_t)s.rec4 * 4 + op_z_base(LC, LC), z, &bar[1 + b]);
    };
    auto load_rec = [&](const Step& s, int b) {
        const int li = s.lls & 255, lj = (s.lls >> 8) & 255;
        const uint32_t bytes = (uint32_t)(a.uniform ? a.maxrec : op_record_units(li, lj)) * 8u;
        mb_expect(&bar[b], bytes);
        bulk_copy(recb + (size_t)b * a.maxrec, a.ops + (size_t)s.rec4 * 4, bytes, &bar[b]);
    };
    auto load_src = [&](const Step& s, zd* buf) {
        const int li = s.lls & 255, lj = (s.lls >> 8) & 255;
        const int c0 = 2 * s.chunk, nr = s.cols >> 2;
        const uint32_t bi = (uint32_t)(2 * li * (li + 2) * 16), bj = (uint32_t)(2 * lj * (lj + 2) * 16);
        mb_expect(&bar[SRC], nr * (bi + bj));
        zd* d = reinterpret_cast<zd*>(buf);
        for (int r = 0; r < nr; r++) {
            const zd* xr = a.x + (size_t)(c0 + r) * a.ld;
            bulk_copy(d + r * a.bs, xr + s.offj, bj, &bar[SRC]);         // source of j -> i
            bulk_copy(d + (2 + r) * a.bs, xr + s.offi, bi, &bar[SRC]);   // source of i -> j
        }
    };
    cta_sync();
    if (warp == NW) {
        // ---- the copying warp: lane 0 runs through the steps and issues the
        // copies, the warp adds a finished tile's outputs to y ----
        if (lane == 0) {
            f_ok = true;
            enter(a.tiles[f_it / a.nchunk]);
            ring[1].lls = 0;
            Step s;
            for (int b = 0; b < 2; b++)
                if (fetch(s)) {
                    ring[b] = s;
                    if (LC && b == 0) {
                        load_rot(s, 0);
                        load_ax(s, 0);
                    }
                    if (!LC && b < a.recs) load_rec(s, b);
                    if (b == 0) load_src(s, buf0);
                }
        }
        cta_sync();
        bool due = false;   // a finished tile waits in ACC
        int row = 0, chunk = 0, nr = 0;
        // lane w: the sphere of slot w / 2 in column w mod 2 of the chunk
        auto flush_begin = [&]() {
            const int sph = lane < a.slots * 2 && (lane & 1) < nr ? a.tsph[(size_t)row * a.slots + (lane >> 1)] : -1;
            const int Ls = LC ? LC : sph >= 0 ? a.order[sph] : 1, nb = Ls * (Ls + 2);
            zd* yr = sph >= 0 ? a.y + (size_t)(2 * chunk + (lane & 1)) * a.ld + a.offset[sph] : nullptr;
            zd* own = ACC + lane * 2 * acs;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (sph >= 0) {
                bulk_add(yr, own, (uint32_t)nb * 16u);
                bulk_add(yr + nb, own + acs, (uint32_t)nb * 16u);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        };
        auto flush_end = [&]() {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
            for (zd* p = ACC + lane; p < ACC + a.slots * 4 * acs; p += 32) *p = mk(0.0, 0.0);
        };
        int dead = 0;   // lane 0: 1, a wait ran out; 2, with the next step's record on its way
        unsigned have = 0xffffffffu;
        int t = 0;
        for (;; t++) {
            const Step st = ring[t & 3];
            const int b = t & 1;
            Step nx;
            nx.lls = 0;
            if (lane == 0 && !fetch(nx)) nx.lls = 0;
            if (due && __any_sync(0xffffffffu, *gave_up)) due = false;   // in C of the last step
            if (due) flush_begin();
            if (!LC && (st.lls & 0xffffu) != have) {
                have = st.lls & 0xffffu;
                cta_sync();
            }
            cta_sync();   // B is done
            Step& s1 = ring[(t + 1) & 3];
            if (lane == 0 && (*gave_up || t == a.give_up_at)) {
                dead = !LC && a.recs == 2 && s1.lls ? 2 : 1;
                s1.lls = 0;   // the other warps read it behind D's barrier
            }
            if (LC && lane == 0 && s1.lls) {   // E_n and O_n stay in registers for D: the next pair's replace them
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                load_rot(s1, b ^ 1);
            }
            if (due) flush_end();
            cta_sync();   // C is done
            if (lane == 0 && s1.lls) {   // the next pair's sources replace a'
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                load_src(s1, b ? buf0 : buf1);
                if (LC) load_ax(s1, b ^ 1);
            }
            if (lane == 0) ring[(t + 2) & 3] = nx;
            cta_sync();   // D is done
            if (!LC && lane == 0 && s1.lls) {   // the record after next (with one buffer, the next) replaces this one
                if (a.recs == 1) nx = s1;
                if (nx.lls) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    load_rec(nx, a.recs == 2 ? b : 0);
                }
            }
            due = st.last != 0;
            row = st.row;
            chunk = st.chunk;
            nr = st.cols >> 2;
            if (!ring[(t + 1) & 3].lls) break;
        }
        if (LC && lane == 0 && !dead && *gave_up) dead = 1;   // in C of the last step
        if (__any_sync(0xffffffffu, dead != 0)) {
            if (lane == 0) {   // the last phase armed of every barrier
                const bool next = dead == 2;
                if (LC) {
                    mb_wait(&bar[0], t & 1);
                    if (SRC) mb_wait(&bar[SRC], t & 1);
                    for (int k = t; k >= 0 && k > t - 2; k--) mb_wait(&bar[1 + (k & 1)], (k >> 1) & 1);
                } else {
                    mb_wait(&bar[a.recs == 2 ? t & 1 : 0], (a.recs == 2 ? t >> 1 : t) & 1);
                    if (next) mb_wait(&bar[(t + 1) & 1], ((t + 1) >> 1) & 1);
                    mb_wait(&bar[SRC], t & 1);
                }
                atomicExch(a.err, MSTMG_ERR_CUDA);
            }
            return;
        }
        flush_begin();   // the last step ends a tile
        flush_end();
        return;
    }
    cta_sync();

    const double* zero = recb - 2;
    const unsigned long long units_rot = a.sched.rot[warp], units_ax = a.sched.ax[warp];
    constexpr int kSteps = LC ? kDeal<(LC ? LC : 1), NW>.steps : 1;
    int abp[2], abm[2];   // uniform orders: rows of a' of orders +-(kr, kr + 8)
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
        abp[mt] = 8 * abase(mt * 8 + kr, LC);
        abm[mt] = 8 * abase(-(mt * 8 + kr), LC);
    }
    unsigned have = 0xffffffffu;   // orders the offset tables hold
    for (int t = 0;; t++) {
        const Step st = ring[t & 3];
        const int b = t & 1, rb = !LC && a.recs == 2 ? b : 0;
        const int Li = LC ? LC : st.lls & 255, Lj = LC ? LC : (st.lls >> 8) & 255;
        const int nmin = Li < Lj ? Li : Lj, nmax = Li < Lj ? Lj : Li;
        const int nr = st.cols >> 2;          // columns of the chunk
        double fe[kSteps], fo[kSteps];        // uniform orders: E_n, O_n of the warp's units, from B to D
        const unsigned ct = st.cols & 3;      // bit r: column r is a conjugate-transpose product
        if (!LC && (st.lls & 0xffffu) != have) {   // the same for the whole CTA
            for (int e = tid; e <= nmax + 1; e += NW * 32) {
                if (e >= 1 && e <= nmax) roff[e] = op_head(nmax) + op_rot_offset(e, nmin);
                if (e <= nmin) zoff[e] = op_z_base(nmax, nmin) + 2 * op_z_offset(e, Li, Lj);
            }
            have = st.lls & 0xffffu;
            cta_sync();
        }
        const int par = !LC && a.recs == 2 ? (t >> 1) & 1 : t & 1;
        if (!mb_wait_warp<LC>(&bar[rb], par) || (SRC && !mb_wait_warp<LC>(&bar[SRC], t & 1))) {
            *gave_up = 1;
            return;
        }
        const double* rec = LC ? body : recb + (size_t)rb * a.maxrec;
        const zd* hdr = reinterpret_cast<const zd*>(LC ? recb + b * op_head(LC) : rec);   // e^{i m phi}, e^{-i m phi}
        zd* src = b ? buf1 : buf0;    // sources, then s' and t'
        zd* ap = b ? buf0 : buf1;     // a'
        zd* tp = src + (nmax * (nmax + 3) / 2) * 8;   // t' after s'

        if constexpr (LC > 0) {
            // Uniform orders: D^T = S C D C^-1 S (S = diag((-1)^n), c_0 = 1/2) and
            // Z^T = S Z S let both directions and both rotations read the
            // blocks row by row; the signs go with a', s' and t'.
            // ---- A + B: shift, phase, even/odd split, forward rotation ----
            // With N = x(-m) and e = c + i d (e^{i m phi}, conjugated in
            // conjugate-transpose columns): p = x(m) + (-1)^m N, q = x(m) -
            // (-1)^m N, s = c p + i d q, t = c q + i d p; where the shift
            // applies t changes sign, i.e. a'(k) and a'(-k) trade places.
            // a'(-k) is kept without its (-1)^k.
            {
                const int dir = kr & 1, mode = kr >> 2, r = (kr >> 1) & 1;   // of the lane's B operand column
                const zd* xs = reinterpret_cast<const zd*>(src) + (dir * 2 + r) * a.bs + mode * LC * (LC + 2);
                const zd* eh = hdr + kq + ((ct >> r) & 1u ? LC + 1 : 0);
                const double sg = kq & 1 ? -1.0 : 1.0;
                const int cto = (int)((ct >> (kq & 1)) & 1u);   // of the lane's output columns
                const int apo = b ? boff : boff + 16 * a.bufc;   // a', a byte offset
                const int wl = apo + 16 * (kq ^ ((kr & 1) << 2));
                warp_units<LC, NW, false>(warp, [&](auto U, auto O0) {
                    constexpr int n = decltype(U)::value, F = n / 4 + 1, MT = n / 8 + 1;   // steps of 4 orders, tiles of 8 rows
                    const double* E = rec + op_head(LC) + op_rot_offset(n, LC) + kr * (n + 1) + kq;
                    constexpr int OO = (n + 1) * (n + 1);
                    const zd* x0 = xs + (LC + 2) * (n - 1) + kq;
                    const zd* xm = xs + n + 1 + (LC + 2) * (kq - 1);
                    double Pr[MT][2], Pi[MT][2], Qr[MT][2], Qi[MT][2];
#pragma unroll
                    for (int ks = 0; ks < F; ks++) {
                        const zd* pp = x0 + 4 * ks;
                        const zd* pm = ks ? xm + 4 * ks * (LC + 2) : kq ? xm : x0;
                        if (4 * ks + 3 > n && kq > n - 4 * ks) pp = pm = reinterpret_cast<const zd*>(zero);
                        const zd X = ldx(pp), N = ldx(pm), e = ldx(eh + 4 * ks);
                        const zd p = mk(fma(sg, N.x, X.x), fma(sg, N.y, X.y)), q = mk(fma(-sg, N.x, X.x), fma(-sg, N.y, X.y));
                        const double sx = fma(e.x, p.x, -(e.y * q.y)), sy = fma(e.x, p.y, e.y * q.x);
                        const double tx = fma(e.x, q.x, -(e.y * p.y)), ty = fma(e.x, q.y, e.y * p.x);
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) {
                            const int o = decltype(O0)::value + mt * F + ks;
                            fe[o] = E[mt * 8 * (n + 1) + 4 * ks];
                            fo[o] = E[mt * 8 * (n + 1) + OO + 4 * ks];
                            mma884(Pr[mt], fe[o], sx, ks == 0);
                            mma884(Pi[mt], fe[o], sy, ks == 0);
                            mma884(Qr[mt], fo[o], tx, ks == 0);
                            mma884(Qi[mt], fo[o], ty, ks == 0);
                        }
                    }
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
                        // a'(k) and a'(-k) of the lane's two columns, times (-1)^n in direction 1
                        const int bp = mt ? abp[1] : abp[0], bm = mt ? abm[1] : abm[0];
                        const int wp = wl + 16 * (cto ? bm : bp) + n * 128, wm = wl + 16 * (cto ? bp : bm) + n * 128;
                        const bool in = n >= mt * 8 + 7 || mt * 8 + kr <= n;
                        constexpr int x = 16 * (n & 3);
                        if (in) sto(sm, wp ^ x, mk(Pr[mt][0] + Qr[mt][0], Pi[mt][0] + Qi[mt][0]));
                        if (in) sto(sm, wm ^ x, mk(Pr[mt][0] - Qr[mt][0], Pi[mt][0] - Qi[mt][0]));
                        if (n & 1) {
                            if (in) sto(sm, wm ^ x ^ 64, mk(-Pr[mt][1] - Qr[mt][1], -Pi[mt][1] - Qi[mt][1]));
                            if (in) sto(sm, wp ^ x ^ 64, mk(Qr[mt][1] - Pr[mt][1], Qi[mt][1] - Pi[mt][1]));
                        } else {
                            if (in) sto(sm, wm ^ x ^ 64, mk(Pr[mt][1] + Qr[mt][1], Pi[mt][1] + Qi[mt][1]));
                            if (in) sto(sm, wp ^ x ^ 64, mk(Pr[mt][1] - Qr[mt][1], Pi[mt][1] - Qi[mt][1]));
                        }
                    }
                });
            }
            cta_sync();
            if (!mb_wait_warp<LC>(&bar[1 + b], (t >> 1) & 1)) {
                *gave_up = 1;
                return;
            }

            // ---- C: axial translation ----
            {
                const int mode = kr >> 2, col = (kr >> 1) + 4 * (kr & 1);
                const int md = kq >> 1, cto = (int)((ct >> (kq & 1)) & 1u);   // of the lane's output columns
                const int so = b ? boff + 16 * a.bufc : boff, to = so + (LC * (LC + 3) / 2) * 128;   // s', t': byte offsets
                warp_units<LC, NW, true>(warp, [&](auto U) {
                    constexpr int m = decltype(U)::value;
                    constexpr int m1 = m ? m : 1, j = LC - m1 + 1, F = (j + 3) / 4, MT = (j + 7) / 8;   // steps of 4 source degrees, tiles of 8 rows
                    const zd* Z = reinterpret_cast<const zd*>(rec + op_z_base(LC, LC) + 2 * op_z_offset(m, LC, LC)) + kr * j + kq;
                    // both modes of m: mode 0 takes m with Z^0 and -m with Z^1, mode 1 the other way round
                    constexpr int bp = (abase(m, LC) + m1) * 8, bm = (abase(-m, LC) + m1) * 8;
                    const int wc = ((m1 + kq) & 3) ^ ((m & 1) << 2) ^ col;
                    const zd* X0 = ap + (wc + kq * 8) + (mode ? bm : bp);
                    const zd* X1 = ap + (wc + kq * 8) + (mode ? bp : bm);
                    double r0[MT][2], i0[MT][2], r1[MT][2], i1[MT][2], n0[MT][2], n1[MT][2];
#pragma unroll
                    for (int ks = 0; ks < F; ks++) {
                        const zd* p0 = X0 + 32 * ks;
                        const zd* p1 = X1 + 32 * ks;
                        if (4 * ks + 4 > j && kq >= j - 4 * ks) p0 = p1 = reinterpret_cast<const zd*>(zero);
                        const zd x0 = ldx(p0), x1 = m ? ldx(p1) : x0;
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) {
                            const zd z0 = ldx(Z + mt * 8 * j + 4 * ks);
                            mma884(r0[mt], z0.x, x0.x, ks == 0);
                            mma884(i0[mt], z0.x, x0.y, ks == 0);
                            if (m) {
                                const zd z1 = ldx(Z + j * j + mt * 8 * j + 4 * ks);
                                mma884(r1[mt], z1.x, x1.x, ks == 0);
                                mma884(i1[mt], z1.x, x1.y, ks == 0);
                                mma884(n1[mt], z1.y, x1.y, ks == 0);
                                mma884(i1[mt], z1.y, x1.x);
                            }
                            mma884(n0[mt], z0.y, x0.y, ks == 0);
                            mma884(i0[mt], z0.y, x0.x);
                        }
                    }
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
                        const int nt = m1 + mt * 8 + kr;
                        const int oc = 16 * (kq ^ (m & 3) ^ ((nt & 1) << 2));
                        const int ws = so + srow(nt, m) * 128 + oc;
                        const bool in = j >= mt * 8 + 8 || nt <= LC;
                        if (m == 0) {   // 1 / c_0, (-1)^nt in direction 1
                            if (in) sto(sm, ws, mk(2.0 * (r0[mt][0] - n0[mt][0]), 2.0 * i0[mt][0]));
                            if (in) sto(sm, ws ^ 64, mk(flip(2.0 * (r0[mt][1] - n0[mt][1]), nt), flip(2.0 * i0[mt][1], nt)));
                        } else {
                            // g0 is g(m) in mode 0, (-1)^m g(-m) in mode 1, g1 the other:
                            // s' = g0 + g1, t' = +-(g0 - g1), both times (-1)^m, times
                            // (-1)^nt in direction 1, t' also times the shift's sign
                            const int wt = to + trow(nt, m) * 128 + oc;
                            const int mc = md ^ cto ^ m;
                            const double a0 = r0[mt][0] - n0[mt][0], a1 = r1[mt][0] - n1[mt][0], b0 = r0[mt][1] - n0[mt][1], b1 = r1[mt][1] - n1[mt][1];
                            if ((m & 1) && in) sto(sm, ws, mk(-a0 - a1, -i0[mt][0] - i1[mt][0]));
                            else if (in) sto(sm, ws, mk(a0 + a1, i0[mt][0] + i1[mt][0]));
                            if (in) sto(sm, wt, mk(flip(a0 - a1, mc), flip(i0[mt][0] - i1[mt][0], mc)));
                            if (in) sto(sm, ws ^ 64, mk(flip(b0 + b1, m ^ nt), flip(i0[mt][1] + i1[mt][1], m ^ nt)));
                            if (in) sto(sm, wt ^ 64, mk(flip(b0 - b1, mc ^ nt ^ 1), flip(i0[mt][1] - i1[mt][1], mc ^ nt ^ 1)));
                        }
                    }
                });
            }
        } else {

            // ---- A + B: shift, phase, even/odd split, forward rotation ----
            // With P = x(m), M = (-1)^m x(-m) and e^{i m phi} = c + i d (d negated
            // in conjugate-transpose columns): s = c (P + M) + i d (P - M),
            // t = +-(c (P - M) + i d (P + M)), - where the shift applies.
            {
                const int dir = kr & 1, mode = kr >> 2, r = (kr >> 1) & 1;   // of the lane's B operand column
                const int Ls = dir ? Li : Lj, ctr = (int)((ct >> r) & 1u), swp = dir ^ ctr;
                const zd* xs = reinterpret_cast<const zd*>(src) + (dir * 2 + r) * a.bs + mode * Ls * (Ls + 2);
                const zd* eh = reinterpret_cast<const zd*>(rec);
                auto unit = [&](auto FC, int n, int mt) {
                    constexpr int F = decltype(FC)::value;   // whole steps of 4 orders m = 1 .. 4 F; then the rest and m = 0
                    const int kk = min(n, nmin), row = mt * 8 + kr, rem = n - 4 * F;
                    const double* E = rec + roff[n] + row * (n + 1);
                    const double* O = E + (kk + 1) * (n + 1) + kq + 1;
                    const bool src_ok = n <= Ls;
                    const zd* x0 = xs + (src_ok ? (Ls + 2) * (n - 1) : 0);
                    const zd* xm = xs + (src_ok ? (n + 1) + (Ls + 2) * kq : 0);
                    double Pr[2] = {0.0, 0.0}, Pi[2] = {0.0, 0.0}, Qr[2] = {0.0, 0.0}, Qi[2] = {0.0, 0.0};
                    auto step = [&](zd xp, zd xn, zd e, int sg, double ea, double oa, bool odd) {
                        const zd M = mk(flip(xn.x, sg), flip(xn.y, sg));
                        const zd p = xp + M, d = xp - M;
                        const double ei = flip(e.y, ctr);
                        mma884(Pr, ea, e.x * p.x - ei * d.y);
                        mma884(Pi, ea, e.x * p.y + ei * d.x);
                        if (odd) {
                            mma884(Qr, oa, flip(e.x * d.x - ei * p.y, swp));
                            mma884(Qi, oa, flip(e.x * d.y + ei * p.x, swp));
                        }
                    };
#pragma unroll
                    for (int ks = 0; ks < F; ks++)
                        step(ldx(x0 + 4 * ks + kq + 1), ldx(xm + 4 * ks * (Ls + 2)), ldx(eh + 4 * ks + kq + 1), (kq + 1) & 1, E[4 * ks + kq + 1],
                             O[4 * ks], true);
                    {   // the rest: lanes kq < rem, m = 0 in lane kq = rem, nothing in the others
                        zd xp = mk(0.0, 0.0), xn = xp, e = xp;
                        double ea = 0.0, oa = 0.0;
                        int sg = (kq + 1) & 1;
                        if (kq < rem) {
                            xp = ldx(x0 + 4 * F + kq + 1);
                            xn = ldx(xm + 4 * F * (Ls + 2));
                            e = ldx(eh + 4 * F + kq + 1);
                            ea = E[4 * F + kq + 1];
                            oa = O[4 * F];
                        } else if (kq == rem) {
                            xp = ldx(x0);
                            xn = xp;
                            e = mk(1.0, 0.0);
                            ea = E[0];
                            sg = 0;
                        }
                        step(xp, xn, e, sg, ea, oa, rem > 0);
                    }
                    if (row <= kk) {
                        const int sk = row & 1;
                        zd* wp = ap + (abase(row, nmax) + n) * 8;
                        zd* wm = ap + (abase(-row, nmax) + n) * 8;
#pragma unroll
                        for (int d = 0; d < 2; d++) {
                            const int wc = acol(n, row, d * 4 + kq);
                            const zd P = mk(Pr[d], Pi[d]), Q = mk(Qr[d], Qi[d]);
                            stx(wp + wc, P + Q);
                            if (row) {
                                const zd D = P - Q;
                                stx(wm + wc, mk(flip(D.x, sk), flip(D.y, sk)));
                            }
                        }
                    }
                };
                for (unsigned long long u = units_rot; u; u >>= 8) {
                    __syncwarp();   // the lanes part in the epilogues
                    const int n = (int)u & 31, mt = ((int)u >> 5) & 7;
                    if (n > nmax || mt * 8 > min(n, nmin)) continue;
                    switch (n >> 2) {
                    case 0: unit(IntC<0>{}, n, mt); break;
                    case 1: unit(IntC<1>{}, n, mt); break;
                    case 2: unit(IntC<2>{}, n, mt); break;
                    case 3: unit(IntC<3>{}, n, mt); break;
                    default: unit(IntC<4>{}, n, mt); break;
                    }
                }
            }
            cta_sync();

            // ---- C: axial translation ----
            {
                const int c = kr >> 1, h = kr & 1, mode = kr >> 2;
                auto unit = [&](auto FC, auto M0, int m, int mt, int dir) {
                    constexpr int F = decltype(FC)::value;   // whole steps of 4 source degrees
                    constexpr bool m0 = decltype(M0)::value;
                    const int m1 = m0 ? 1 : m;
                    const int Lt = dir ? Lj : Li, Ls = dir ? Li : Lj;
                    const int rows = Li - m1 + 1, cols = Lj - m1 + 1, row = mt * 8 + kr, rem = Ls - m1 + 1 - 4 * F;
                    const zd* Z = reinterpret_cast<const zd*>(rec + zoff[m]) + (dir ? row + kq * cols : row * cols + kq);
                    const int zst = dir ? 4 * cols : 4, zrc = rows * cols;
                    // both modes of m: mode 0 takes m with Z^0 and -m with Z^1, mode 1 the other way round
                    const int wc = acol(m1 + kq, m, dir * 4 + c);
                    const double* X0 = reinterpret_cast<const double*>(ap + (abase(mode ? -m : m, nmax) + m1 + kq) * 8 + wc);
                    const double* X1 = m0 ? X0 : reinterpret_cast<const double*>(ap + (abase(mode ? m : -m, nmax) + m1 + kq) * 8 + wc);
                    double g0[2] = {0.0, 0.0}, g1[2] = {0.0, 0.0};
                    auto step = [&](int ks, bool in) {
                        zd z0 = mk(0.0, 0.0), z1 = z0;
                        double a0 = 0.0, b0 = 0.0, a1 = 0.0, b1 = 0.0;
                        if (in) {
                            z0 = ldx(Z + ks * zst);
                            a0 = X0[64 * ks + h];
                            b0 = flip(X0[64 * ks + (h ^ 1)], h ^ 1);
                            if (!m0) {
                                z1 = ldx(Z + zrc + ks * zst);
                                a1 = X1[64 * ks + h];
                                b1 = flip(X1[64 * ks + (h ^ 1)], h ^ 1);
                            }
                        }
                        mma884(g0, z0.x, a0);
                        if (!m0) mma884(g1, z1.x, a1);
                        mma884(g0, z0.y, b0);
                        if (!m0) mma884(g1, z1.y, b1);
                    };
#pragma unroll
                    for (int ks = 0; ks < F; ks++) step(ks, true);
                    if (rem) step(F, kq < rem);
                    const int nt = m1 + row;
                    if (nt <= Lt) {
                        const int oc = scol(nt, m, dir * 4 + kq);
                        zd* ws = src + srow(nt, m) * 8 + oc;
                        if (m0) {
                            stx(ws, mk(g0[0], g0[1]));
                        } else {
                            const int sg = m & 1;
                            const bool md = kq >> 1;
                            const zd gp = md ? mk(g1[0], g1[1]) : mk(g0[0], g0[1]), gm0 = md ? mk(g0[0], g0[1]) : mk(g1[0], g1[1]);
                            const zd gm = mk(flip(gm0.x, sg), flip(gm0.y, sg));
                            stx(ws, gp + gm);
                            stx(tp + trow(nt, m) * 8 + oc, gp - gm);
                        }
                    }
                };
                for (unsigned long long u = units_ax; u; u >>= 8) {
                    __syncwarp();   // the lanes part in the epilogues
                    const int m = (int)u & 31, mt = ((int)u >> 5) & 1, dir = ((int)u >> 6) & 1;
                    const int j = (dir ? Li : Lj) - (m ? m : 1) + 1;   // source degrees
                    if (m > nmin || mt * 8 > (dir ? Lj : Li) - (m ? m : 1)) continue;
                    if (m == 0) {
                        switch (j >> 2) {
                        case 0: unit(IntC<0>{}, IntC<1>{}, 0, mt, dir); break;
                        case 1: unit(IntC<1>{}, IntC<1>{}, 0, mt, dir); break;
                        case 2: unit(IntC<2>{}, IntC<1>{}, 0, mt, dir); break;
                        case 3: unit(IntC<3>{}, IntC<1>{}, 0, mt, dir); break;
                        default: unit(IntC<4>{}, IntC<1>{}, 0, mt, dir); break;
                        }
                    } else {
                        switch (j >> 2) {
                        case 0: unit(IntC<0>{}, IntC<0>{}, m, mt, dir); break;
                        case 1: unit(IntC<1>{}, IntC<0>{}, m, mt, dir); break;
                        case 2: unit(IntC<2>{}, IntC<0>{}, m, mt, dir); break;
                        case 3: unit(IntC<3>{}, IntC<0>{}, m, mt, dir); break;
                        default: unit(IntC<4>{}, IntC<0>{}, m, mt, dir); break;
                        }
                    }
                }
            }
        }
        cta_sync();
        if constexpr (LC > 0) {
            // ---- D: back rotation, phase, shift, into the tile's outputs ----
            // With e = e^{-i k phi}, conjugated in conjugate-transpose columns:
            // out(k) = (-1)^k (P + Q) e, out(-k) = (P - Q) conj(e); the shift's
            // sign came with t'.
            {
                const int colB = (kr >> 1) + 4 * (kr & 1);
                const int mode = kq >> 1, r = kq & 1;   // of this lane's output columns
                zd* acc0 = ACC + ((((st.lls >> 16) & 255) * 2 + r) * 2 + mode) * acs + kr;
                zd* acc1 = ACC + (((st.lls >> 24) * 2 + r) * 2 + mode) * acs + kr;
                const zd* eh = hdr + kr + ((ct >> r) & 1u ? 0 : LC + 1);
                const int wl = colB ^ kq;
                warp_units<LC, NW, false>(warp, [&](auto U, auto O0) {
                    constexpr int n = decltype(U)::value, F = n / 4 + 1, MT = n / 8 + 1;
                    const zd* S = src + srow(n, 0) * 8 + kq * 8 + (wl ^ ((n & 1) << 2));
                    const zd* Tt = tp + trow(n, 0) * 8 + kq * 8 + (wl ^ ((n & 1) << 2));
                    double Pr[MT][2], Pi[MT][2], Qr[MT][2], Qi[MT][2];
#pragma unroll
                    for (int ks = 0; ks < F; ks++) {
                        const zd* ps = S + 32 * ks;
                        const zd* pt = ks || kq ? Tt + 32 * ks : reinterpret_cast<const zd*>(zero);   // no t'(0)
                        if (4 * ks + 3 > n && kq > n - 4 * ks) ps = pt = reinterpret_cast<const zd*>(zero);
                        const zd s = ldx(ps), tt = ldx(pt);
#pragma unroll
                        for (int mt = 0; mt < MT; mt++) {
                            const int o = decltype(O0)::value + mt * F + ks;
                            mma884(Pr[mt], fe[o], s.x, ks == 0);
                            mma884(Pi[mt], fe[o], s.y, ks == 0);
                            mma884(Qr[mt], fo[o], tt.x, ks == 0);
                            mma884(Qi[mt], fo[o], tt.y, ks == 0);
                        }
                    }
#pragma unroll
                    for (int mt = 0; mt < MT; mt++) {
                        const zd e = ldx(eh + mt * 8);
                        const double ck = flip(e.x, kr), sk = flip(e.y, kr);
                        const int op = (LC + 2) * (n - 1) + mt * 8, on = n + 1 + (LC + 2) * (mt * 8 - 1);
                        const bool off = (n < mt * 8 + 7 && mt * 8 + kr > n) || r >= nr, off0 = off || (mt == 0 && kr == 0);
#pragma unroll
                        for (int d = 0; d < 2; d++) {
                            const zd gk = mk(Pr[mt][d] + Qr[mt][d], Pi[mt][d] + Qi[mt][d]), gm = mk(Pr[mt][d] - Qr[mt][d], Pi[mt][d] - Qi[mt][d]);
                            zd* ak = (d ? acc1 : acc0) + op;
                            zd* an = (d ? acc1 : acc0) + kr * (LC + 1) + on;
                            const zd vk = off ? mk(0.0, 0.0) : ldx(ak), vm = off0 ? mk(0.0, 0.0) : ldx(an);
                            if (!off) stx(ak, mk(fma(gk.x, ck, fma(-gk.y, sk, vk.x)), fma(gk.x, sk, fma(gk.y, ck, vk.y))));
                            if (!off0) stx(an, mk(fma(gm.x, e.x, fma(gm.y, e.y, vm.x)), fma(gm.y, e.x, fma(-gm.x, e.y, vm.y))));
                        }
                    }
                });
            }
        } else {
            // ---- D: back rotation, phase, shift, into the tile's outputs ----
            // With e^{i k phi} = c + i d (d negated unless the column is a
            // conjugate transpose): out(k) = (P + Q)(c + i d), out(-k) = (-1)^k
            // (P - Q)(c - i d), Q negated where the shift applies.
            {
                const int colB = (kr >> 1) + 4 * (kr & 1);
                const int mode = kq >> 1, r = kq & 1;   // of this lane's output columns
                const int cto = (int)((ct >> r) & 1u);
                auto unit = [&](auto FC, int n, int mt) {
                    constexpr int F = decltype(FC)::value;   // whole steps of 4 orders m = 1 .. 4 F; then the rest and m = 0
                    const int kk = min(n, nmin), row = mt * 8 + kr, rem = kk - 4 * F;
                    const double* E = rec + roff[n] + row;
                    const double* O = E + (kk + 1) * (n + 1) + (kq + 1) * (n + 1);
                    const int wc = scol(n, kq + 1, colB);
                    const zd* S = src + srow(n, kq + 1) * 8 + wc;
                    const zd* Tt = tp + trow(n, kq + 1) * 8 + wc;
                    double Pr[2] = {0.0, 0.0}, Pi[2] = {0.0, 0.0}, Qr[2] = {0.0, 0.0}, Qi[2] = {0.0, 0.0};
                    auto step = [&](zd s, zd tt, double ea, double oa, bool odd) {
                        mma884(Pr, ea, s.x);
                        mma884(Pi, ea, s.y);
                        if (odd) {
                            mma884(Qr, oa, tt.x);
                            mma884(Qi, oa, tt.y);
                        }
                    };
#pragma unroll
                    for (int ks = 0; ks < F; ks++) step(ldx(S + 32 * ks), ldx(Tt + 32 * ks), E[(4 * ks + kq + 1) * (n + 1)], O[4 * ks * (n + 1)], true);
                    {
                        zd s = mk(0.0, 0.0), tt = s;
                        double ea = 0.0, oa = 0.0;
                        if (kq < rem) {
                            s = ldx(S + 32 * F);
                            tt = ldx(Tt + 32 * F);
                            ea = E[(4 * F + kq + 1) * (n + 1)];
                            oa = O[4 * F * (n + 1)];
                        } else if (kq == rem) {
                            s = ldx(src + srow(n, 0) * 8 + scol(n, 0, colB));
                            ea = E[0];
                        }
                        step(s, tt, ea, oa, rem > 0);
                    }
                    if (row <= n && r < nr) {
                        zd e = ldx(reinterpret_cast<const zd*>(rec) + row);
                        if (row == 0) e.x = 2.0;   // out(0) = 2 P: E(m, 0) holds d(m, 0) / 2
                        const double ei = flip(e.y, cto ^ 1);
                        const int sk = row & 1;
#pragma unroll
                        for (int d = 0; d < 2; d++) {
                            const int Lt = d ? Lj : Li, slot = (st.lls >> (d ? 24 : 16)) & 255;
                            if (n > Lt) continue;
                            zd* acc = ACC + ((slot * 2 + r) * 2 + mode) * acs;
                            zd* op = acc + row + (Lt + 2) * (n - 1);
                            const int sq = d ^ cto;
                            const zd Q = mk(flip(Qr[d], sq), flip(Qi[d], sq));
                            const zd gk = mk(Pr[d], Pi[d]) + Q, gm = mk(Pr[d], Pi[d]) - Q;
                            const zd vk = ldx(op);
                            stx(op, mk(vk.x + (gk.x * e.x - gk.y * ei), vk.y + (gk.x * ei + gk.y * e.x)));
                            if (row) {
                                zd* on = acc + (n + 1) + (Lt + 2) * (row - 1);
                                const zd vm = ldx(on);
                                const double cs = flip(e.x, sk), sn = flip(ei, sk);
                                stx(on, mk(vm.x + (gm.x * cs + gm.y * sn), vm.y + (gm.y * cs - gm.x * sn)));
                            }
                        }
                    }
                };
                for (unsigned long long u = units_rot; u; u >>= 8) {
                    __syncwarp();   // the lanes part in the epilogues
                    const int n = (int)u & 31, mt = ((int)u >> 5) & 7;
                    if (n > nmax) continue;
                    const int kk = min(n, nmin);
                    switch (kk >> 2) {
                    case 0: unit(IntC<0>{}, n, mt); break;
                    case 1: unit(IntC<1>{}, n, mt); break;
                    case 2: unit(IntC<2>{}, n, mt); break;
                    case 3: unit(IntC<3>{}, n, mt); break;
                    default: unit(IntC<4>{}, n, mt); break;
                    }
                }
            }
        }
        if (st.last) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the copying warp's reductions read ACC
        cta_sync();
        if (!ring[(t + 1) & 3].lls) break;
    }
}

namespace {

// Units in descending order of MMAs, each to the warp with the least so far.
bool deal(std::vector<std::pair<int, int>> units, int nw, int cap, unsigned long long* out)
{
    std::stable_sort(units.begin(), units.end(), [](const auto& p, const auto& q) { return p.first > q.first; });
    std::vector<int> load(nw, 0), count(nw, 0);
    for (int i = 0; i < nw; i++) out[i] = 0;
    for (const auto& u : units) {
        const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        if (count[k] == cap) return false;
        out[k] |= (unsigned long long)u.second << (8 * count[k]++);
        load[k] += u.first + 4;   // a unit's set-up and epilogue cost about four MMAs
    }
    return true;
}

bool make_sched(int L, int nw, MmaSched& s)
{
    std::vector<std::pair<int, int>> rot, ax;
    for (int n = 1; n <= L; n++)
        for (int mt = 0; mt * 8 <= n; mt++) rot.push_back({2 * (n / 4 + 1 + (n + 3) / 4), n | mt << 5});
    for (int m = 0; m <= L; m++) {
        const int j = L - (m ? m : 1) + 1;
        for (int mt = 0; mt * 8 < j; mt++)
            for (int dir = 0; dir < 2; dir++) ax.push_back({(m ? 4 : 2) * ((j + 3) / 4), 128 | m | mt << 5 | dir << 6});
    }
    return deal(rot, nw, 8, s.rot) && deal(ax, nw, 8, s.ax);
}

template <int LC, int NW, int MINB> int launch_nw(MmaArgs& a, int nsm, cudaStream_t st)
{
    const int nb = 2 * a.L * (a.L + 2);
    // source blocks and the accumulators' modes 2 of 8 complex apart: the
    // lanes of an access phase on different banks
    a.bs = nb + (10 - nb % 8) % 8;
    a.bufc = std::max(8 * (nb / 2), 4 * a.bs);
    a.acs = nb / 2 + (10 - (nb / 2) % 8) % 8;
    a.nchunk = (a.ncols + 1) / 2;
    if (LC == 0 && !make_sched(a.L, NW, a.sched)) return -1;
    // two record buffers; one for orders whose buffers would not fit (16)
    a.bufc = (a.bufc + 7) & ~7;
    const size_t work = MMA_HEAD + 16 * MMA_PAD + 128 + 16 * (2 * (size_t)a.bufc + 4 * (size_t)a.slots * a.acs);
    a.recs = work + 16 * (size_t)a.maxrec <= 227 * 1024 ? 2 : 1;
    const size_t smem = work + 8 * (LC ? (size_t)a.maxrec + op_head(LC) : a.recs * (size_t)a.maxrec);
    if (smem > 227 * 1024) return -1;
    auto kern = translate_mma_kernel<LC, NW, MINB>;
    allow_smem(kern, smem);
    int per_sm = (int)((228 * 1024) / (smem + 1024));
    if (per_sm > MINB) per_sm = MINB;
    if (per_sm < 1) per_sm = 1;
    if (a.ctas_per_sm >= 1 && a.ctas_per_sm < per_sm) per_sm = a.ctas_per_sm;
    const long long items = (long long)a.ntiles * a.nchunk;
    const int blocks = (int)std::min<long long>((long long)nsm * per_sm, items);
    if (blocks < 1) return 0;
    kern<<<blocks, (NW + 1) * 32, smem, st>>>(a);
    launch_counter() += 1;
    return 0;
}

}  // namespace

// Warps a CTA and CTAs per SM by order, the fastest of 2 to 8 warps and the
// CTAs that fit (us, 2 columns FP64; spheres x order: 1200 x 4 1840, 1000 x 5
// 1737, 700 x 6 1182, 700 x 7 1356, 500 x 8 889, 500 x 9 1202, 300 x 10 635;
// when they were chosen order 9 took 1172, at 4 warps x 3 CTAs 1389, at 8 x 2
// 2160; order 5 1700, at 4 x 4 2030).
int launch_translate_mma(MmaArgs& a, int nsm, cudaStream_t st)
{
    if (a.uniform) {
        switch (a.L) {
        case 3: return launch_nw<3, 2, 8>(a, nsm, st);
        case 4: return launch_nw<4, 2, 8>(a, nsm, st);
        case 5: return launch_nw<5, 2, 8>(a, nsm, st);
        case 6: return launch_nw<6, 3, 5>(a, nsm, st);
        case 7: return launch_nw<7, 3, 4>(a, nsm, st);
        case 8: return launch_nw<8, 3, 4>(a, nsm, st);
        case 9: return launch_nw<9, 3, 4>(a, nsm, st);
        case 10: return launch_nw<10, 4, 3>(a, nsm, st);
        default: break;
        }
    }
    if (a.L <= 5) return launch_nw<0, 2, 8>(a, nsm, st);
    if (a.L <= 7) return launch_nw<0, 4, 4>(a, nsm, st);
    if (a.L <= 11) return launch_nw<0, 8, 2>(a, nsm, st);
    return launch_nw<0, 16, 1>(a, nsm, st);
}

// FP32 columns in and out of the FP64 pass: x to FP64 with y cleared, and y
// rounded back (added to what is there with `add`)
__global__ void mma_widen_kernel(int n, const float4* x, double2* xd, double2* yd)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const float4 v = x[k];
        xd[2 * k] = make_double2((double)v.x, (double)v.y);
        xd[2 * k + 1] = make_double2((double)v.z, (double)v.w);
        yd[2 * k] = yd[2 * k + 1] = make_double2(0.0, 0.0);
    }
}
__global__ void mma_narrow_kernel(int n, const double2* yd, float4* y, int add)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const double2 a = yd[2 * k], b = yd[2 * k + 1];
        float4 v = make_float4((float)a.x, (float)a.y, (float)b.x, (float)b.y);
        if (add) {
            const float4 o = y[k];
            v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
        }
        y[k] = v;
    }
}
__global__ void pair_offsets_kernel(int np, int rec, long long* opoff)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < np; q += gridDim.x * blockDim.x) opoff[q] = (long long)q * rec;
}
__global__ void mma_pairs_kernel(int np, const int2* pairs, const uchar2* slots, const int* order, const int* offset, const long long* opoff,
                                 MmaPair* out)
{
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < np; q += gridDim.x * blockDim.x) {
        const int i = pairs[q].x, j = pairs[q].y;
        out[q] = MmaPair{offset[i], offset[j], (unsigned)order[i] | (unsigned)order[j] << 8 | (unsigned)slots[q].x << 16 | (unsigned)slots[q].y << 24,
                         (unsigned)(opoff[q] / 4)};
    }
}
static int cvt_blocks(int n, int nsm) { return std::max(1, std::min((n + 255) / 256, 8 * nsm)); }
void launch_pair_offsets(int np, int rec, long long* opoff, int nsm, cudaStream_t st)
{
    pair_offsets_kernel<<<cvt_blocks(np, nsm), 256, 0, st>>>(np, rec, opoff);
    launch_counter() += 1;
}
void launch_mma_pairs(int np, const int2* pairs, const uchar2* slots, const int* order, const int* offset, const long long* opoff,
                      MmaPair* out, int nsm, cudaStream_t st)
{
    mma_pairs_kernel<<<cvt_blocks(np, nsm), 256, 0, st>>>(np, pairs, slots, order, offset, opoff, out);
    launch_counter() += 1;
}
void launch_mma_widen(size_t values, const zf* x, zd* xd, zd* yd, int nsm, cudaStream_t st)
{
    const int n = (int)(values / 2);   // a vector holds an even number of values
    mma_widen_kernel<<<cvt_blocks(n, nsm), 256, 0, st>>>(n, reinterpret_cast<const float4*>(x), reinterpret_cast<double2*>(xd),
                                                         reinterpret_cast<double2*>(yd));
    launch_counter() += 1;
}
void launch_mma_narrow(size_t values, const zd* yd, zf* y, bool add, int nsm, cudaStream_t st)
{
    const int n = (int)(values / 2);
    mma_narrow_kernel<<<cvt_blocks(n, nsm), 256, 0, st>>>(n, reinterpret_cast<const double2*>(yd), reinterpret_cast<float4*>(y), add);
    launch_counter() += 1;
}

// Self-test of the bounded wait: one CTA waits on an mbarrier whose
// transaction never arrives (an expected byte count with no copy issued), gives
// up after `limit` polls per thread and records MSTMG_ERR_CUDA in *err -- the
// path the translation kernel takes when a bulk copy does not complete.  No
// asynchronous operation is in flight when it returns.
__global__ void wait_selftest_kernel(int limit, int* err)
{
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mb_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) mb_expect(&bar, 16u);
    __syncthreads();
    if (!mb_wait(&bar, 0u, limit)) {
        if (threadIdx.x == 0) atomicExch(err, MSTMG_ERR_CUDA);
    }
}

int launch_wait_selftest(int limit, int* err, cudaStream_t st)
{
    wait_selftest_kernel<<<1, 64, 0, st>>>(limit, err);
    launch_counter() += 1;
    return 0;
}
