// translate_mma.cuh -- the pair translation pass on the FP64 tensor cores.
#pragma once
#include "common.cuh"

#define MMA_WARPS_MAX 16

// One pair of a tile, in tile order (16 bytes): the blocks of its spheres in
// a vector (complex units), orders and tile slots (order i | order j << 8 |
// slot i << 16 | slot j << 24), and its operator record (units of 4 doubles).
struct MmaPair {
    int offi, offj;
    unsigned lls;
    unsigned rec4;
};

// Work units of a pair for tiles whose largest order is L, dealt to the warps
// of a CTA, up to 8 codes of 8 bits a warp, lowest byte first, 0 ends.
// Rotation unit: degree n | row tile << 5; axial unit: order m | row tile << 5
// | direction << 6 | 128.
struct MmaSched {
    unsigned long long rot[MMA_WARPS_MAX], ax[MMA_WARPS_MAX];
};

struct MmaArgs {
    int ntiles;
    const int4* tiles;      // (first pair, pairs, row of tsph, 0)
    const MmaPair* pairs;
    const int* tsph;        // the spheres of every tile row by slot (`slots` a row), -1: none
    const int* order;
    const int* offset;
    const double* ops;      // operator records (oplayout.cuh)
    const zd* x;            // ld x ncols
    zd* y;                  // ld x ncols, accumulated
    int ld, ncols;
    unsigned contran;       // column k is a conjugate-transpose product when bit (k mod period) is set
    int period;
    int L, uniform;         // largest order of the tiles; 1: every pair has both orders L
    int slots;              // tile slots in use (2, 4 or 8)
    int maxrec;             // largest record of the tiles, doubles
    int* err;
    int give_up_at;         // -1; self-test: a wait of every CTA's pair number give_up_at is taken to have run out
    int recs;               // record buffers (1 or 2, set by the launcher)
    int ctas_per_sm;        // 0: as many as fit
    const int* skip;        // may be null: the pass does nothing when either of two words is not 0
    // set by the launcher
    int nchunk;
    int bs, bufc, acs;      // source block stride, one work buffer, accumulator mode stride (complex units)
    MmaSched sched;
};

// one CTA runs the kernel's bounded mbarrier wait on a barrier no copy completes
int launch_wait_selftest(int limit, int* err, cudaStream_t st);
// opoff[q] = q rec, and the pairs' descriptors from their spheres and slots
void launch_pair_offsets(int np, int rec, long long* opoff, int nsm, cudaStream_t st);
void launch_mma_pairs(int np, const int2* pairs, const uchar2* slots, const int* order, const int* offset, const long long* opoff,
                      MmaPair* out, int nsm, cudaStream_t st);
// 0: launched; -1: no configuration fits (order too large for shared memory)
int launch_translate_mma(MmaArgs& a, int nsm, cudaStream_t st);
// FP32 columns: xd = x and yd = 0; y = yd, or y += yd with `add` (an even number of values)
void launch_mma_widen(size_t values, const zf* x, zd* xd, zd* yd, int nsm, cudaStream_t st);
void launch_mma_narrow(size_t values, const zd* yd, zf* y, bool add, int nsm, cudaStream_t st);
