// ranorient.cuh -- orientation-averaged scattering matrix from the T matrix (ranorient.cu).
#pragma once
#include "common.cuh"
#include <cstddef>
#include <algorithm>

#define RO_NT 128
#define RO_ORDER_MAX 35   // largest T-matrix order taken

struct RoArgs {
    int nodr;              // T-matrix order
    float2* tc;            // nblkt x nblkt single-precision GB-modified T matrix
    zd* trace;             // 4 nodr: per-order traces (coherent part)
    zd* dm;                // ro_dm_elems(nodr), zeroed by the caller: [u][ku][n,p][n1,p1]
    zd* dmcf;
    zd* bg;                // bm of a chunk of items (ro_sizes)
    zd* bcf;               // coherent bm, all w
    zd* part;              // terms of the expansion coefficients per (w, n)
    int bgi;               // items bg has room for
    int vw0;               // first w of vtab
    double* vtab;          // vector-coupling rows of a chunk's w
    double* sm;            // 16 x (2 nodr + 1) expansion coefficients
    double* smcf;          // coherent part
    const double* bcof;    // bcof table (nbc + 1)^2
    const double* fnr;     // sqrt table
    int nbc;
    double rimed_re;
};

// elements of the workspaces
struct RoSizes {
    size_t bg, bcf, part, vtab;
    int bgi;
};
RoSizes ro_sizes(int nodr);
size_t ro_vtab_w(int nodr);
size_t ro_dm_elems(int nodr);
// returns -1 for orders above RO_ORDER_MAX
int launch_ranorient(const RoArgs& a, const zd* tmat, int nang, const double* bcofd, double* smat, int nsm, cudaStream_t st);
