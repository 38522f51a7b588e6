// capi_pass.cu -- the pair operators and the translation passes behind the C
// ABI: operator generation, the rotation kernels (tiles / order-generic), the
// tensor-core pass of many columns, the FFT path (node_selection, the kernel
// spectra and fft_external_to_external_expansion), sphereinteraction and the
// translation-pass entry points.
#include "ctx.cuh"

// ---------------------------------------------------------------------------
// operators and the translation pass
// ---------------------------------------------------------------------------
DenseArgs dense_args(mstmg_ctx* c)
{
    DenseArgs d;
    d.npairs = c->ndense;
    d.pairs = c->dpairs.p;
    d.order = c->d_order.p;
    d.offset = c->d_offset.p;
    d.pos = c->pos.p;
    d.off = c->doff.p;
    d.rec64 = nullptr;
    d.rec32 = nullptr;
    d.rimed_re = c->opts.medium_re;
    d.rimed_im = c->opts.medium_im;
    d.pmed = c->hs.on() ? c->hs.dmed.p : nullptr;
    d.g.tc = c->gt_tc.p;
    d.g.nmax = c->gt_nmax;
    d.g.nd = c->gt_nmax * (c->gt_nmax + 2);
    d.g.fnr = c->gt_fnr.p;
    d.g.bcd = c->gt_bcd.p;
    return d;
}

// Generate the stored pair operators a pass in FP64 (want64) or FP32 (want32)
// reads, those that are not there yet or with `force` all of them: the dense
// records of that precision, and the rotation records, which serve both.
int ensure_ops_both(mstmg_ctx* c, bool want64, bool want32, bool force)
{
    const bool dense64 = want64 && c->ndense > 0 && (force || !c->dense64_ready);
    const bool dense32 = want32 && c->ndense > 0 && (force || !c->dense32_ready);
    if (dense64 || dense32) {
        DenseArgs d = dense_args(c);
        const void* was[2] = {c->dop64.p, c->dop32.p};
        if (dense64) {
            CK(c->dop64.alloc(c->dense_units));
            d.rec64 = c->dop64.p;
        }
        if (dense32) {
            CK(c->dop32.alloc(c->dense_units));
            d.rec32 = c->dop32.p;
        }
        if (was[0] != c->dop64.p || was[1] != c->dop32.p) c->layout_gen++;
        launch_dense_gen(d, c->st);
        CK(cudaGetLastError());
        if (dense64) c->dense64_ready = true;
        if (dense32) c->dense32_ready = true;
    }
    if (c->npairs == 0 || !(want64 || want32) || (c->rot_ready && !force)) return MSTMG_OK;
    {
        const void* was = c->op64.p;
        cudaError_t e = c->op64.alloc(c->op_units);
        if (e != cudaSuccess && c->give_back()) {
            cudaGetLastError();
            e = c->op64.alloc(c->op_units);
        }
        CK(e);
        if (was != c->op64.p) c->layout_gen++;
    }
    NvtxRange nvtx_("pair operator generation");
    OpGenArgs a;
    a.npairs = c->npairs;
    a.pairs = c->pairs.p;
    a.pos = c->pos.p;
    a.order = c->d_order.p;
    a.opoff = c->opoff.p;
    a.op64 = c->op64.p;
    a.vcc = c->vcc.p;
    a.vnmax = c->vn;
    a.fnr = c->fnr.p;
    a.rfnr = c->rfnr.p;
    a.bcofd = c->bcofd.p;
    a.rimed_re = c->opts.medium_re;
    a.rimed_im = c->opts.medium_im;
    a.pmed = c->hs.on() ? c->hs.pmed.p : nullptr;
    a.err = c->err.p;
    CK(c->opgen_xi.alloc(opgen_xi_scratch(std::max(c->npairs, c->hs.nhp))));
    a.xi = c->opgen_xi.p;
    launch_opgen(a, c->nsm, c->st);
    CK(cudaGetLastError());
    if (c->hs.nhp > 0) {
        // regular translations between hosts and the spheres they hold, in
        // the host's index (external_to_internal_expansion, modules:6579-6592)
        HostSpheres& h = c->hs;
        CK(h.hop64.alloc(h.hunits));
        OpGenArgs b = a;
        b.npairs = h.nhp;
        b.pairs = h.hpairs.p;
        b.pos = h.xpos.p;
        b.opoff = h.hopoff.p;
        b.op64 = h.hop64.p;
        b.pmed = h.hmed.p;
        b.regular = 1;
        launch_opgen(b, c->nsm, c->st);
        CK(cudaGetLastError());
        h.hops_ready = true;
    }
    c->rot_ready = true;
    return MSTMG_OK;
}

// y[:, 0:nrhs] += the host-sphere couplings of x (external_to_internal_expansion)
template <typename T> int translate_hosts(mstmg_ctx* c, const cpx<T>* x, cpx<T>* y, int nrhs, unsigned contran)
{
    HostSpheres& h = c->hs;
    if (!h.on()) return MSTMG_OK;
    if (h.nhp > 0) {
        if (!h.hops_ready) {
            set_err("internal error: host-sphere operators not generated");
            return MSTMG_ERR_ARG;
        }
        TransArgs<T> a;
        a.npairs = h.nhp;
        a.pairs = h.hpairs.p;
        a.order = c->d_order.p;
        a.offset = c->d_offset.p;
        a.ops = h.hop64.p;
        a.opoff = h.hopoff.p;
        a.x = x;
        a.y = y;
        a.ld = c->neqns;
        a.nrhs = nrhs;
        a.contran = contran;
        a.lmax = h.hlmax;
        a.maxrec = h.hmaxrec;
        a.err = c->err.p;
        launch_translate<T>(a, c->nsm, c->st);
    }
    launch_mtransfer<T>(h.nzp, h.zpairs.p, c->d_order.p, c->d_offset.p, x, y, c->neqns, nrhs, c->st);
    CK(cudaGetLastError());
    return MSTMG_OK;
}
template int translate_hosts<double>(mstmg_ctx*, const zd*, zd*, int, unsigned);
template int translate_hosts<float>(mstmg_ctx*, const zf*, zf*, int, unsigned);

template <typename T> void mie_all(mstmg_ctx* c, int idir, int conj_in, const cpx<T>* x, cpx<T>* y)
{
    SlotMaps sm = c->sm();
    const bool d = sizeof(T) == 8;
    const cpx<T>* an = d ? (const cpx<T>*)c->an.p : (const cpx<T>*)c->an32.p;
    if (c->hs.on()) {
        const HostSpheres& h = c->hs;
        launch_hmie<T>(sm.nslots, c->n, sm.slot, sm.order, sm.offset, sm.mie_offset, h.d_hoff.p, an,
                       d ? (const cpx<T>*)h.dn.p : (const cpx<T>*)h.dn32.p, d ? (const cpx<T>*)h.un.p : (const cpx<T>*)h.un32.p,
                       d ? (const cpx<T>*)h.vn.p : (const cpx<T>*)h.vn32.p, idir, conj_in, x, y, c->st);
    } else {
        launch_mie<T>(sm.nslots, sm.slot, sm.order, sm.offset, sm.mie_offset, an, idir, conj_in, x, y, c->st);
    }
}
template void mie_all<double>(mstmg_ctx*, int, int, const zd*, zd*);
template void mie_all<float>(mstmg_ctx*, int, int, const zf*, zf*);

int ensure_ops(mstmg_ctx* c, int prec, bool force) { return ensure_ops_both(c, prec == 0, prec == 1, force); }

// FP64 copies of up to ncols FP32 columns for translate<float>; called ahead
// of a stream capture, which cannot allocate
int ensure_wide(mstmg_ctx* c, int ncols)
{
    std::lock_guard<std::recursive_mutex> lk(c->wide_mu);
    const size_t need = 2 * (size_t)c->neqns * ncols;
    if (c->tgroups_host.empty() || c->wide.n >= need) return MSTMG_OK;
    c->layout_gen++;
    CK(c->wide.alloc(need));
    return MSTMG_OK;
}

// y[:, 0:ncols] = H x[:, 0:ncols]  (y zeroed here); column k is a
// conjugate-transpose product when bit (k mod period) of contran is set
// (period 32, one bit a column, or 1, 2 or 4).  skip (may be null; tiles of
// pairs only): the pass is empty when either of two device words is not 0.
template <typename T> int translate(mstmg_ctx* c, const cpx<T>* x, cpx<T>* y, int ncols, unsigned contran, int period, const int* skip)
{
    NvtxRange nvtx_(sizeof(T) == 8 ? "translation pass FP64" : "translation pass FP32");
    const size_t ld = (size_t)c->neqns;
    const bool wide = sizeof(T) == 4 && !c->tgroups_host.empty();   // FP32 columns through the FP64 tiles
    const bool parts = c->hs.on() || c->ndense > 0;                 // contributions before the tiles'
    if (!wide || parts) CK(cudaMemsetAsync(y, 0, sizeof(cpx<T>) * ld * ncols, c->st));
    // the parts that take up to four columns a launch
    auto groups = [&](auto&& part) -> int {
        for (int k = 0; k < ncols; k += 4) {
            const int w = std::min(4, ncols - k);
            unsigned m = 0;
            for (int r = 0; r < w; r++) m |= ((contran >> ((k + r) % period)) & 1u) << r;
            if (int rc = part(x + k * ld, y + k * ld, w, m)) return rc;
        }
        return MSTMG_OK;
    };
    if (c->hs.on())
        if (int rh = groups([&](const cpx<T>* xk, cpx<T>* yk, int w, unsigned m) { return translate_hosts<T>(c, xk, yk, w, m); })) return rh;
    if (c->ndense > 0) {
        const T* drec = sizeof(T) == 8 ? (const T*)c->dop64.p : (const T*)c->dop32.p;
        groups([&](const cpx<T>* xk, cpx<T>* yk, int w, unsigned m) {
            launch_dense_apply<T>(dense_args(c), drec, xk, yk, c->neqns, w, m, c->st);
            return MSTMG_OK;
        });
        CK(cudaGetLastError());
    }
    // a sharded context: shard 0 adds the FFT path's far field, every shard its near-pair tiles
    const bool far = c->fft && c->fft->on && c->shard == 0;
    auto far_field = [&]() -> int {
        if (!far) return MSTMG_OK;
        return groups([&](const cpx<T>* xk, cpx<T>* yk, int w, unsigned m) { return fft_far<T>(c, xk, yk, w, m); });
    };
    if (c->npairs == 0) return far_field();
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (c->timing) {
        for (cudaEvent_t* ev : {&e0, &e1}) {
            if (!c->ev_pool.empty()) { *ev = c->ev_pool.back(); c->ev_pool.pop_back(); }
            else CK(cudaEventCreate(ev));
        }
        CK(cudaEventRecord(e0, c->st));
    }
    int rt = 0;
    if (!c->tgroups_host.empty()) {
        std::unique_lock<std::recursive_mutex> lk(c->wide_mu, std::defer_lock);
        if (sizeof(T) == 4) lk.lock();
        MmaArgs a;
        a.pairs = c->tpairs.p;
        a.tsph = c->tsph.p;
        a.order = c->d_order.p;
        a.offset = c->d_offset.p;
        a.ops = c->op64.p;
        if constexpr (sizeof(T) == 8) {
            a.x = x;
            a.y = y;
        } else {
            const size_t vals = ld * ncols;
            if (int rw = ensure_wide(c, ncols)) return rw;
            a.x = c->wide.p;
            a.y = c->wide.p + vals;
            launch_mma_widen(vals, x, c->wide.p, c->wide.p + vals, c->nsm, c->st);
        }
        a.ld = c->neqns;
        a.ncols = ncols;
        a.contran = contran;
        a.period = period;
        a.slots = c->tslots;
        a.err = c->err.p;
        a.give_up_at = c->give_up_at;
        a.ctas_per_sm = c->opts.tile_ctas_per_sm;
        a.skip = skip;
        for (const auto& g : c->tgroups) {
            if (g.count == 0) continue;
            a.ntiles = g.count;
            a.tiles = c->tiles.p + g.first;
            a.L = g.L;
            a.uniform = g.uniform;
            a.maxrec = g.maxrec;
            if ((rt = launch_translate_mma(a, c->nsm, c->st)) != 0) break;
        }
        if constexpr (sizeof(T) == 4) launch_mma_narrow(ld * ncols, a.y, y, parts, c->nsm, c->st);
    } else {
        TransArgs<T> a;
        a.npairs = c->npairs;
        a.pairs = c->pairs.p;
        a.order = c->d_order.p;
        a.offset = c->d_offset.p;
        a.ops = c->op64.p;
        a.opoff = c->opoff.p;
        a.ld = c->neqns;
        a.lmax = c->pair_lmax;
        a.uniform = c->pair_uniform ? 1 : 0;
        a.maxrec = c->maxrec;
        a.err = c->err.p;
        groups([&](const cpx<T>* xk, cpx<T>* yk, int w, unsigned m) {
            a.x = xk;
            a.y = yk;
            a.nrhs = w;
            a.contran = m;
            launch_translate<T>(a, c->nsm, c->st);
            return MSTMG_OK;
        });
    }
    if (rt != 0) {
        if (e0) c->ev_pool.push_back(e0);
        if (e1) c->ev_pool.push_back(e1);
        set_err("translation pass: no kernel configuration for this order");
        return MSTMG_ERR_UNSUPPORTED;
    }
    CK(cudaGetLastError());
    if (c->timing) {
        CK(cudaEventRecord(e1, c->st));
        c->pending.push_back({e0, e1, sizeof(T) == 8 ? 0 : 1});
    }
    if (sizeof(T) == 8) c->passes64++;
    else c->passes32++;
    return far_field();
}

// ---------------------------------------------------------------------------
// the tensor-core pass of many FP32 columns (tcpass.cu)
// ---------------------------------------------------------------------------

// One sphere order (5..10), pairs translated directly (no FFT, no dense
// pairs): the cases the dense TF32 images serve.
bool tc_eligible(const mstmg_ctx* c)
{
    if (c->opts.tensor_core < 0 || c->tc_state < 0 || c->nshards > 1 || c->hs.on()) return false;
    if (!c->tiled || c->ndense > 0 || (c->fft && c->fft->on) || c->npairs == 0) return false;
    return c->lmax >= 5 && tc_geom(c->lmax).NP <= 128;
}

// Build the dense operator images of every ordered pair (both directions of
// each pair of the context's list), unless they would take more than a third
// of the free device memory (the context then keeps the rotation kernels).
int ensure_tc(mstmg_ctx* c)
{
    if (c->tc_state == 1) return MSTMG_OK;
    if (!tc_eligible(c)) return MSTMG_ERR_UNSUPPORTED;
    NvtxRange nvtx_("tensor-core operator images");
    const TcGeom g = tc_geom(c->lmax);
    std::vector<int2> pr(c->npairs);
    CK(cudaMemcpyAsync(pr.data(), c->pairs.p, sizeof(int2) * c->npairs, cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    std::vector<std::vector<int>> nbr(c->n);
    for (const int2& q : pr) {
        nbr[q.x].push_back(q.y);
        nbr[q.y].push_back(q.x);
    }
    std::vector<int> rstart(c->n + 1, 0), rsrc;
    std::vector<int2> ent;
    rsrc.reserve(2 * (size_t)c->npairs);
    ent.reserve(2 * (size_t)c->npairs);
    for (int i = 0; i < c->n; i++) {
        std::sort(nbr[i].begin(), nbr[i].end());
        rstart[i] = (int)rsrc.size();
        for (int j : nbr[i]) {
            rsrc.push_back(j);
            ent.push_back(make_int2(i, j));
        }
    }
    rstart[c->n] = (int)rsrc.size();
    const size_t need = ent.size() * tc_himg_floats(g) * sizeof(float);
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    if (need > fr / 3 && c->give_back()) CK(cudaMemGetInfo(&fr, &tot));
    if (need > fr / 3) {
        c->tc_state = -1;
        set_err("tensor-core operator images (" + std::to_string(need >> 20) + " MiB) exceed a third of the free device memory");
        return MSTMG_ERR_UNSUPPORTED;
    }
    if (int rg = ensure_gentran(c, c->lmax)) return rg;
    const void* was = c->tc_h.p;
    CK(c->tc_h.alloc(ent.size() * tc_himg_floats(g)));
    CK(c->tc_ent.alloc(ent.size()));
    CK(c->tc_rstart.alloc(rstart.size()));
    CK(c->tc_rsrc.alloc(rsrc.size()));
    if (was != c->tc_h.p) c->layout_gen++;
    CK(cudaMemcpyAsync(c->tc_ent.p, ent.data(), sizeof(int2) * ent.size(), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(c->tc_rstart.p, rstart.data(), sizeof(int) * rstart.size(), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(c->tc_rsrc.p, rsrc.data(), sizeof(int) * rsrc.size(), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemsetAsync(c->tc_h.p, 0, need, c->st));   // the padded rows and sources stay zero
    TcGenArgs a;
    a.nent = (int)ent.size();
    a.ent = c->tc_ent.p;
    a.pos = c->pos.p;
    a.geo = g;
    a.rimed_re = c->opts.medium_re;
    a.rimed_im = c->opts.medium_im;
    a.g.tc = c->gt_tc.p;
    a.g.nmax = c->gt_nmax;
    a.g.nd = c->gt_nmax * (c->gt_nmax + 2);
    a.g.fnr = c->gt_fnr.p;
    a.g.bcd = c->gt_bcd.p;
    a.himg = c->tc_h.p;
    launch_tc_gen(a, c->st);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(c->st));   // the host vectors above are freed on return
    c->tc_nent = (int)ent.size();
    c->tc_state = 1;
    return MSTMG_OK;
}

// y[:, 0:ncols] = H x[:, 0:ncols] (no conjugate-transpose columns) on the
// tensor cores; y zeroed here
int tc_translate(mstmg_ctx* c, const zf* x, zf* y, int ncols)
{
    NvtxRange nvtx_("translation pass FP32 tensor cores");
    if (int rc = ensure_tc(c)) return rc;
    const TcGeom g = tc_geom(c->lmax);
    const int nmt = (ncols + TC_M - 1) / TC_M;
    const int mtn = tc_tiles_per_cta(g, nmt);
    const void* was = c->tc_a.p;
    CK(c->tc_a.alloc((size_t)((nmt + mtn - 1) / mtn * mtn) * c->n * tc_aimg_floats(g)));
    if (was != c->tc_a.p) c->layout_gen++;
    CK(cudaMemsetAsync(y, 0, sizeof(zf) * (size_t)c->neqns * ncols, c->st));
    TcPassArgs a;
    a.nsph = c->n;
    a.geo = g;
    a.ld = c->neqns;
    a.ncols = ncols;
    a.nmt = nmt;
    a.rstart = c->tc_rstart.p;
    a.rsrc = c->tc_rsrc.p;
    a.nent = c->tc_nent;
    a.himg = c->tc_h.p;
    a.aimg = c->tc_a.p;
    a.x = x;
    a.y = y;
    a.err = c->err.p;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (c->timing) {
        for (cudaEvent_t* ev : {&e0, &e1}) {
            if (!c->ev_pool.empty()) { *ev = c->ev_pool.back(); c->ev_pool.pop_back(); }
            else CK(cudaEventCreate(ev));
        }
        CK(cudaEventRecord(e0, c->st));
    }
    if (launch_tc_pass(a, c->nsm, c->st) != 0) {
        if (e0) c->ev_pool.push_back(e0);
        if (e1) c->ev_pool.push_back(e1);
        set_err("tensor-core pass: unsupported geometry");
        return MSTMG_ERR_UNSUPPORTED;
    }
    CK(cudaGetLastError());
    if (c->timing) {
        CK(cudaEventRecord(e1, c->st));
        c->pending.push_back({e0, e1, 2});
    }
    c->passes32++;
    c->tc_passes++;
    return MSTMG_OK;
}

// Many columns: y[:, 0:ncols] = H x[:, 0:ncols], where column k is a
// conjugate-transpose product when bit (k & 1) of pattern2 is set (BiCG packs
// [p_1, w_1, p_2, w_2, ...]: pattern2 = 2).
template <typename T> int translate_many(mstmg_ctx* c, const cpx<T>* x, cpx<T>* y, int ncols, unsigned pattern2)
{
    if constexpr (sizeof(T) == 4) {
        // many plain columns: the tensor-core pass when the context has (or can
        // build) its dense operator images
        if (pattern2 == 0 && ncols >= TC_MIN_COLS && tc_eligible(c)) {
            int rc = tc_translate(c, x, y, ncols);
            if (rc != MSTMG_ERR_UNSUPPORTED) return rc;
        }
    }
    return translate<T>(c, x, y, ncols, pattern2, 2);
}

int interaction_impl(mstmg_ctx* c, int nrhs, const double* ain, double* aout, const int* con_tran, const int* mie_mult,
                            int initial_run, const int* rhs_list, int skip_external)
{
    if (!c || nrhs < 1 || nrhs > 4 || !ain || !aout) {
        set_err("mstmg_interaction: bad arguments (nrhs must be 1..4)");
        return MSTMG_ERR_ARG;
    }
    int rc = skip_external ? MSTMG_OK : ensure_ops(c, 0, initial_run != 0);
    if (rc) return rc;
    const int ne = c->neqns;
    unsigned mask = 0;
    CK(copy_in(c->X64.p, ain, sizeof(zd) * (size_t)ne * nrhs, c->st));
    // columns left out of rhs_list are not translated: their output is zero
    if (rhs_list)
        for (int r = 0; r < nrhs; r++)
            if (!rhs_list[r]) CK(cudaMemsetAsync(c->X64.p + (size_t)r * ne, 0, sizeof(zd) * ne, c->st));
    for (int r = 0; r < nrhs; r++) {
        int ct = con_tran ? con_tran[r] : 0;
        int mm = mie_mult ? mie_mult[r] : 1;
        zd* col = c->X64.p + (size_t)r * ne;
        if (ct) {
            mask |= 1u << r;
            if (mm) mie_all<double>(c, -1, 1, col, col);
            else launch_conj_copy<double>(ne, col, col, c->st);
        }
    }
    if (skip_external) {
        // no pair translation: only the host-sphere couplings (none without
        // host spheres; no plane boundaries on this path)
        CK(cudaMemsetAsync(c->Y64.p, 0, sizeof(zd) * (size_t)ne * nrhs, c->st));
        if (c->hs.on()) {
            rc = ensure_ops(c, 0, initial_run != 0);
            if (rc) return rc;
            rc = translate_hosts<double>(c, c->X64.p, c->Y64.p, nrhs, mask);
            if (rc) return rc;
        }
    } else {
        rc = translate<double>(c, c->X64.p, c->Y64.p, nrhs, mask);
        if (rc) return rc;
    }
    for (int r = 0; r < nrhs; r++) {
        int ct = con_tran ? con_tran[r] : 0;
        int mm = mie_mult ? mie_mult[r] : 1;
        zd* col = c->Y64.p + (size_t)r * ne;
        if (!ct) {
            if (mm) mie_all<double>(c, 1, 0, col, col);
        } else {
            launch_conj_copy<double>(ne, col, col, c->st);
        }
    }
    CK(cudaGetLastError());
    CK(copy_out(aout, c->Y64.p, sizeof(zd) * (size_t)ne * nrhs, c->st));
    CK(cudaStreamSynchronize(c->st));
    return check_kernel_err(c);
}

extern "C" int mstmg_interaction(mstmg_ctx* c, int nrhs, const double* ain, double* aout, const int* con_tran, const int* mie_mult,
                                 int initial_run)
{
    NvtxRange nvtx_("mstmg_interaction");
    return interaction_impl(c, nrhs, ain, aout, con_tran, mie_mult, initial_run, nullptr, 0);
}

extern "C" int mstmg_interaction_ex(mstmg_ctx* c, int nrhs, const double* ain, double* aout, const int* con_tran, const int* mie_mult,
                                    int initial_run, const int* rhs_list, int fft_option, int store_matrix_option,
                                    int skip_external_translation)
{
    NvtxRange nvtx_("mstmg_interaction_ex");
    if (!c) return MSTMG_ERR_ARG;
    const bool fft_on = c->fft && c->fft->on;
    if ((fft_option == 1 && !fft_on) || (fft_option == 0 && fft_on)) {
        set_err("mstmg_interaction_ex: fft_option differs from the context's set-up (mstmg_fft_setup decides it per context)");
        return MSTMG_ERR_UNSUPPORTED;
    }
    (void)store_matrix_option;   // the pair operators are always stored
    return interaction_impl(c, nrhs, ain, aout, con_tran, mie_mult, initial_run, rhs_list, skip_external_translation);
}

// ---------------------------------------------------------------------------
// FFT translation (fft_translation-5.f90)
// ---------------------------------------------------------------------------

static int check235(int n) /* fft:1052-1066 */
{
    int nn = n, ifac = 2;
    for (int ll = 1; ll <= 3; ll++) {
        while (nn % ifac == 0) nn /= ifac;
        ifac += ll;
    }
    return nn == 1;
}
static int correct235(int n) /* fft:1068-1076 (n >= 1: a flat extent gives one cell) */
{
    int n1 = n < 1 ? 1 : n;
    while (!check235(n1)) n1++;
    return n1;
}

// Far part: y += S Jns conv(Jsn S x) for up to 4 columns per pass.
template <typename T> int fft_far(mstmg_ctx* c, const cpx<T>* x, cpx<T>* y, int ncols, unsigned contran)
{
    FftState& F = *c->fft;
    const int pi = sizeof(T) == 8 ? 0 : 1;
    const size_t per = (size_t)2 * F.nbN * F.N8;
    DevBuf<cpx<T>>& A = *reinterpret_cast<DevBuf<cpx<T>>*>(sizeof(T) == 8 ? (void*)&F.A64 : (void*)&F.A32);
    DevBuf<cpx<T>>& G = *reinterpret_cast<DevBuf<cpx<T>>*>(sizeof(T) == 8 ? (void*)&F.G64 : (void*)&F.G32);
    const cpx<T>* Jsn = sizeof(T) == 8 ? (const cpx<T>*)F.Jsn64.p : (const cpx<T>*)F.Jsn32.p;
    const cpx<T>* Jns = sizeof(T) == 8 ? (const cpx<T>*)F.Jns64.p : (const cpx<T>*)F.Jns32.p;
    if (!Jsn || !Jns) {
        set_err("FFT translation: node translations missing for this precision");
        return MSTMG_ERR_CUDA;
    }
    CK(A.alloc(4 * per));
    CK(G.alloc(4 * per));
    FftMArgs m;
    m.nsph = c->n;
    m.No = F.No;
    m.nbmax = c->lmax * (c->lmax + 2);
    m.N8 = F.N8;
    m.order = c->d_order.p;
    m.offset = c->d_offset.p;
    m.joff = F.joff.p;
    m.slot = F.slot.p;
    const size_t ld = (size_t)c->neqns;
    for (int k0 = 0; k0 < ncols; k0 += 4) {
        const int w = std::min(4, ncols - k0);
        const unsigned mask = (contran >> k0) & 0xFu;
        if (!F.have[pi][w]) {
            int nn[3] = {2 * F.cd[2], 2 * F.cd[1], 2 * F.cd[0]};
            if (cufftPlanMany(&F.plan[pi][w], 3, nn, nullptr, 1, (int)F.N8, nullptr, 1, (int)F.N8, sizeof(T) == 8 ? CUFFT_Z2Z : CUFFT_C2C,
                              w * 2 * F.nbN) != CUFFT_SUCCESS) {
                set_err("FFT translation: cufftPlanMany failed");
                return MSTMG_ERR_CUDA;
            }
            F.have[pi][w] = true;
        }
        cufftSetStream(F.plan[pi][w], c->st);
        CK(cudaMemsetAsync(A.p, 0, sizeof(cpx<T>) * w * per, c->st));
        launch_fft_s2n<T>(m, Jsn, x + (size_t)k0 * ld, (int)ld, w, mask, A.p, c->st);
        cufftResult fr;
        if (sizeof(T) == 8) fr = cufftExecZ2Z(F.plan[pi][w], (cufftDoubleComplex*)A.p, (cufftDoubleComplex*)A.p, CUFFT_FORWARD);
        else fr = cufftExecC2C(F.plan[pi][w], (cufftComplex*)A.p, (cufftComplex*)A.p, CUFFT_FORWARD);
        if (fr != CUFFT_SUCCESS) {
            set_err("FFT translation: forward transform failed");
            return MSTMG_ERR_CUDA;
        }
        launch_fft_mul<T>(F.nbN, F.N8, w, F.H.p, A.p, G.p, c->st);
        if (sizeof(T) == 8) fr = cufftExecZ2Z(F.plan[pi][w], (cufftDoubleComplex*)G.p, (cufftDoubleComplex*)G.p, CUFFT_INVERSE);
        else fr = cufftExecC2C(F.plan[pi][w], (cufftComplex*)G.p, (cufftComplex*)G.p, CUFFT_INVERSE);
        if (fr != CUFFT_SUCCESS) {
            set_err("FFT translation: inverse transform failed");
            return MSTMG_ERR_CUDA;
        }
        launch_fft_n2s<T>(m, Jns, G.p, w, mask, y + (size_t)k0 * ld, (int)ld, c->st);
        CK(cudaGetLastError());
    }
    return MSTMG_OK;
}

// Tiles of a given pair list: the spheres of `members`, in that order, form
// groups; a tile holds the pairs of pr between two groups or inside one.
int group_tiles(mstmg_ctx* c, const std::vector<int>& members, const std::vector<int2>& pr, TileSet& t)
{
    const int n = c->n;
    int pl = 1;
    for (const int2& q : pr) pl = std::max(pl, std::max(c->order[q.x], c->order[q.y]));
    const int B = tile_group_size(c, (long long)pr.size(), pl);
    std::vector<int> grp(n, -1), gs(n, 0);
    for (size_t k = 0; k < members.size(); k++) {
        grp[members[k]] = (int)(k / B);
        gs[members[k]] = (int)(k % B);
    }
    const long long ng = ((long long)members.size() + B - 1) / B;
    std::vector<long long> key(pr.size());
    std::vector<int> idx(pr.size());
    for (size_t q = 0; q < pr.size(); q++) {
        if (grp[pr[q].x] < 0 || grp[pr[q].y] < 0) {
            set_err("internal error: a pair's sphere is in no tile group");
            return MSTMG_ERR_ARG;
        }
        const long long ga = std::min(grp[pr[q].x], grp[pr[q].y]), gb = std::max(grp[pr[q].x], grp[pr[q].y]);
        key[q] = ga * ng + gb;
        idx[q] = (int)q;
    }
    std::stable_sort(idx.begin(), idx.end(), [&](int u, int v) { return key[u] < key[v]; });
    t = TileSet();
    t.slots = 2 * B;
    t.pr.resize(pr.size());
    t.ps.resize(pr.size());
    for (size_t q = 0; q < idx.size();) {
        const long long kk = key[idx[q]];
        const int ga = (int)(kk / ng);
        const size_t start = q, row = t.ts.size();
        t.ts.resize(row + t.slots, -1);
        for (; q < idx.size() && key[idx[q]] == kk; q++) {
            const int2 p2 = pr[idx[q]];
            const unsigned char si = (unsigned char)(grp[p2.x] == ga ? gs[p2.x] : B + gs[p2.x]);
            const unsigned char sj = (unsigned char)(grp[p2.y] == ga ? gs[p2.y] : B + gs[p2.y]);
            t.pr[q] = p2;
            t.ps[q] = make_uchar2(si, sj);
            t.ts[row + si] = p2.x;
            t.ts[row + sj] = p2.y;
        }
        t.tl.push_back(make_int4((int)start, (int)(q - start), (int)t.tl.size(), 0));
    }
    return MSTMG_OK;
}

// node_selection (fft:654-825) with target box = the sphere-centre extents,
// the near-pair list, the node translations and the kernel spectra.
int fft_build(mstmg_ctx* c)
{
    FftState& F = *c->fft;
    const int n = c->n;
    double tmin[3] = {1e10, 1e10, 1e10}, tmax[3] = {-1e10, -1e10, -1e10};
    for (int i = 0; i < n; i++)
        for (int m = 0; m < 3; m++) {
            tmin[m] = std::min(tmin[m], c->hpos[3 * (size_t)i + m]);
            tmax[m] = std::max(tmax[m], c->hpos[3 * (size_t)i + m]);
        }
    double amean = 0.0, svol = 0.0;
    for (int i = 0; i < n; i++) {
        amean += c->radius[i];
        svol += c->radius[i] * c->radius[i] * c->radius[i];
    }
    svol = std::pow(svol, 1.0 / 3.0);
    amean = amean / (double)n;
    double tvol = 1.0;
    for (int m = 0; m < 3; m++) tvol *= std::max(tmax[m] - tmin[m], amean);
    double dc = F.d_in;
    if (!(F.d_in > 0.0)) {
        double fv = F.fv_in;
        if (fv <= 0.0) {
            fv = 4.0 * MSTMG_REF_PI / 3.0 * svol * svol * svol / tvol;
            fv = std::min(fv, 1.0);
            fv = std::max(fv, 0.02);
        }
        dc = std::pow(4.0 * MSTMG_REF_PI / 3.0 / fv / (double)n, 1.0 / 3.0) * svol;
    }
    for (int m = 0; m < 3; m++) F.cd[m] = correct235((int)std::ceil((tmax[m] - tmin[m]) / dc));
    dc = 0.0;
    for (int m = 0; m < 3; m++) dc = std::max(dc, (tmax[m] - tmin[m]) / (double)F.cd[m]);
    F.dcell = dc;
    for (int m = 0; m < 3; m++) F.cb[m] = tmin[m];
    F.No = F.no_in > 0 ? F.no_in : -F.no_in + (int)std::ceil(dc);
    F.nbN = F.No * (F.No + 2);
    if (F.No < 1 || F.nbN > FFT_NBN_MAX || 2 * F.No > GT_WMAX || F.No + c->lmax > GT_WMAX) {
        set_err("FFT translation: node order out of range (1..20)");
        return MSTMG_ERR_UNSUPPORTED;
    }
    if (c->ndense > 0) {
        set_err("FFT translation: spheres below translation_switch_order are not supported on this path");
        return MSTMG_ERR_UNSUPPORTED;
    }
    F.N8 = (size_t)8 * F.cd[0] * F.cd[1] * F.cd[2];
    const double hr_bytes = 16.0 * 2.0 * F.nbN * F.nbN * (double)F.N8;
    if (hr_bytes > 16.0e9) {
        set_err("FFT translation: kernel table above 16 GB (grid or node order too large)");
        return MSTMG_ERR_UNSUPPORTED;
    }
    // cells of the spheres, stencil, near pairs (j > i in neighbouring cells, the reference's order)
    std::vector<int> snode(3 * (size_t)n), slot(n);
    const int N0 = 2 * F.cd[0], N1 = 2 * F.cd[1];
    std::vector<std::vector<int>> members((size_t)F.cd[0] * F.cd[1] * F.cd[2]);
    for (int i = 0; i < n; i++) {
        int cc[3];
        for (int m = 0; m < 3; m++) {
            int nd = (int)std::floor((c->hpos[3 * (size_t)i + m] - tmin[m]) / dc) + 1;
            nd = std::min(nd, F.cd[m]);
            cc[m] = std::max(nd, 1);
            snode[3 * (size_t)i + m] = cc[m];
        }
        slot[i] = (cc[0] - 1) + N0 * ((cc[1] - 1) + N1 * (cc[2] - 1));
        members[(size_t)(cc[0] - 1) + (size_t)F.cd[0] * ((cc[1] - 1) + (size_t)F.cd[1] * (cc[2] - 1))].push_back(i);
    }
    F.nnb = 0;
    for (int iz = -1; iz <= 1; iz++)
        for (int iy = -1; iy <= 1; iy++)
            for (int ix = -1; ix <= 1; ix++) {
                int ir = ix * ix + iy * iy + iz * iz;
                if ((F.model_in == 0 && ir > 0) || (F.model_in == 1 && ir > 1) || (F.model_in == 2 && ir > 2)) continue;
                F.nbv[3 * F.nnb] = ix;
                F.nbv[3 * F.nnb + 1] = iy;
                F.nbv[3 * F.nnb + 2] = iz;
                F.nnb++;
            }
    std::vector<int2> pr;
    for (int i = 0; i < n; i++)
        for (int q = 0; q < F.nnb; q++) {
            int sx = snode[3 * (size_t)i] - F.nbv[3 * q], sy = snode[3 * (size_t)i + 1] - F.nbv[3 * q + 1], sz = snode[3 * (size_t)i + 2] - F.nbv[3 * q + 2];
            if (sx < 1 || sy < 1 || sz < 1 || sx > F.cd[0] || sy > F.cd[1] || sz > F.cd[2]) continue;
            for (int j : members[(size_t)(sx - 1) + (size_t)F.cd[0] * ((sy - 1) + (size_t)F.cd[1] * (sz - 1))])
                if (j > i) pr.push_back(make_int2(i, j));
        }
    // Tiles of the near pairs: the spheres, taken cell by cell, form the
    // groups, so the near pairs of nearby spheres share the tiles' output
    // accumulation as the tiles of a whole cluster do.
    const int lmin = *std::min_element(c->order.begin(), c->order.end());
    c->tiled = !c->opts.generic_kernel && lmin == c->lmax && lmin >= c->opts.translation_switch_order && tiled_order(c->lmax) && !pr.empty();
    TileSet ts;
    if (!c->opts.generic_kernel) {
        std::vector<int> flat;
        for (const auto& cm : members) flat.insert(flat.end(), cm.begin(), cm.end());
        if (int rg = group_tiles(c, flat, pr, ts)) return rg;
        pr.swap(ts.pr);
    }
    int rc = upload_pairs(c, pr, (int)pr.size(), c->opts.generic_kernel ? nullptr : &ts);   // synchronises: the host vectors above are done with
    if (rc) return rc;
    // node translations
    std::vector<long long> joff(n + 1);
    long long tot = 0;
    for (int i = 0; i < n; i++) {
        joff[i] = tot;
        tot += 2LL * F.nbN * c->order[i] * (c->order[i] + 2);
    }
    joff[n] = tot;
    CK(F.snode.alloc(3 * (size_t)n));
    CK(F.slot.alloc(n));
    CK(F.joff.alloc(n + 1));
    CK(cudaMemcpyAsync(F.snode.p, snode.data(), sizeof(int) * 3 * n, cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(F.slot.p, slot.data(), sizeof(int) * n, cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(F.joff.p, joff.data(), sizeof(long long) * (n + 1), cudaMemcpyHostToDevice, c->st));
    const int nmax = std::max(F.No, c->lmax);
    std::vector<double> tcv, bd(GT_WMAX + 2);
    gentran_constants(nmax, tcv);
    mstmg::Tables& big = big_tables();
    for (int k = 0; k < (int)bd.size(); k++) bd[k] = big.bc(k, k);
    DevBuf<double> dtc, dbd, dfnr;
    CK(dtc.alloc(tcv.size()));
    CK(dbd.alloc(bd.size()));
    CK(dfnr.alloc(big.fnr.size()));
    CK(cudaMemcpyAsync(dtc.p, tcv.data(), sizeof(double) * tcv.size(), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(dbd.p, bd.data(), sizeof(double) * bd.size(), cudaMemcpyHostToDevice, c->st));
    CK(cudaMemcpyAsync(dfnr.p, big.fnr.data(), sizeof(double) * big.fnr.size(), cudaMemcpyHostToDevice, c->st));
    GtConst g;
    g.tc = dtc.p;
    g.nmax = nmax;
    g.nd = nmax * (nmax + 2);
    g.fnr = dfnr.p;
    g.bcd = dbd.p;
    CK(F.Jsn64.alloc(tot));
    CK(F.Jns64.alloc(tot));
    FftJArgs ja;
    ja.nsph = n;
    ja.No = F.No;
    ja.order = c->d_order.p;
    ja.pos = c->pos.p;
    ja.snode = F.snode.p;
    ja.dcell = dc;
    for (int m = 0; m < 3; m++) ja.cb[m] = F.cb[m];
    ja.joff = F.joff.p;
    ja.Jsn = F.Jsn64.p;
    ja.Jns = F.Jns64.p;
    ja.rimed_re = c->opts.medium_re;
    ja.rimed_im = c->opts.medium_im;
    ja.g = g;
    launch_fft_j(ja, c->st);
    CK(cudaGetLastError());
    CK(F.Jsn32.alloc(tot));
    CK(F.Jns32.alloc(tot));
    launch_d2f((int)tot, F.Jsn64.p, F.Jsn32.p, c->st);
    launch_d2f((int)tot, F.Jns64.p, F.Jns32.p, c->st);
    // kernel spectra: real-space kernels (single-precision sums), double FFT, stored in single precision
    {
        DevBuf<zd> hr;
        const size_t nel = (size_t)2 * F.nbN * F.nbN;
        CK(hr.alloc(nel * F.N8));
        FftHArgs ha;
        for (int m = 0; m < 3; m++) ha.cd[m] = F.cd[m];
        ha.No = F.No;
        ha.nnb = F.nnb;
        for (int q = 0; q < 81; q++) ha.nbv[q] = F.nbv[q];
        ha.dcell = dc;
        ha.rimed_re = c->opts.medium_re;
        ha.rimed_im = c->opts.medium_im;
        ha.hr = hr.p;
        ha.g = g;
        launch_fft_hbuild(ha, c->nsm, c->st);
        CK(cudaGetLastError());
        cufftHandle hp;
        int nn[3] = {2 * F.cd[2], 2 * F.cd[1], 2 * F.cd[0]};
        // in batches of at most 1225 transforms (one mode of a node order 5 kernel)
        const int chunk = std::min<int>((int)nel, F.nbN * F.nbN);
        if (cufftPlanMany(&hp, 3, nn, nullptr, 1, (int)F.N8, nullptr, 1, (int)F.N8, CUFFT_Z2Z, chunk) != CUFFT_SUCCESS) {
            set_err("FFT translation: kernel plan failed");
            return MSTMG_ERR_CUDA;
        }
        cufftSetStream(hp, c->st);
        bool ok = true;
        for (size_t b = 0; b + (size_t)chunk <= nel && ok; b += chunk)
            ok = cufftExecZ2Z(hp, (cufftDoubleComplex*)(hr.p + b * F.N8), (cufftDoubleComplex*)(hr.p + b * F.N8), CUFFT_FORWARD) == CUFFT_SUCCESS;
        cufftDestroy(hp);
        if (!ok) {
            set_err("FFT translation: kernel transform failed");
            return MSTMG_ERR_CUDA;
        }
        CK(F.H.alloc(nel * F.N8));
        launch_fft_round(nel * F.N8, hr.p, F.H.p, c->st);
        CK(cudaGetLastError());
        CK(cudaStreamSynchronize(c->st));
    }
    F.on = true;
    return check_kernel_err(c);
}

extern "C" int mstmg_fft_setup(mstmg_ctx* c, double cell_volume_fraction, double d_cell, int node_order, int neighbor_node_model,
                               int* cell_dim, double* d_cell_out, int* node_order_out, int* near_pairs)
{
    if (int rc0 = reject_ensemble(c, "mstmg_fft_setup")) return rc0;
    if (int rh = reject_hosts(c, "mstmg_fft_setup")) return rh;
    NvtxRange nvtx_("mstmg_fft_setup");
    if (!c || c->n < 2 || neighbor_node_model < 0 || neighbor_node_model > 2) {
        set_err("mstmg_fft_setup: bad arguments (two or more spheres, neighbor_node_model 0..2)");
        return MSTMG_ERR_ARG;
    }
    if (!c->fft) c->fft.reset(new FftState());
    FftState& F = *c->fft;
    F.drop_plans();
    F.on = false;
    F.fv_in = cell_volume_fraction;
    F.d_in = d_cell;
    F.no_in = node_order;
    F.model_in = neighbor_node_model;
    int rc = fft_build(c);
    if (rc) return rc;
    if (cell_dim)
        for (int m = 0; m < 3; m++) cell_dim[m] = F.cd[m];
    if (d_cell_out) *d_cell_out = F.dcell;
    if (node_order_out) *node_order_out = F.No;
    if (near_pairs) *near_pairs = c->npairs;
    return MSTMG_OK;
}

extern "C" int mstmg_translation_pass(mstmg_ctx* c, int prec, int ncols, const int* con_tran, const double* x, double* y)
{
    NvtxRange nvtx_("mstmg_translation_pass");
    if (!c || ncols < 1 || ncols > 256 || !x || !y || prec < 0 || prec > 2) {
        set_err("mstmg_translation_pass: bad arguments");
        return MSTMG_ERR_ARG;
    }
    if (prec == 2) {   // the tensor-core pass, required
        for (int k = 0; con_tran && k < ncols; k++)
            if (con_tran[k]) {
                set_err("mstmg_translation_pass: the tensor-core pass takes no conjugate-transpose columns");
                return MSTMG_ERR_UNSUPPORTED;
            }
        if (!tc_eligible(c)) {
            set_err("mstmg_translation_pass: no tensor-core pass for this context (one sphere order 5..10, direct pairs)");
            return MSTMG_ERR_UNSUPPORTED;
        }
    }
    int rc = prec == 2 ? MSTMG_OK : ensure_ops(c, prec, false);
    if (rc) return rc;
    const size_t ne = (size_t)c->neqns, cols = ne * ncols;
    // a period-2 con_tran pattern goes through the many-column path; anything
    // else in groups of up to 4 columns with their own masks
    bool per2 = true;
    for (int k = 2; k < ncols; k++) per2 = per2 && ((con_tran ? con_tran[k] != 0 : false) == (con_tran ? con_tran[k - 2] != 0 : false));
    unsigned pattern2 = 0;
    if (con_tran && con_tran[0]) pattern2 |= 1u;
    if (con_tran && ncols > 1 && con_tran[1]) pattern2 |= 2u;
    DevBuf<zd> x64, y64;
    CK(x64.alloc(cols));
    CK(y64.alloc(cols));
    CK(copy_in(x64.p, x, sizeof(zd) * cols, c->st));
    auto groups = [&](auto* xp, auto* yp) -> int {
        using TT = std::remove_pointer_t<decltype(xp)>;
        using T = decltype(TT::x);
        if (per2) return translate_many<T>(c, xp, yp, ncols, pattern2);
        for (int k = 0; k < ncols; k += 4) {
            int w = std::min(4, ncols - k);
            unsigned m = 0;
            for (int r = 0; r < w; r++)
                if (con_tran && con_tran[k + r]) m |= 1u << r;
            int rr = translate<T>(c, xp + k * ne, yp + k * ne, w, m);
            if (rr) return rr;
        }
        return MSTMG_OK;
    };
    if (prec == 0) {
        if ((rc = groups(x64.p, y64.p))) return rc;
    } else {
        DevBuf<zf> x32, y32;
        CK(x32.alloc(cols));
        CK(y32.alloc(cols));
        launch_d2f((int)cols, x64.p, x32.p, c->st);
        if (prec == 2) rc = tc_translate(c, x32.p, y32.p, ncols);
        else rc = groups(x32.p, y32.p);
        if (rc) return rc;
        CK(cudaMemsetAsync(y64.p, 0, sizeof(zd) * cols, c->st));
        launch_add_correction_f((int)cols, y64.p, y32.p, c->st);
        CK(cudaGetLastError());
        CK(copy_out(y, y64.p, sizeof(zd) * cols, c->st));
        CK(cudaStreamSynchronize(c->st));
        return check_kernel_err(c);
    }
    CK(copy_out(y, y64.p, sizeof(zd) * cols, c->st));
    CK(cudaStreamSynchronize(c->st));
    return check_kernel_err(c);
}

extern "C" int mstmg_selftest_pass_wait(mstmg_ctx* c, int pair, int ncols, const int* con_tran, const double* x, double* y, int* status)
{
    if (!c || !status || pair < 0) {
        set_err("mstmg_selftest_pass_wait: bad arguments");
        return MSTMG_ERR_ARG;
    }
    if (c->tgroups_host.empty()) {
        set_err("mstmg_selftest_pass_wait: no pairs on tiles in this context");
        return MSTMG_ERR_UNSUPPORTED;
    }
    c->give_up_at = pair;
    const int rc = mstmg_translation_pass(c, 0, ncols, con_tran, x, y);
    c->give_up_at = -1;
    *status = rc;
    // a wait that gave up leaves the device as it was; any other CUDA error does not
    CK(cudaStreamSynchronize(c->st));
    return rc == MSTMG_ERR_CUDA ? MSTMG_OK : rc;
}

extern "C" int mstmg_time_translation(mstmg_ctx* c, int prec, int nrhs, int reps, double* ms)
{
    if (!c || nrhs < 1 || nrhs > 256 || reps < 1 || prec < 0 || prec > 2) return MSTMG_ERR_ARG;
    if (prec == 2 && !tc_eligible(c)) {
        set_err("mstmg_time_translation: no tensor-core pass for this context");
        return MSTMG_ERR_UNSUPPORTED;
    }
    int rc = prec == 2 ? ensure_tc(c) : ensure_ops(c, prec, false);
    if (rc) return rc;
    DevBuf<zd> x64, y64;
    DevBuf<zf> x32, y32;
    const size_t cols = (size_t)c->neqns * nrhs;
    if (prec == 0) {
        CK(x64.alloc(cols));
        CK(y64.alloc(cols));
        CK(cudaMemsetAsync(x64.p, 0, sizeof(zd) * cols, c->st));
    } else {
        CK(x32.alloc(cols));
        CK(y32.alloc(cols));
        CK(cudaMemsetAsync(x32.p, 0, sizeof(zf) * cols, c->st));
    }
    auto pass = [&]() -> int {
        if (prec == 0) return translate_many<double>(c, x64.p, y64.p, nrhs, nrhs >= 2 ? 2u : 0u);
        if (prec == 2) return tc_translate(c, x32.p, y32.p, nrhs);   // plain columns on the tensor cores
        return translate_many<float>(c, x32.p, y32.p, nrhs, nrhs >= 2 ? 2u : 0u);
    };
    if ((rc = pass())) return rc;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    CK(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        set_err("mstmg_time_translation: cudaEventCreate failed");
        return MSTMG_ERR_CUDA;
    }
    cudaEventRecord(e0, c->st);
    for (int k = 0; k < reps && rc == 0; k++) rc = pass();
    cudaEventRecord(e1, c->st);
    cudaError_t es = cudaEventSynchronize(e1);
    float t = 0.f;
    if (es == cudaSuccess) es = cudaEventElapsedTime(&t, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    CK(es);
    if (ms) *ms = t / reps;
    return check_kernel_err(c);
}

template int translate<float>(mstmg_ctx*, const zf*, zf*, int, unsigned, int, const int*);
template int translate<double>(mstmg_ctx*, const zd*, zd*, int, unsigned, int, const int*);
template int translate_many<float>(mstmg_ctx*, const zf*, zf*, int, unsigned);
template int translate_many<double>(mstmg_ctx*, const zd*, zd*, int, unsigned);
