// Batched plain CF solver: many instances (cosmology x source redshift x closure) with uneven plane
// counts and k grids, solved by one persistent launch, then inverted to dP/dln mu.  The device work
// list, the tile autotuner and the CUDA-graph capture of a whole step live here; the kernels are in
// cfbatch.cu.
//
// No counterpart in the reference, which solves one pipeline.run per instance
// (pipeline.py:114-274).
#include <chrono>
#include <cmath>
#include <numeric>

#include "host.cuh"

struct CfbState {
    int n_inst = 0, n_planes = 0, nstate = 0;
    int shape_class = 0;                       // log2 buckets of the largest k grid and the mean cells
    long long n_cells = 0, total_k = 0;
    int nm = 0, nb = 0;                        // template planes: the cells' forms present on the device
    bool have[2] = {true, true};               // (filled per precision on first use)
    std::vector<CfbInst> inst;
    std::vector<double> cost;                  // per instance: cells x k (+ chain) work
    std::vector<int> order;                    // instances by cost, longest first
    // tuned launch shape per precision: k-points per work item (= threads per CTA), CTAs per SM
    int kt[2] = {128, 128}, cps[2] = {0, 0};
    bool tuned[2] = {false, false};
    // the captured step per (precision, n_lnmu) and its item list
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    int graph_nm[2] = {0, 0}, graph_kt[2] = {0, 0}, graph_cps[2] = {0, 0};
};

void cfb_state_free(CfbState* s) {
    if (!s) return;
    for (auto& g : s->graph) if (g) cudaGraphExecDestroy(g);
    delete s;
}

int cfb_n_inst(const CfbState* s) { return s ? s->n_inst : 0; }

void cfb_inst_grid(const CfbState* s, int i, long long* k_off, int* nk, double* dk, double* k0) {
    const CfbInst& I = s->inst[(size_t)i];
    *k_off = I.k_off;
    *nk = I.nk;
    *dk = I.dk;
    *k0 = I.k0;
}

namespace sglh {
namespace {

// work items (instance, k tile, part, parts) for a tile width, instances in `order`, split as `nparts` says
std::vector<int4> cfb_items(const CfbState& S, int kt, const std::vector<int>& order, const std::vector<int>& nparts) {
    std::vector<int4> items;
    for (int i : order) {
        const int tiles = (S.inst[(size_t)i].nk + kt - 1) / kt, np = nparts.empty() ? 1 : nparts[(size_t)i];
        for (int t = 0; t < tiles; ++t)
            for (int q = 0; q < np; ++q) items.push_back(make_int4(i, t, q, np));
    }
    return items;
}

// The parts of each gauss instance's cells: a batch with few (instance, k tile) pairs (planes solved at 128 nodes each)
// would leave CTAs idle or one item running alone at the end, so its items are cut into about four per resident
// CTA, of whole segments (cfb_segment).  6 x 64 planes of 131072 cells at 128 nodes: solve 10.6 -> 6.0 ms.  part_off: where
// a split instance's segment sums start, -1 where it is not split; *elems of them in all.  Nothing is split when they would
// take more than kCfbPartBytes.
constexpr long long kCfbPartBytes = 1LL << 30;

std::vector<int> cfb_nparts(const CfbState& S, int kt, int ctas, std::vector<long long>* part_off, long long* elems) {
    long long tiles = 0;
    for (const CfbInst& I : S.inst) tiles += (I.nk + kt - 1) / kt;
    const long long want = std::min<long long>(64, (4LL * ctas + tiles - 1) / tiles);
    std::vector<int> np(S.inst.size(), 1);
    part_off->assign(S.inst.size(), -1);
    *elems = 0;
    for (size_t i = 0; i < S.inst.size(); ++i) {
        const CfbInst& I = S.inst[i];
        const long long cells = I.c1 - I.c0, seg = cfb_segment(cells);
        if (I.closure == 0) np[i] = (int)std::max<long long>(1, std::min(want, cells / seg));
        if (np[i] > 1) {
            (*part_off)[i] = *elems;
            *elems += (cells + seg - 1) / seg * I.nk;
        }
    }
    if (*elems * 16 > kCfbPartBytes) {
        np.assign(np.size(), 1);
        part_off->assign(part_off->size(), -1);
        *elems = 0;
    }
    return np;
}

// a prepared solve: work items, grid and the buffers of split instances
struct CfbRun {
    int4* items = nullptr;
    int n_items = 0, ctas = 0, kt = 0;
    int* counter = nullptr;
    double2* lnphi = nullptr; double2* parts = nullptr;
    long long* part_off = nullptr;
};

sgl_status cfb_prepare(sgl_ctx* ctx, int precision, int kt, int cps, const std::vector<int4>* given, const std::string& tag,
                       CfbRun& R) {
    CfbState& S = *ctx->cfb;
    const int P = precision == SGL_FP64 ? 0 : 1;
    const int res = cfb_resident_ctas(precision, kt);
    if (res < 1) return fail(ctx, SGL_ERR_CUDA, "batched CF kernel: no resident CTA for this tile width");
    R.kt = kt;
    R.ctas = kNumSMs * std::max(1, std::min(cps, res));
    long long part_elems = 0;
    std::vector<int4> own;
    std::vector<long long> part_off;
    if (!given) {
        const std::vector<int> np = cfb_nparts(S, kt, R.ctas, &part_off, &part_elems);
        own = cfb_items(S, kt, S.order, np);
        given = &own;
    }
    if (given->size() > (size_t)INT32_MAX) return fail(ctx, SGL_ERR_UNSUPPORTED, "batched CF kernel: too many work items");
    R.n_items = (int)given->size();
    R.items = dbuf<int4>(ctx, "cfb_items_" + tag, std::max<size_t>(1, given->size()));
    R.counter = dbuf<int>(ctx, "cfb_counter", 1);
    R.lnphi = dbuf<double2>(ctx, "cfb_lnphi", (size_t)std::max<long long>(1, S.total_k));
    if (!R.items || !R.counter || !R.lnphi) return fail(ctx, SGL_ERR_CUDA, "device allocation failed (batched CF solve)");
    CKS(upload(ctx, R.items, given->data(), given->size()));
    if (part_elems > 0) {
        R.parts = dbuf<double2>(ctx, "cfb_parts_" + tag, (size_t)part_elems);
        R.part_off = dbuf<long long>(ctx, "cfb_part_off_" + tag, part_off.size());
        if (!R.parts || !R.part_off) return fail(ctx, SGL_ERR_CUDA, "device allocation failed (batched CF solve)");
        CKS(upload(ctx, R.part_off, part_off.data(), part_off.size()));
    }
    if (!S.have[P]) {
        // template planes: the cells in this precision's form
        double* kap = nullptr; double* w = nullptr;
        float* kh = nullptr; float* kl = nullptr; float* wf = nullptr;
        if (P == 0) {
            kap = dbuf<double>(ctx, "cfb_kap", (size_t)S.n_cells);
            w = dbuf<double>(ctx, "cfb_w", (size_t)S.n_cells);
        } else {
            kh = dbuf<float>(ctx, "cfb_kh", (size_t)S.n_cells);
            kl = dbuf<float>(ctx, "cfb_kl", (size_t)S.n_cells);
            wf = dbuf<float>(ctx, "cfb_wf", (size_t)S.n_cells);
        }
        if (P == 0 ? !kap || !w : !kh || !kl || !wf) return fail(ctx, SGL_ERR_CUDA, "device allocation failed (batched CF cells)");
        launch_cfb_fill_separable(precision, S.n_cells, S.nm, S.nb, (const double*)ctx->arena.find("cfb_tF"),
                                  (const double*)ctx->arena.find("cfb_tg"), (const double*)ctx->arena.find("cfb_tu"),
                                  (const double*)ctx->arena.find("cfb_tv"), kap, w, kh, kl, wf, ctx->stream);
        CKLAUNCH();
        S.have[P] = true;
    }
    return SGL_OK;
}

void cfb_enqueue(sgl_ctx* ctx, int precision, const CfbRun& R) {
    CfbState& S = *ctx->cfb;
    launch_cfb_persistent(precision, R.kt, R.ctas, (const CfbInst*)ctx->arena.find("cfb_inst"), R.items, R.n_items,
                          R.counter, (const long long*)ctx->arena.find("cfb_pcells"),
                          (const double*)ctx->arena.find("cfb_kap"), (const double*)ctx->arena.find("cfb_w"),
                          (const float*)ctx->arena.find("cfb_kh"), (const float*)ctx->arena.find("cfb_kl"),
                          (const float*)ctx->arena.find("cfb_wf"), (const double*)ctx->arena.find("cfb_vpD"),
                          (const double*)ctx->arena.find("cfb_vpK"), (const double*)ctx->arena.find("cfb_vpw"),
                          S.nstate, R.lnphi, ctx->stream, R.parts, S.n_inst,
                          (const long long*)ctx->arena.find("cfb_koffs"), R.part_off, S.total_k);
}

sgl_status cfb_launch(sgl_ctx* ctx, int precision, int kt, int cps, const std::vector<int4>* items,
                      const std::string& tag) {
    CfbRun R;
    CKS(cfb_prepare(ctx, precision, kt, cps, items, tag, R));
    cfb_enqueue(ctx, precision, R);
    CKLAUNCH();
    return SGL_OK;
}

// The launch shape used when none was tuned: 64 k-points per item in mixed precision (two warps wait at the barriers of a
// plane's few cells; 41 gauss and vp instances: step 19.4 ms, 128 wide 19.6; planes at 128 nodes the same within 2%), 128
// in FP64, and every resident CTA.  Timing all shapes on first use, as this did, cost 0.6 s per context.
// The items of a vp instance are not split and come first; where they do not fill the chip, as many CTAs per SM as share
// them evenly (at least 3, for the gauss items beside them), because more of them meet on some SMs and set the time.  CTAs
// per SM -> step in ms, mixed: 420 vp items 2: 3.70, 3: 2.29, 4: 2.56, 8: 3.91, all (16): 3.90; 248 items 2: 1.63, 3: 1.41,
// all 1.82; 760 items 4: 3.02, 5: 3.34, all 4.25; 908 items 6: 4.82, all 5.14; 1728 items 8 and more: 4.85.
void cfb_default_shape(sgl_ctx* ctx, int precision) {
    CfbState& S = *ctx->cfb;
    const int P = precision == SGL_FP64 ? 0 : 1;
    S.kt[P] = P == 1 ? 64 : 128;
    S.cps[P] = std::max(1, cfb_resident_ctas(precision, S.kt[P]));
    if (P == 1) {
        long long vp = 0;
        for (const CfbInst& I : S.inst)
            if (I.closure == 1) vp += (I.nk + S.kt[P] - 1) / S.kt[P];
        if (vp > 0) S.cps[P] = (int)std::min<long long>(S.cps[P], std::max<long long>(3, (vp + kNumSMs - 1) / kNumSMs));
    }
    S.tuned[P] = true;
}

// The launch shape.  FP64 (the parity path, whose FP64 pipe makes every term slow here) takes a fixed
// shape: 128 k-points per item, as many CTAs per SM as fit.  The mixed path times each (tile width,
// CTAs per SM) allowed by occupancy on a sample of the batch and keeps the fastest: instances evenly
// spread in cost order (at most 256), then every s-th of their work items so that a timed launch holds
// about kTuneTerms cell-k terms, the same fraction for every tile width; a tune costs about a second.
sgl_status cfb_tune(sgl_ctx* ctx, int precision) {
    CfbState& S = *ctx->cfb;
    const int P = precision == SGL_FP64 ? 0 : 1;
    if (precision == SGL_FP64) {
        S.kt[P] = 128;
        S.cps[P] = std::max(1, cfb_resident_ctas(precision, 128));
        S.tuned[P] = true;
        ctx->cfb_shapes[2LL * S.shape_class + P] = {S.kt[P], S.cps[P]};
        return SGL_OK;
    }
    constexpr double kTuneTerms = 2e10;
    std::vector<int> sample;
    const size_t stride = std::max<size_t>(1, S.order.size() / 256);
    double scost = 0.0;
    for (size_t i = 0; i < S.order.size(); i += stride) {
        sample.push_back(S.order[i]);
        scost += S.cost[(size_t)S.order[i]];
    }
    const size_t istride = scost > kTuneTerms ? (size_t)std::ceil(scost / kTuneTerms) : 1;
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    double best = 1e300;
    for (int kt : {64, 128, 256}) {
        const int res = cfb_resident_ctas(precision, kt);
        std::vector<int4> items = cfb_items(S, kt, sample, {});
        if (istride > 1) {
            std::vector<int4> sub;
            for (size_t q = 0; q < items.size(); q += istride) sub.push_back(items[q]);
            items.swap(sub);
        }
        for (int cps : {1, 2, 4, 8, 16}) {
            if (cps > res) continue;
            CKS(cfb_launch(ctx, precision, kt, cps, &items, "tune"));       // warm
            cudaEventRecord(a, ctx->stream);
            CKS(cfb_launch(ctx, precision, kt, cps, &items, "tune"));
            cudaEventRecord(b, ctx->stream);
            CK(cudaEventSynchronize(b));
            float ms = 0.f;
            cudaEventElapsedTime(&ms, a, b);
            if (ms < best) { best = ms; S.kt[P] = kt; S.cps[P] = cps; }
        }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    S.tuned[P] = true;
    ctx->cfb_shapes[2LL * S.shape_class + P] = {S.kt[P], S.cps[P]};
    return sync_stream(ctx);
}

// Validates a batch's instance table and uploads it (instances, k offsets, plane offsets, vp chain
// tables); the cells follow from the caller
sgl_status cfb_tables(sgl_ctx* ctx, int n_inst, const int32_t* inst_plane0, const int64_t* plane_cells,
                      const int32_t* nk, const double* dk, const int32_t* closure, const double* V, int nstate,
                      const double* vp_D, const double* vp_K, const double* vp_w) {
    if (!ctx) return SGL_ERR_VALUE;
    if (n_inst < 1 || !inst_plane0 || !plane_cells || !nk || !dk || !closure || !V)
        return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: invalid sizes or NULL arrays");
    if (inst_plane0[0] != 0) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: inst_plane0[0] must be 0");
    const int n_planes = inst_plane0[n_inst];
    if (n_planes < 1 || plane_cells[0] != 0) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: invalid plane offsets");
    for (int i = 0; i < n_inst; ++i) {
        if (inst_plane0[i + 1] <= inst_plane0[i]) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: an instance has no plane");
        if (nk[i] < 2 || !(dk[i] > 0) || !std::isfinite(dk[i]) || !std::isfinite(V[i]) || (closure[i] != 0 && closure[i] != 1))
            return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: invalid k grid, V or closure of instance " + std::to_string(i));
    }
    for (int p = 0; p < n_planes; ++p)
        if (plane_cells[p + 1] < plane_cells[p]) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: plane_cells not ascending");
    const long long nc = plane_cells[n_planes];
    if (nc < 1) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: no cells");
    int n_vp = 0;
    for (int i = 0; i < n_inst; ++i) n_vp += closure[i] == 1;
    if (n_vp > 0 && (nstate < 2 || nstate > 8 || !vp_D || !vp_K || !vp_w))
        return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: vp instances need 2..8 chain states and their tables");
    CK(cudaSetDevice(ctx->device));
    CKS(sync_stream(ctx));
    if (ctx->cfb) cfb_state_free(ctx->cfb);
    ctx->cfb = new CfbState();
    CfbState& S = *ctx->cfb;
    S.n_inst = n_inst; S.n_planes = n_planes; S.nstate = n_vp > 0 ? nstate : 0; S.n_cells = nc;
    S.inst.resize((size_t)n_inst);
    S.cost.resize((size_t)n_inst);
    long long koff = 0;
    int slot = 0;
    std::vector<long long> k_offs((size_t)n_inst + 1, 0);
    for (int i = 0; i < n_inst; ++i) {
        CfbInst& I = S.inst[(size_t)i];
        I.p0 = inst_plane0[i]; I.p1 = inst_plane0[i + 1];
        I.c0 = plane_cells[I.p0]; I.c1 = plane_cells[I.p1];
        I.k_off = koff; I.nk = nk[i]; I.dk = dk[i]; I.V = V[i]; I.closure = closure[i];
        I.vp_slot = closure[i] == 1 ? slot++ : -1; I.geom = 0; I.k0 = 0.0;
        k_offs[(size_t)i] = koff;
        koff += nk[i];
        // work: cells x k, the chain about 2 S^2 cell-terms per plane
        S.cost[(size_t)i] = (double)nk[i] * ((double)(I.c1 - I.c0) + (closure[i] == 1 ? 2.0 * nstate * nstate * (I.p1 - I.p0) : 0.0));
    }
    k_offs[(size_t)n_inst] = koff;
    S.total_k = koff;
    // batches of the same shape class (largest k grid, mean cells per instance, both in powers of
    // two) reuse the launch shapes the autotuner found for the first of them
    {
        int max_nk = 0;
        for (int i = 0; i < n_inst; ++i) max_nk = std::max(max_nk, nk[i]);
        const int kb = (int)std::ceil(std::log2((double)max_nk));
        const int cb = (int)std::ceil(std::log2(std::max(1.0, (double)nc / n_inst)));
        S.shape_class = 100 * kb + cb;
        for (int q = 0; q < 2; ++q) {
            auto it = ctx->cfb_shapes.find(2LL * S.shape_class + q);
            if (it != ctx->cfb_shapes.end()) { S.kt[q] = it->second.first; S.cps[q] = it->second.second; S.tuned[q] = true; }
        }
    }
    S.order.resize((size_t)n_inst);
    std::iota(S.order.begin(), S.order.end(), 0);
    std::stable_sort(S.order.begin(), S.order.end(), [&](int x, int y) { return S.cost[(size_t)x] > S.cost[(size_t)y]; });
    DBUF(d_inst, CfbInst, "cfb_inst", n_inst);
    DBUF(d_koffs, long long, "cfb_koffs", n_inst + 1);
    DBUF(d_pc, long long, "cfb_pcells", n_planes + 1);
    DBUF(d_vpD, double, "cfb_vpD", std::max(1, n_planes * std::max(1, S.nstate)));
    DBUF(d_vpK, double, "cfb_vpK", std::max(1, n_vp * S.nstate * S.nstate));
    DBUF(d_vpw, double, "cfb_vpw", std::max(1, n_vp * S.nstate));
    CKS(upload(ctx, d_inst, S.inst.data(), S.inst.size()));
    CKS(upload(ctx, d_koffs, k_offs.data(), k_offs.size()));
    CKS(upload(ctx, d_pc, (const long long*)plane_cells, (size_t)n_planes + 1));
    if (n_vp > 0) {
        CKS(upload(ctx, d_vpD, vp_D, (size_t)n_planes * S.nstate));
        CKS(upload(ctx, d_vpK, vp_K, (size_t)n_vp * S.nstate * S.nstate));
        CKS(upload(ctx, d_vpw, vp_w, (size_t)n_vp * S.nstate));
    }
    return sync_stream(ctx);          // k_offs goes out of scope
}

}  // namespace
}  // namespace sglh

extern "C" {

sgl_status sgl_cfb_set(sgl_ctx* ctx, int n_inst, const int32_t* inst_plane0, const int64_t* plane_cells,
                       const double* kap, const double* w, const int32_t* nk, const double* dk, const int32_t* closure,
                       const double* V, int nstate, const double* vp_D, const double* vp_K, const double* vp_w) {
    if (!ctx) return SGL_ERR_VALUE;
    CKS(cfb_tables(ctx, n_inst, inst_plane0, plane_cells, nk, dk, closure, V, nstate, vp_D, vp_K, vp_w));
    CfbState& S = *ctx->cfb;
    const long long nc = S.n_cells;
    if (!kap || !w) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set: no cells");
    std::vector<float> kh((size_t)nc), kl((size_t)nc), wf((size_t)nc);
    for (long long c = 0; c < nc; ++c) {
        const ff f = ff_from_double(kap[c]);
        kh[(size_t)c] = f.hi; kl[(size_t)c] = f.lo; wf[(size_t)c] = (float)w[c];
    }
    DBUF(d_kap, double, "cfb_kap", nc);
    DBUF(d_w, double, "cfb_w", nc);
    DBUF(d_kh, float, "cfb_kh", nc);
    DBUF(d_kl, float, "cfb_kl", nc);
    DBUF(d_wf, float, "cfb_wf", nc);
    CKS(upload(ctx, d_kap, kap, (size_t)nc));
    CKS(upload(ctx, d_w, w, (size_t)nc));
    CKS(upload(ctx, d_kh, kh.data(), kh.size()));
    CKS(upload(ctx, d_kl, kl.data(), kl.size()));
    CKS(upload(ctx, d_wf, wf.data(), wf.size()));
    return sync_stream(ctx);          // the host staging vectors go out of scope
}

sgl_status sgl_cfb_set_separable(sgl_ctx* ctx, int nm, int nb, const double* F, const double* g, int n_inst,
                                 const int32_t* inst_plane0, const int32_t* nk, const double* dk, const double* k0,
                                 int geom, const double* V, const double* u, const double* v) {
    if (!ctx) return SGL_ERR_VALUE;
    if (nm < 1 || nb < 1 || !F || !g || !u || !v || n_inst < 1 || !inst_plane0)
        return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set_separable: invalid template or NULL arrays");
    if (inst_plane0[0] != 0 || inst_plane0[n_inst] < 1) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set_separable: invalid plane offsets");
    const int n_planes = inst_plane0[n_inst];
    const long long per = (long long)nm * nb;
    std::vector<int64_t> pc((size_t)n_planes + 1);
    for (int p = 0; p <= n_planes; ++p) pc[(size_t)p] = per * p;
    std::vector<int32_t> closure((size_t)n_inst, 0);
    if (geom && !k0) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set_separable: log-spaced k points need k0");
    if (k0)
        for (int i = 0; i < n_inst; ++i)
            if (!std::isfinite(k0[i]) || (!geom && !(k0[i] >= 0)) || (geom && k0[i] + (nk[i] - 1) * dk[i] > 700.0))
                return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_set_separable: invalid k0");
    CKS(cfb_tables(ctx, n_inst, inst_plane0, pc.data(), nk, dk, closure.data(), V, 0, nullptr, nullptr, nullptr));
    const long long nc = ctx->cfb->n_cells;
    if (k0) {
        CfbState& S = *ctx->cfb;
        for (int i = 0; i < n_inst; ++i) {
            S.inst[(size_t)i].k0 = k0[i];
            S.inst[(size_t)i].geom = geom ? 1 : 0;
        }
        DBUF(d_inst, CfbInst, "cfb_inst", n_inst);
        CKS(upload(ctx, d_inst, S.inst.data(), S.inst.size()));
    }
    for (long long e = 0; e < per; ++e) if (!std::isfinite(F[e])) return fail(ctx, SGL_ERR_VALUE, "non-finite template F");
    for (int b = 0; b < nb; ++b) if (!std::isfinite(g[b])) return fail(ctx, SGL_ERR_VALUE, "non-finite template g");
    for (long long e = 0; e < (long long)n_planes * nm; ++e)
        if (!std::isfinite(u[e]) || !std::isfinite(v[e])) return fail(ctx, SGL_ERR_VALUE, "non-finite plane factors");
    DBUF(d_F, double, "cfb_tF", per);
    DBUF(d_g, double, "cfb_tg", nb);
    DBUF(d_u, double, "cfb_tu", (long long)n_planes * nm);
    DBUF(d_v, double, "cfb_tv", (long long)n_planes * nm);
    CKS(upload(ctx, d_F, F, (size_t)per));
    CKS(upload(ctx, d_g, g, (size_t)nb));
    CKS(upload(ctx, d_u, u, (size_t)n_planes * nm));
    CKS(upload(ctx, d_v, v, (size_t)n_planes * nm));
    // the cells themselves follow in the first solve, in its precision's form
    CfbState& S = *ctx->cfb;
    S.nm = nm;
    S.nb = nb;
    S.have[0] = S.have[1] = false;
    return sync_stream(ctx);
}

sgl_status sgl_cfb_tune(sgl_ctx* ctx, int precision, int* kt, int* ctas_per_sm) {
    if (!ctx) return SGL_ERR_VALUE;
    if (!ctx->cfb) return fail(ctx, SGL_ERR_STATE, "sgl_cfb_tune: no batch set");
    if (precision != SGL_FP64 && precision != SGL_MIXED) return fail(ctx, SGL_ERR_VALUE, "unknown precision");
    CK(cudaSetDevice(ctx->device));
    CKS(cfb_tune(ctx, precision));
    const int P = precision == SGL_FP64 ? 0 : 1;
    if (kt) *kt = ctx->cfb->kt[P];
    if (ctas_per_sm) *ctas_per_sm = ctx->cfb->cps[P];
    return SGL_OK;
}

sgl_status sgl_cfb_lnphi(sgl_ctx* ctx, int precision, double* out) {
    if (!ctx) return SGL_ERR_VALUE;
    if (!ctx->cfb) return fail(ctx, SGL_ERR_STATE, "sgl_cfb_lnphi: no batch set");
    if (precision != SGL_FP64 && precision != SGL_MIXED) return fail(ctx, SGL_ERR_VALUE, "unknown precision");
    CK(cudaSetDevice(ctx->device));
    CfbState& S = *ctx->cfb;
    const int P = precision == SGL_FP64 ? 0 : 1;
    if (!S.tuned[P]) cfb_default_shape(ctx, precision);
    CKS(cfb_launch(ctx, precision, S.kt[P], S.cps[P], nullptr, "run"));
    if (out) CK(cudaMemcpyAsync(out, ctx->arena.find("cfb_lnphi"), (size_t)S.total_k * 16, cudaMemcpyDeviceToHost, ctx->stream));
    return sync_stream(ctx);
}

sgl_status sgl_cfb_pdf(sgl_ctx* ctx, int precision, const double* lnmu, int n_lnmu, double* P_out, int use_graph,
                       double* ms_out) {
    if (!ctx) return SGL_ERR_VALUE;
    if (!ctx->cfb) return fail(ctx, SGL_ERR_STATE, "sgl_cfb_pdf: no batch set");
    if (precision != SGL_FP64 && precision != SGL_MIXED) return fail(ctx, SGL_ERR_VALUE, "unknown precision");
    if (n_lnmu < 1 || !lnmu || !P_out) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_pdf: invalid ln mu grid or output");
    for (int m = 0; m < n_lnmu; ++m) if (!std::isfinite(lnmu[m])) return fail(ctx, SGL_ERR_VALUE, "non-finite ln mu");
    CK(cudaSetDevice(ctx->device));
    CfbState& S = *ctx->cfb;
    for (const CfbInst& I : S.inst)
        if (I.k0 != 0.0 || I.geom) return fail(ctx, SGL_ERR_VALUE, "sgl_cfb_pdf: the inversion needs k grids n dk");
    const int P = precision == SGL_FP64 ? 0 : 1;
    if (!S.tuned[P]) cfb_default_shape(ctx, precision);
    // every buffer of the step exists before a capture (no allocation inside it)
    CfbRun R;
    CKS(cfb_prepare(ctx, precision, S.kt[P], S.cps[P], nullptr, std::string("run") + (P ? "m" : "d"), R));
    // (named per precision: a buffer that the other precision's call grows would move under this one's graph)
    const std::string suffix = P ? "m" : "d";
    void* phi = ctx->arena.get("cfb_phi_" + suffix, (size_t)std::max<long long>(1, S.total_k) * 2 * (P ? 4 : 8));
    DBUF(d_lnmu, double, "cfb_lnmu_" + suffix, n_lnmu);
    DBUF(d_P, double, "cfb_P_" + suffix, (long long)S.n_inst * n_lnmu);
    if (!phi) return fail(ctx, SGL_ERR_CUDA, "device allocation failed (cfb phi)");
    const cudaStream_t st = ctx->stream;
    auto enqueue = [&]() {
        cfb_enqueue(ctx, precision, R);
        launch_cfb_pdf(precision, (const CfbInst*)ctx->arena.find("cfb_inst"), S.n_inst, R.lnphi, S.total_k,
                       (const long long*)ctx->arena.find("cfb_koffs"), phi, d_lnmu, n_lnmu, d_P, st);
    };
    CKS(upload(ctx, d_lnmu, lnmu, (size_t)n_lnmu));
    const bool reuse = use_graph && S.graph[P] && S.graph_nm[P] == n_lnmu && S.graph_kt[P] == S.kt[P] &&
                       S.graph_cps[P] == S.cps[P];
    if (use_graph && !reuse) {
        // capture the whole step once: counter reset, persistent solve, Phi, inversion
        CKS(sync_stream(ctx));
        if (S.graph[P]) { cudaGraphExecDestroy(S.graph[P]); S.graph[P] = nullptr; }
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        enqueue();
        const cudaError_t ce = cudaStreamEndCapture(st, &g);
        if (ce != cudaSuccess) return fail(ctx, SGL_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(ce));
        const cudaError_t ie = cudaGraphInstantiate(&S.graph[P], g, 0);
        cudaGraphDestroy(g);
        if (ie != cudaSuccess) { S.graph[P] = nullptr; return fail(ctx, SGL_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ie)); }
        S.graph_nm[P] = n_lnmu; S.graph_kt[P] = S.kt[P]; S.graph_cps[P] = S.cps[P];
    }
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    cudaEventRecord(a, st);
    if (use_graph) CK(cudaGraphLaunch(S.graph[P], st));
    else enqueue();
    cudaEventRecord(b, st);
    CKLAUNCH();
    CK(cudaMemcpyAsync(P_out, d_P, (size_t)S.n_inst * n_lnmu * sizeof(double), cudaMemcpyDeviceToHost, st));
    CKS(sync_stream(ctx));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (ms_out) *ms_out = ms;
    for (long long e = 0; e < (long long)S.n_inst * n_lnmu; ++e)
        if (!std::isfinite(P_out[e])) return fail(ctx, SGL_ERR_NONFINITE, "batched PDF returned non-finite values");
    return SGL_OK;
}

}  // extern "C"
