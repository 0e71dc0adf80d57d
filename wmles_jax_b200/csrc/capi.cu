// C ABI of libwmles_cuda.so (include/wmles_cuda.h): case set-up and step orchestration.
//
// A wm_case owns one case's device data (metrics, ghost programs, wall geometry, work
// states, inflow/sponge buffers).  Launches run on a View: the concatenated device tables
// (blocks, per-case constants, wall faces, stage tiles, ghost-program segments) and the
// reduction scratch of a set of cases.  Every wm_case carries a View of itself for the
// single-case entry points; a wm_batch is a View over several resident cases, so one
// launch per kernel and stage advances all of them.  The stage work list is cut for the
// whole view (tile shapes and chunks along i by how many cases share the GPU).  Per-case
// reductions are exact in any order (CFL minimum; constant-mass-flux sum in bins), so a case's
// result depends neither on the tiles nor on what else is in the batch.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "wm_internal.cuh"
#include "stage.cuh"
#include "aux.cuh"
#include "stats.cuh"
#include "derived.cuh"
#include "geom.cuh"

using namespace wm;

namespace {

thread_local std::string g_err;

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define CK(call)                                                                             \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return fail(WM_E_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_),   \
                        __FILE__, __LINE__);                                                 \
    } while (0)

struct GhostProg {
    int count = 0;
    int *dst = nullptr, *src = nullptr, *ops = nullptr, *op_code = nullptr;
    double* op_nrm = nullptr;
};

// launch accounting / event timing (wm_profile_*)
struct Prof {
    long long nlaunch[WM_NKINDS] = {0, 0, 0, 0, 0};
    bool on = false;
    struct Rec { int kind; cudaEvent_t a, b; };
    std::vector<Rec> recs;
    std::vector<cudaEvent_t> pool;

    cudaEvent_t event() {
        if (!pool.empty()) {
            cudaEvent_t e = pool.back();
            pool.pop_back();
            return e;
        }
        cudaEvent_t e = nullptr;
        cudaEventCreate(&e);
        return e;
    }
    void reset(bool enable) {
        for (auto& r : recs) { pool.push_back(r.a); pool.push_back(r.b); }
        recs.clear();
        for (int k = 0; k < WM_NKINDS; ++k) nlaunch[k] = 0;
        on = enable;
    }
    ~Prof() {
        for (auto& r : recs) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
        for (cudaEvent_t e : pool) cudaEventDestroy(e);
    }
};

// brackets one launch of `kind`: counts it and, when profiling, records an event pair
struct LaunchScope {
    Prof* p;
    int slot = -1;
    cudaStream_t s;
    LaunchScope(Prof* p_, int kind, cudaStream_t s_, int n = 1) : p(p_), s(s_) {
        p->nlaunch[kind] += n;
        if (p->on && n > 0) {
            Prof::Rec r{kind, p->event(), p->event()};
            cudaEventRecord(r.a, s);
            p->recs.push_back(r);
            slot = (int)p->recs.size() - 1;
        }
    }
    ~LaunchScope() {
        if (slot >= 0) cudaEventRecord(p->recs[slot].b, s);
    }
};

struct Owner {
    std::vector<void*> allocs;
    ~Owner() {
        for (void* p : allocs) cudaFree(p);
    }
    template <typename T>
    int alloc(T** p, size_t count) {
        void* v = nullptr;
        if (count == 0) count = 1;
        cudaError_t e = cudaMalloc(&v, sizeof(T) * count);
        if (e != cudaSuccess) return fail(WM_E_CUDA, "cudaMalloc(%zu bytes): %s", sizeof(T) * count, cudaGetErrorString(e));
        allocs.push_back(v);
        *p = static_cast<T*>(v);
        return WM_OK;
    }
    template <typename T>
    int upload(T** p, const T* host, size_t count) {
        int r = alloc(p, count);
        if (r) return r;
        if (count && host) CK(cudaMemcpy(*p, host, sizeof(T) * count, cudaMemcpyHostToDevice));
        return WM_OK;
    }
};

struct View;

}  // namespace

namespace wm {
int set_error(int code, const char* msg) {
    g_err = msg;
    return code;
}
}  // namespace wm

struct wm_case {
    int device = 0;
    Owner mem;
    // host copies of the case-local descriptors (block / wall indices local to the case)
    std::vector<BlockDev> hb;
    CaseDev hc{};
    std::vector<WallDev> hw;
    int chunk_req = 0;                   // planes per stage-kernel CTA requested (0: automatic)
    StageOpts opts{};
    std::vector<double*> work[2];
    GhostProg prog_rhs, prog_all;
    double* stash = nullptr;
    double* d_bc = nullptr;
    bool has_inflow = false;
    int inflow_block = -1;
    double *d_modes = nullptr, *d_table = nullptr, *inflow_buf = nullptr, *inflow_raw = nullptr;
    double* inflow_prof = nullptr;       // 6 x inflow_n time-independent profile factors
    double* inflow_cz = nullptr;         // extruded inflow plane: cos / sin (kz z) tables (else null)
    BlockDev* d_inflow_block = nullptr;  // the inflow block's descriptor, for the set-up kernels
    wm_inflow inflow{};
    long long inflow_n = 0;
    std::vector<double*> spmean;         // per block, null without sponge
    std::vector<int> sp_rows;            // (block, interior row) pairs of the rows that reach into the sponge
    double* ps_part = nullptr;           // plane-statistics scratch (PS_NQ x max Nj x PS_CHUNKS)
    unsigned* ps_counter = nullptr;
    View* self = nullptr;                // the case as a view of one case
    unsigned* d_status = nullptr;        // status word (WM_ST_* bits)
    Prof prof;
    ~wm_case();
};

namespace {

struct View {
    Owner mem;
    std::vector<wm_case*> members;
    int nblocks = 0, ncases = 0;
    std::vector<BlockDev> hb;
    std::vector<CaseDev> hc;
    std::vector<WallDev> hw;
    // stage work lists, of the general blocks and of those extruded along k (each one launch): the
    // blocks' (j,k) columns, cut along i
    struct Work {
        std::vector<int> blocks;         // view blocks
        std::vector<Tile> tiles;
        std::vector<int> cta_first;      // balanced split: CTA c runs tiles [cta_first[c], cta_first[c+1])
                                         // (empty: one tile per CTA)
        Tile* d_tiles = nullptr;
        int* d_cta_first = nullptr;
        int ctas() const { return cta_first.empty() ? (int)tiles.size() : (int)cta_first.size() - 1; }
    } work[2];
    std::vector<int> case_block_start;
    std::vector<GhostSeg> seg_rhs, seg_all;
    int total_rhs = 0, total_all = 0;
    BlockDev* d_blocks = nullptr;
    CaseDev* d_cases = nullptr;
    WallDev* d_walls = nullptr;
    GhostSeg *d_seg_rhs = nullptr, *d_seg_all = nullptr;
    double *cmf_sum = nullptr, *cmf_delta = nullptr;   // constant mass flux: per case three sums, the shift
    unsigned long long* dt_key = nullptr;   // CFL pass: per-case minimum keys
    unsigned* counters = nullptr;        // [0]: CFL reduction, [1]: constant-mass-flux reduction
    std::vector<int> cta_start[2];       // CFL pass of the general and of the extruded blocks: first chunk of
                                         // each view block (+ total)
    std::vector<int> gcta_start;         // same for the blocks' ghost cells (output ghost fill)
    int max_wall_faces = 0;
    std::vector<int> sp_rows;            // (view block, row) pairs of the sponge rows of every case
    int* d_sp_rows = nullptr;
    bool any_sponge = false, any_cmf = false;
    StageOpts opts{};
};

int upload_prog(wm_case* c, GhostProg* g, const wm_ghost_program& p) {
    g->count = p.count;
    int r;
    if ((r = c->mem.upload(&g->dst, p.dst, 2 * (size_t)p.count))) return r;
    if ((r = c->mem.upload(&g->src, p.src, 2 * (size_t)p.count))) return r;
    if ((r = c->mem.upload(&g->ops, p.ops, 2 * (size_t)p.count))) return r;
    if ((r = c->mem.upload(&g->op_code, p.op_code, (size_t)p.nops))) return r;
    if ((r = c->mem.upload(&g->op_nrm, p.op_nrm, 3 * (size_t)p.nops))) return r;
    return WM_OK;
}

// every index of a ghost-cell program inside its arrays: the gather kernel trusts them
int validate_program(const wm_case_desc* d, const wm_ghost_program& p, const char* name) {
    if (p.count < 0 || p.nops < 0) return fail(WM_E_INVALID, "%s: negative count", name);
    if (p.count > 0 && (!p.dst || !p.src || !p.ops)) return fail(WM_E_INVALID, "%s: null arrays", name);
    if (p.nops > 0 && (!p.op_code || !p.op_nrm)) return fail(WM_E_INVALID, "%s: null op arrays", name);
    auto cells = [&](int b) {
        const wm_block& B = d->blocks[b];
        return (long long)(B.n[0] + 2 * B.ng) * (B.n[1] + 2 * B.ng) * (B.n[2] + 2 * B.ng);
    };
    long long inflow_n = 0;
    if (d->inflow) {
        const wm_block& B = d->blocks[d->inflow->block];
        inflow_n = (long long)B.ng * (B.n[1] + 2 * B.ng) * (B.n[2] + 2 * B.ng);
    }
    for (int e = 0; e < p.count; ++e) {
        const int db = p.dst[2 * e], dc = p.dst[2 * e + 1];
        if (db < 0 || db >= d->nblocks || dc < 0 || dc >= cells(db))
            return fail(WM_E_INVALID, "%s entry %d: destination out of range", name, e);
        const int kind = p.src[2 * e] >> 24, sb = p.src[2 * e] & 0xffffff, sc = p.src[2 * e + 1];
        const bool ok = kind == WM_SRC_CELL ? (sb < d->nblocks && sc >= 0 && sc < cells(sb))
                        : kind == WM_SRC_INFLOW ? (d->inflow && sc >= 0 && sc < inflow_n)
                        : kind == WM_SRC_CONST ? (sb < d->nbc) : false;
        if (!ok) return fail(WM_E_INVALID, "%s entry %d: source out of range", name, e);
        const int o0 = p.ops[2 * e], no = p.ops[2 * e + 1];
        if (o0 < 0 || no < 0 || (long long)o0 + no > p.nops)
            return fail(WM_E_INVALID, "%s entry %d: map chain out of range", name, e);
    }
    for (int o = 0; o < p.nops; ++o) {
        const int code = p.op_code[o] & 0xff, bc = (p.op_code[o] >> 8) & 0xff;
        if (code < WM_OP_SLIP || code > WM_OP_FARFIELD || ((code != WM_OP_SLIP) && bc >= d->nbc))
            return fail(WM_E_INVALID, "%s map %d: bad code or BC id", name, o);
    }
    return WM_OK;
}

int validate(const wm_case_desc* d) {
    if (!d) return fail(WM_E_INVALID, "null descriptor");
    if (d->nblocks < 1 || d->nblocks > WM_MAX_BLOCKS)
        return fail(WM_E_INVALID, "nblocks=%d outside [1, %d]", d->nblocks, WM_MAX_BLOCKS);
    if (d->scheme < 0 || d->scheme > WM_SCHEME_HYBRID) return fail(WM_E_INVALID, "unknown scheme %d", d->scheme);
    if (d->kep_order != 2 && d->kep_order != 4) return fail(WM_E_INVALID, "kep_order must be 2 or 4");
    if (d->sgs < 0 || d->sgs > WM_SGS_VREMAN) return fail(WM_E_INVALID, "unknown sgs %d", d->sgs);
    if (d->precision != WM_PREC_FP64 && d->precision != WM_PREC_MIXED)
        return fail(WM_E_INVALID, "unknown precision %d", d->precision);
    if (d->tile < -1 || d->tile > 3) return fail(WM_E_INVALID, "unknown tile shape %d", d->tile);
    if (d->tile == 3 && d->precision == WM_PREC_FP64)
        return fail(WM_E_UNSUPPORTED, "tile 3 (16x32) is built for the mixed form only");
    for (int b = 0; b < d->nblocks; ++b) {
        const wm_block& B = d->blocks[b];
        if (B.ng != 3) return fail(WM_E_UNSUPPORTED, "block %d: ng=%d (this library supports ng=3)", b, B.ng);
        for (int a = 0; a < 3; ++a)
            if (B.n[a] < B.ng) return fail(WM_E_INVALID, "block %d: n[%d]=%d < ng", b, a, B.n[a]);
        if (!B.metrics) return fail(WM_E_INVALID, "block %d: null metrics", b);
    }
    for (int w = 0; w < d->nwalls; ++w) {
        const wm_wall& W = d->walls[w];
        if (W.block < 0 || W.block >= d->nblocks || W.axis < 0 || W.axis > 2 || W.side < 0 || W.side > 1)
            return fail(WM_E_INVALID, "wall %d: bad block/axis/side", w);
        const int n = d->blocks[W.block].n[W.axis];
        if (W.n_match < 1 || W.n_match > n) return fail(WM_E_INVALID, "wall %d: n_match=%d", w, W.n_match);
    }
    if (d->cmf_dir >= 0 && !(d->cmf_volume > 0)) return fail(WM_E_INVALID, "cmf_volume must be positive");
    if (d->cmf_dir > 2) return fail(WM_E_INVALID, "cmf_dir=%d", d->cmf_dir);
    if (!(d->cfl > 0)) return fail(WM_E_INVALID, "cfl must be positive");
    for (int w = 0; w < d->nwalls; ++w) {
        const wm_wall& W = d->walls[w];
        if (!W.geom) return fail(WM_E_INVALID, "wall %d: null geometry", w);
        if (W.n_iter < 0 || W.n_iter > 1000) return fail(WM_E_INVALID, "wall %d: n_iter=%d", w, W.n_iter);
    }
    if (d->nbc < 0 || (d->nbc > 0 && !d->bc_table)) return fail(WM_E_INVALID, "bad BC table");
    if (d->inflow) {
        const wm_inflow& I = *d->inflow;
        if (I.block < 0 || I.block >= d->nblocks) return fail(WM_E_INVALID, "inflow block %d", I.block);
        if (I.n_modes < 1 || I.n_tab < 2 || !I.modes || !I.table) return fail(WM_E_INVALID, "bad inflow tables");
        if (!(I.L > 0)) return fail(WM_E_INVALID, "inflow length scale must be positive");
        const int Nk = d->blocks[I.block].n[2] + 2 * d->blocks[I.block].ng;
        if (Nk > IN_ROW_MAX_NK)
            return fail(WM_E_UNSUPPORTED, "inflow block: %d cells along k with ghosts, above %d", Nk, IN_ROW_MAX_NK);
    }
    if (d->sponge.enabled && !(d->sponge.x_end_l > d->sponge.x_start_l && d->sponge.L > 0))
        return fail(WM_E_INVALID, "bad sponge extent");
    int r;
    if ((r = validate_program(d, d->ghost_rhs, "ghost_rhs"))) return r;
    if ((r = validate_program(d, d->ghost_all, "ghost_all"))) return r;
    return WM_OK;
}

// (j,k) tile columns of a block
long long columns(const BlockDev& B) {
    return (long long)((B.n[1] + B.tj - 1) / B.tj) * ((B.n[2] + B.tk - 1) / B.tk);
}

// the tile of a block's column at (j0, k0) over planes [i0, i1)
Tile make_tile(const BlockDev& B, int b, int j0, int k0, int i0, int i1) {
    return Tile{b, j0, k0, i0, i1, std::min(B.tj, B.ng + B.n[1] - j0), std::min(B.tk, B.ng + B.n[2] - k0)};
}

// planes per stage-kernel CTA: wave quantisation against the chunk prologue cost
int choose_chunk(const std::vector<BlockDev>& hb, const std::vector<int>& blocks, const StageOpts& opts, int requested) {
    if (requested > 0) return requested;
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int occ = stage_ctas_per_sm(opts);
    if (occ < 1) occ = 1;
    const long long slots = (long long)sms * occ;
    int nimax = 0;
    for (int b : blocks) nimax = std::max(nimax, hb[b].n[0]);
    double best = 1e300;
    int best_ic = nimax;
    for (int ic = 1; ic <= nimax; ++ic) {
        long long ctas = 0;
        for (int b : blocks) ctas += columns(hb[b]) * ((hb[b].n[0] + ic - 1) / ic);
        const long long waves = (ctas + slots - 1) / slots;
        const double cost = double(waves) * (std::min(ic, nimax) + SEG_PLANES);
        if (cost < best - 1e-9) { best = cost; best_ic = ic; }
    }
    return best_ic;
}

// resident stage-kernel CTAs of the whole GPU
int stage_slots(const StageOpts& opts) {
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int occ = stage_ctas_per_sm(opts);
    return sms * (occ < 1 ? 1 : occ);
}

// wave split, for work lists with fewer (j,k) columns than resident CTAs and one plane count n0:
// every column is cut at the same planes into q = slots / C equal chunks over [0, n0 - x)
// (q full waves, all columns in lockstep, so halo reads of neighbouring columns hit L2), and
// the last x planes of every column go to the r = slots - q C CTAs left over, each taking
// the tail of columns m, m + r, m + 2 r, ... in turn (again in lockstep).  x balances the
// chunk length against the tail CTAs' segments (split_planes); 0: no such split is the cheapest
void build_waves(const std::vector<BlockDev>& hb, View::Work* v, int slots) {
    struct Col { int b, j0, k0; };
    std::vector<Col> cols;
    const int n0 = hb[v->blocks[0]].n[0];
    for (int b : v->blocks) {
        const BlockDev& B = hb[b];
        if (B.n[0] != n0) return;
        for (int j0 = B.ng; j0 < B.ng + B.n[1]; j0 += B.tj)
            for (int k0 = B.ng; k0 < B.ng + B.n[2]; k0 += B.tk) cols.push_back(Col{b, j0, k0});
    }
    const int C = (int)cols.size();
    int x = 0;
    split_planes(C, n0, slots, nullptr, &x);
    if (x == 0) return;
    const int q = slots / C, r = slots - q * C, L = (n0 - x + q - 1) / q;
    v->tiles.clear();
    v->cta_first.assign(1, 0);
    for (int w = 0; w < q; ++w)
        for (const Col& c : cols) {
            const int ng = hb[c.b].ng;
            const int lo = w * L, hi = std::min((w + 1) * L, n0 - x);
            if (hi > lo) v->tiles.push_back(make_tile(hb[c.b], c.b, c.j0, c.k0, ng + lo, ng + hi));
            v->cta_first.push_back((int)v->tiles.size());
        }
    for (int t = 0; t < r; ++t) {
        for (int c = t; c < C; c += r) {
            const int ng = hb[cols[c].b].ng;
            v->tiles.push_back(make_tile(hb[cols[c].b], cols[c].b, cols[c].j0, cols[c].k0, ng + n0 - x, ng + n0));
        }
        v->cta_first.push_back((int)v->tiles.size());
    }
}

// Rounding constants of a case's sum of rho u V (constant mass flux), one per bin: 3 x 2^51 u, so that
// x + c - c is x to a multiple of u.  The bins take a value apart, each what the one above left over:
// |x| < 2^e and fewer than 2^n cells make every sum of the first bin's parts a multiple of u = 2^(e+n-52)
// below 2^53 u, which FP64 adds without rounding, so in any order to the same bits; the parts left over are below u / 2,
// and the next bin has u 2^(n-53).  What the third leaves is under 2^(e + 3 n - 158) a cell, for 2^22 cells and a
// total of 2^-30 x 2^e a cell some 2^-62 of the total.  2^e is 2^30 times the mean cell's volume times the
// target or, where that is larger (a target of zero), the speed of sound; values beyond it are still added,
// but rounded, as any sum is.
void cmf_bins(CaseDev& C, double cells) {
    int n, e;
    std::frexp(std::max(cells, 8.0), &n);
    const double c = std::isfinite(C.c_ref) ? C.c_ref : 0.0;
    std::frexp(std::max(std::fabs(C.cmf_target), c) * (C.cmf_volume / cells), &e);
    for (int m = 0, u = e + 30 + n - 52; m < 3; ++m, u += n - 53) C.cmf_bin[m] = std::ldexp(3.0, u + 51);
}

// Tile shapes of a view: the blocks of like extents on their share of the GPU, among those of a launch.  A case's results do
// not depend on them, so that it has one shape alone and another among many: 64 channels of 16^3
// in a batch, float form, took 736 us a step with the shapes of the cases alone and 210 with the batch's.
void view_tiles(std::vector<BlockDev>& hb, const std::vector<int>& blocks, const StageOpts& opts, int slots) {
    double cells = 0.0;
    auto size = [](const BlockDev& B) { return (double)B.n[0] * B.n[1] * B.n[2]; };
    for (int b : blocks) cells += size(hb[b]);
    for (int b : blocks) hb[b].tj = 0;
    for (int b : blocks) {
        if (hb[b].tj) continue;
        auto same = [&](int o) { return std::equal(hb[b].n, hb[b].n + 3, hb[o].n); };
        const int count = (int)std::count_if(blocks.begin(), blocks.end(), same);
        int tj, tk;
        tile_shape(opts, hb[b].n, count, (int)(slots * (count * size(hb[b]) / cells) + 0.5), &tj, &tk);
        for (int o : blocks)
            if (same(o)) { hb[o].tj = tj; hb[o].tk = tk; }
    }
}

// chunked split: every column cut into chunks of ic planes, one chunk per CTA
void build_tiles(const std::vector<BlockDev>& hb, View::Work* v, int ic) {
    v->tiles.clear();
    v->cta_first.clear();
    for (int b : v->blocks) {
        const BlockDev& B = hb[b];
        const int ng = B.ng;
        for (int i0 = ng; i0 < ng + B.n[0]; i0 += ic)
            for (int j0 = ng; j0 < ng + B.n[1]; j0 += B.tj)
                for (int k0 = ng; k0 < ng + B.n[2]; k0 += B.tk)
                    v->tiles.push_back(make_tile(B, b, j0, k0, i0, std::min(i0 + ic, ng + B.n[0])));
    }
}

bool same_opts(const StageOpts& a, const StageOpts& b) {
    return a.precision == b.precision && a.scheme == b.scheme && a.kep_order == b.kep_order &&
           a.limiter == b.limiter && a.sgs == b.sgs && a.tile == b.tile;
}

// Row and k tables of a block extruded along k (left null otherwise): its stage kernel takes the
// metrics of a row from shared memory instead of loading 21 per face and 20 per gradient
// record, and leaves out the products with their zero components (stage.cu).  The factor per k of
// the i- and j-face areas is taken from the first interior row's i face (their larger component).
// The tables reproduce the metrics to a few units in the last place (tolerance 16).
int extruded_tables(wm_case* c, BlockDev& B, int precision) {
    B.rows = B.ktab = nullptr;
    B.rows32 = B.ktab32 = nullptr;
    const int Nk = B.N[2], k0 = B.ng;
    const size_t n = (size_t)B.ncell, row = ((size_t)B.ng * B.N[1] + B.ng) * Nk;
    std::vector<double> sx(Nk), sy(Nk), id(Nk), kt(2 * (size_t)Nk);
    CK(cudaMemcpy(sx.data(), B.met + WM_MET_SIX * n + row, sizeof(double) * Nk, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(sy.data(), B.met + WM_MET_SIY * n + row, sizeof(double) * Nk, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(id.data(), B.met + WM_MET_IDK * n + row, sizeof(double) * Nk, cudaMemcpyDeviceToHost));
    const std::vector<double>& s = std::fabs(sx[k0]) >= std::fabs(sy[k0]) ? sx : sy;
    for (int k = 0; k < Nk; ++k) {
        kt[2 * k] = s[k] / s[k0];
        kt[2 * k + 1] = id[k];
        if (!(kt[2 * k] > 0.0)) return WM_OK;
    }
    // two allocations (each costs the driver a call that may take long), kept also when the check fails: a
    // cudaFree here would wait for the device.  The first: the table, the check's flag, the rounded table
    const size_t nk = kt.size(), nr = (size_t)B.N[0] * B.N[1] * RT_N;
    const bool mixed = precision == WM_PREC_MIXED;
    int ok = 1;
    kt.resize(nk + 1 + (mixed ? (nk + 1) / 2 : 0));
    std::memcpy(&kt[nk], &ok, sizeof(ok));
    double *d_kt = nullptr, *rows = nullptr;
    int r;
    if ((r = c->mem.upload(&d_kt, kt.data(), kt.size()))) return r;
    int* flag = reinterpret_cast<int*>(d_kt + nk);
    CK(launch_ext_check(B.met, B.N, B.ng, k0, d_kt, 16 * 2.220446049250313e-16, flag, 0));
    CK(cudaMemcpy(&ok, flag, sizeof(int), cudaMemcpyDeviceToHost));
    if (!ok) return WM_OK;
    if ((r = c->mem.alloc(&rows, nr + (mixed ? nr / 2 : 0)))) return r;
    CK(launch_ext_rows(B.met, B.N, k0, rows, 0));
    B.rows = rows;
    B.ktab = d_kt;
    if (mixed) {
        float *rows32 = reinterpret_cast<float*>(rows + nr), *kt32 = reinterpret_cast<float*>(d_kt + nk + 1);
        CK(launch_to_f32(rows, rows32, (long long)nr, 0));
        CK(launch_to_f32(d_kt, kt32, (long long)nk, 0));
        B.rows32 = rows32;
        B.ktab32 = kt32;
    }
    return WM_OK;
}

GhostSeg segment(const wm_case* c, const GhostProg& p, int start, int block0) {
    GhostSeg g{};
    g.dst = p.dst; g.src = p.src; g.ops = p.ops; g.op_code = p.op_code; g.op_nrm = p.op_nrm;
    g.bc = c->d_bc;
    g.inflow = c->inflow_buf;
    g.inflow_n = c->inflow_n;
    g.start = start; g.count = p.count; g.block0 = block0;
    g.gamma = c->hc.gamma; g.gm1 = c->hc.gm1; g.Rg = c->hc.Rg;
    return g;
}

// concatenated device tables and reduction scratch of `cases`
int build_view(View* v, wm_case* const* cases, int n) {
    if (n < 1 || n > MAX_CASES) return fail(WM_E_INVALID, "a view holds 1..%d cases, got %d", MAX_CASES, n);
    for (int ci = 0; ci < n; ++ci) {
        wm_case* c = cases[ci];
        if (!c) return fail(WM_E_INVALID, "null case %d", ci);
        if (ci > 0 && !same_opts(c->opts, cases[0]->opts))
            return fail(WM_E_UNSUPPORTED, "cases of one batch must share precision, scheme, SGS model and tile shape");
        const int bo = (int)v->hb.size(), wo = (int)v->hw.size();
        if (bo + (int)c->hb.size() > WM_MAX_BLOCKS)
            return fail(WM_E_UNSUPPORTED, "a batch holds at most %d blocks", WM_MAX_BLOCKS);
        v->members.push_back(c);
        v->case_block_start.push_back(bo);
        for (BlockDev B : c->hb) {
            B.case_id = ci;
            for (int f = 0; f < 6; ++f)
                if (B.wall[f] >= 0) B.wall[f] += wo;
            v->hb.push_back(B);
        }
        for (WallDev W : c->hw) {
            W.block += bo;
            v->max_wall_faces = std::max(v->max_wall_faces, W.nt1 * W.nt2);
            v->hw.push_back(W);
        }
        v->hc.push_back(c->hc);
        v->seg_rhs.push_back(segment(c, c->prog_rhs, v->total_rhs, bo));
        v->total_rhs += c->prog_rhs.count;
        v->seg_all.push_back(segment(c, c->prog_all, v->total_all, bo));
        v->total_all += c->prog_all.count;
        for (size_t p = 0; p < c->sp_rows.size(); p += 2) {
            v->sp_rows.push_back(bo + c->sp_rows[p]);
            v->sp_rows.push_back(c->sp_rows[p + 1]);
        }
        v->any_sponge = v->any_sponge || c->hc.sponge;
        v->any_cmf = v->any_cmf || c->hc.cmf_dir >= 0;
    }
    v->case_block_start.push_back((int)v->hb.size());
    v->nblocks = (int)v->hb.size();
    v->ncases = n;
    v->opts = cases[0]->opts;
    // the chunk length is chosen for the whole set (results do not depend on it)
    int req = cases[0]->chunk_req;
    for (int ci = 1; ci < n; ++ci)
        if (cases[ci]->chunk_req != req) req = 0;
    for (int b = 0; b < v->nblocks; ++b) v->work[v->hb[b].rows ? 1 : 0].blocks.push_back(b);
    for (View::Work& w : v->work) {
        if (w.blocks.empty()) continue;
        view_tiles(v->hb, w.blocks, v->opts, stage_slots(v->opts));
        const int ic = choose_chunk(v->hb, w.blocks, v->opts, req);
        build_tiles(v->hb, &w, ic);
        if (req != 0) continue;
        build_waves(v->hb, &w, stage_slots(v->opts));
    }
    for (std::vector<int>& start : v->cta_start) start.assign(1, 0);   // one interior cell per thread of the CFL pass
    v->gcta_start.assign(1, 0);                 // one ghost cell per thread
    for (const BlockDev& B : v->hb) {
        const int chunks = (int)(((long long)B.n[0] * B.n[1] * B.n[2] + DT_NT - 1) / DT_NT);
        for (int x = 0; x < 2; ++x)
            v->cta_start[x].push_back(v->cta_start[x].back() + (x == (B.rows ? 1 : 0) ? chunks : 0));
        v->gcta_start.push_back(v->gcta_start.back() + (int)((ghost_cells(B) + DT_NT - 1) / DT_NT));
    }
    int r;
    Owner& m = v->mem;
    if ((r = m.upload(&v->d_blocks, v->hb.data(), v->hb.size()))) return r;
    if ((r = m.upload(&v->d_cases, v->hc.data(), v->hc.size()))) return r;
    if ((r = m.upload(&v->d_walls, v->hw.data(), v->hw.size()))) return r;
    for (View::Work& w : v->work) {
        if ((r = m.upload(&w.d_tiles, w.tiles.data(), w.tiles.size()))) return r;
        if (!w.cta_first.empty())
            if ((r = m.upload(&w.d_cta_first, w.cta_first.data(), w.cta_first.size()))) return r;
    }
    if ((r = m.upload(&v->d_seg_rhs, v->seg_rhs.data(), v->seg_rhs.size()))) return r;
    if ((r = m.upload(&v->d_seg_all, v->seg_all.data(), v->seg_all.size()))) return r;
    if (!v->sp_rows.empty())
        if ((r = m.upload(&v->d_sp_rows, v->sp_rows.data(), v->sp_rows.size()))) return r;
    if ((r = m.alloc(&v->cmf_sum, 4 * (size_t)n))) return r;
    v->cmf_delta = v->cmf_sum + 3 * (size_t)n;
    CK(cudaMemset(v->cmf_sum, 0, sizeof(double) * 4 * n));
    {
        const std::vector<unsigned long long> empty((size_t)n, DT_KEY_EMPTY);
        if ((r = m.upload(&v->dt_key, empty.data(), empty.size()))) return r;
    }
    if ((r = m.alloc(&v->counters, 2))) return r;
    CK(cudaMemset(v->counters, 0, 2 * sizeof(unsigned)));
    return WM_OK;
}

int fill_inflow(View* v, Prof* pf, const double* times, double time_dt, const double* const* dt, cudaStream_t s) {
    for (int ci = 0; ci < v->ncases; ++ci) {
        wm_case* c = v->members[ci];
        if (!c->has_inflow) continue;
        const int vb = v->case_block_start[ci] + c->inflow_block;
        const BlockDev& B = v->hb[vb];
        InflowArgs I{};
        I.block = v->d_blocks + vb;
        I.modes = c->d_modes; I.table = c->d_table;
        I.n_modes = c->inflow.n_modes; I.n_tab = c->inflow.n_tab;
        I.U_inf = c->inflow.U_inf; I.L = c->inflow.L; I.rho_inf = c->inflow.rho_inf; I.p_inf = c->inflow.p_inf;
        I.gm1 = c->hc.gm1;
        I.time0 = times[ci]; I.time_dt = time_dt; I.dt = dt ? dt[ci] : nullptr;
        I.raw = c->inflow_raw;
        I.out = c->inflow_buf;
        I.prof = c->inflow_prof;
        I.cz = c->inflow_cz;
        LaunchScope ls(pf, WM_KIND_SOURCE, s, IN_LAUNCHES);
        CK(launch_inflow(I, B.N[1], B.N[2], B.ng, s));
    }
    return WM_OK;
}

// one RHS evaluation fused with RK stage `stage` (0 = plain RHS) for every case of the view;
// state pointers per view block, time steps and times per case
int run_stage(View* v, Prof* pf, int stage, double* const* q_in, const double* const* q0, double* const* q_out,
              const double* const* dt, const double* times, double time_dt, cudaStream_t s) {
    int r;
    if ((r = fill_inflow(v, pf, times, time_dt, dt, s))) return r;
    // ghost cells the RHS reads, wall-model flux overrides and sponge means: one launch
    SurfaceArgs U{};
    U.G.segs = v->d_seg_rhs; U.G.nseg = v->ncases; U.G.total = v->total_rhs; U.G.stash = nullptr;
    for (int b = 0; b < v->nblocks; ++b) { U.G.q[b] = q_in[b]; U.G.ncell[b] = v->hb[b].ncell; }
    U.W.blocks = v->d_blocks; U.W.cases = v->d_cases; U.W.walls = v->d_walls;
    U.W.nwalls = (int)v->hw.size(); U.W.max_faces = v->max_wall_faces;
    for (int b = 0; b < v->nblocks; ++b) U.W.q[b] = q_in[b];
    std::vector<const double*> spm(v->nblocks, nullptr);
    if (v->any_sponge) {
        U.S.blocks = v->d_blocks; U.S.cases = v->d_cases; U.S.nblocks = v->nblocks;
        U.S.nrows = (int)v->sp_rows.size() / 2; U.S.rows = v->d_sp_rows;
        for (int ci = 0; ci < v->ncases; ++ci)
            for (size_t b = 0; b < v->members[ci]->hb.size(); ++b) {
                const int vb = v->case_block_start[ci] + (int)b;
                U.S.q[vb] = q_in[vb];
                U.S.mean[vb] = v->members[ci]->spmean[b];
                spm[vb] = U.S.mean[vb];
            }
    }
    {
        const bool any = U.G.total > 0 || !v->hw.empty() || v->any_sponge;
        LaunchScope ls(pf, WM_KIND_GHOST, s, any ? 1 : 0);
        CK(launch_surface(U, s));
    }
    StageArgs A{};
    A.blocks = v->d_blocks; A.cases = v->d_cases; A.walls = v->d_walls;
    A.cmf_ctas = v->work[0].ctas() + v->work[1].ctas();
    A.stage = stage;
    A.ncases = v->ncases;
    A.cmf_sum = (stage == 3 && v->any_cmf) ? v->cmf_sum : nullptr;
    A.cmf_counter = v->counters + 1;
    A.cmf_delta = v->cmf_delta;
    for (int ci = 0; ci < v->ncases; ++ci) A.dt[ci] = dt ? dt[ci] : nullptr;
    for (int b = 0; b < v->nblocks; ++b) {
        A.p[b].q_in = q_in[b];
        A.p[b].q0 = q0 ? q0[b] : q_in[b];
        A.p[b].q_out = q_out[b];
        A.p[b].spmean = spm[b];
    }
    for (int x = 0; x < 2; ++x) {
        const View::Work& w = v->work[x];
        if (w.tiles.empty()) continue;
        A.ext = x;
        A.tiles = w.d_tiles;
        A.cta_first = w.d_cta_first;
        A.nctas = w.ctas();
        LaunchScope ls(pf, WM_KIND_STAGE, s);
        CK(launch_stage(A, v->opts, s));
    }
    return WM_OK;
}

// the CFL / constraint pass over q; with q_src (a step's input) it also sets the ghost
// cells of q (the step's output) from q_src's
int run_dt(View* v, Prof* pf, double* const* q, bool apply_cmf, bool want_dt, double* const* dt_out,
           const double* const* q_src, cudaStream_t s) {
    DtArgs D{};
    D.blocks = v->d_blocks; D.cases = v->d_cases; D.nblocks = v->nblocks;
    for (int b = 0; b <= v->nblocks; ++b) D.gcta_start[b] = v->gcta_start[b];
    for (int b = 0; b < v->nblocks; ++b) D.q_src[b] = q_src ? q_src[b] : nullptr;
    D.ncases = v->ncases;
    for (int ci = 0; ci <= v->ncases; ++ci) D.case_block_start[ci] = v->case_block_start[ci];
    for (int b = 0; b < v->nblocks; ++b) D.q[b] = q[b];
    D.cmf_delta = apply_cmf ? v->cmf_delta : nullptr;
    D.want_dt = want_dt ? 1 : 0;
    D.met32 = v->opts.precision == WM_PREC_MIXED ? 1 : 0;
    D.dt_key = v->dt_key; D.counter = v->counters;
    for (int ci = 0; ci < v->ncases; ++ci) D.dt_out[ci] = dt_out ? dt_out[ci] : nullptr;
    // one launch per kind of block in the view; the ghost cells ride on the last
    for (int x = 0; x < 2; ++x) {
        if (v->work[x].blocks.empty()) continue;
        D.ext = x;
        D.finish = x == 1 || v->work[1].blocks.empty() ? 1 : 0;
        D.ncta = v->cta_start[x].back();
        for (int b = 0; b <= v->nblocks; ++b) D.cta_start[b] = v->cta_start[x][b];
        D.ngcta = q_src && D.finish ? v->gcta_start.back() : 0;
        LaunchScope ls(pf, WM_KIND_DT, s);
        CK(launch_dt(D, s));
    }
    return WM_OK;
}

// SSP-RK3 of every case of the view with work states w0/w1 (per view block), then the
// constraint pass; with want_next the pass also writes each case's next CFL time step
int run_step(View* v, Prof* pf, double* const* q_in, double* const* q_out, double* const* w0, double* const* w1,
             const double* const* dt, double* const* dt_next, const double* times, bool want_next, cudaStream_t s) {
    int r;
    if ((r = run_stage(v, pf, 1, q_in, q_in, w0, dt, times, 0.0, s))) return r;
    if ((r = run_stage(v, pf, 2, w0, q_in, w1, dt, times, 1.0, s))) return r;
    if ((r = run_stage(v, pf, 3, w1, q_in, q_out, dt, times, 0.5, s))) return r;
    // constraint, next time step and the output's ghost cells in one pass
    return run_dt(v, pf, q_out, v->any_cmf, want_next, dt_next, q_in, s);
}

}  // namespace

wm_case::~wm_case() { delete self; }

namespace {
// every per-block (or per-case) pointer of an argument array is set: a null one would
// become a device fault
int check_ptrs(const void* const* p, int n, const char* what) {
    if (!p) return fail(WM_E_INVALID, "null %s array", what);
    for (int i = 0; i < n; ++i)
        if (!p[i]) return fail(WM_E_INVALID, "null %s[%d]", what, i);
    return WM_OK;
}
}  // namespace

struct wm_batch {
    View view;
    Prof prof;
    std::vector<double*> w0, w1;     // per view block: the member cases' work states
    unsigned* d_status = nullptr;    // member cases' status words, gathered (wm_batch_status)
};

namespace {
const char* status_names(unsigned st) {
    static thread_local std::string s;
    s.clear();
    const char* names[] = {"non-finite state", "non-positive density", "non-positive pressure",
                           "non-finite or non-positive time step", "wall-model Newton not settled"};
    for (int b = 0; b < 5; ++b)
        if (st & (1u << b)) { if (!s.empty()) s += ", "; s += names[b]; }
    return s.c_str();
}
}  // namespace

extern "C" {

int wm_version(void) { return WM_ABI_VERSION; }
const char* wm_last_error(void) { return g_err.c_str(); }

void wm_case_destroy(wm_case* c) { delete c; }

int wm_case_create(const wm_case_desc* d, wm_case** out) {
    if (!out) return fail(WM_E_INVALID, "null output handle");
    *out = nullptr;
    int r = validate(d);
    if (r) return r;
    wm_case* c = new wm_case();
    auto bail = [&](int code) { delete c; return code; };
    // a failed CUDA call frees the partly built case (its allocations are owned by it)
#define CKB(call)                                                                            \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return bail(fail(WM_E_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), \
                             __FILE__, __LINE__));                                           \
    } while (0)
    CKB(cudaGetDevice(&c->device));

    // ---- physical constants
    const wm_gas& g = d->gas;
    CaseDev& C = c->hc;
    C.gamma = g.gamma; C.Rg = g.R; C.Pr = g.Pr; C.Prt = g.Pr_t; C.mu_ref = g.mu_ref; C.T_ref = g.T_ref;
    C.S_suth = g.S_suth;
    C.gm1 = g.gamma - 1.0;
    C.cp = g.gamma * g.R / C.gm1;
    C.inv_gm1 = 1.0 / C.gm1; C.inv_Rg = 1.0 / g.R; C.inv_Tref = 1.0 / g.T_ref;
    C.TrefS = g.T_ref + g.S_suth; C.inv_Pr = 1.0 / g.Pr; C.inv_Prt = 1.0 / g.Pr_t;
    C.th0 = d->th0; C.inv_dth = 1.0 / (d->th1 - d->th0);
    C.sgs_c = d->sgs_coeff;
    C.cfl = d->cfl;
    C.nu_fac = std::max(4.0 / 3.0, g.gamma / g.Pr);
    C.c_ref = std::sqrt(g.gamma * g.R * g.T_ref);
    C.Pr13 = std::pow(g.Pr, 1.0 / 3.0);
    C.Pr3 = std::pow(g.Pr, 3.0);
    C.kader_beta = std::pow(3.85 * std::pow(g.Pr, 1.0 / 3.0) - 1.3, 2.0) + 2.12 * std::log(g.Pr);
    C.cmf_dir = d->cmf_dir; C.cmf_target = d->cmf_target; C.cmf_volume = d->cmf_volume;
    C.sponge = d->sponge.enabled;
    if (C.sponge) {
        C.sp_xs = d->sponge.x_start_l;
        C.sp_inv_dx = 1.0 / (d->sponge.x_end_l - d->sponge.x_start_l);
        C.sp_sigma0 = d->sponge.strength * d->sponge.U_inf / d->sponge.L;
        C.sp_invL = 1.0 / d->sponge.L;
    }
    // automatic tile (-1): one kernel variant per precision (so cases created with the default
    // can share a batch), the tile shape chosen per block and view (view_tiles)
    c->opts = StageOpts{d->precision, d->scheme, d->kep_order, d->limiter, d->sgs, d->tile < 0 ? -1 : d->tile};

    // ---- blocks, metrics, work buffers
    c->hb.resize(d->nblocks);
    double cells = 0.0;
    for (int b = 0; b < d->nblocks; ++b) cells += (double)d->blocks[b].n[0] * d->blocks[b].n[1] * d->blocks[b].n[2];
    if (C.cmf_dir >= 0) cmf_bins(C, cells);
    for (int b = 0; b < d->nblocks; ++b) {
        const wm_block& src = d->blocks[b];
        BlockDev& B = c->hb[b];
        B.ng = src.ng;
        for (int a = 0; a < 3; ++a) { B.n[a] = src.n[a]; B.N[a] = src.n[a] + 2 * src.ng; }
        B.case_id = 0;
        B.plane = (long long)B.N[1] * B.N[2];
        B.ncell = B.plane * B.N[0];
        for (int f = 0; f < 6; ++f) B.wall[f] = -1;
        B.div_nj.set(B.n[1]);
        B.div_nk.set(B.n[2]);
        if (B.ncell * WM_NMET >= (1LL << 31))
            return bail(fail(WM_E_UNSUPPORTED, "block %d: %lld cells exceed the 32-bit metric index range "
                             "(split the block)", b, B.ncell));
        // the metric table may sit in host or device memory (wm_block_geometry's output);
        // the mixed form's FP32 copy is rounded on the device from the case's FP64 copy
        const size_t nmet = (size_t)WM_NMET * B.ncell;
        cudaPointerAttributes pa{};
        CKB(cudaPointerGetAttributes(&pa, src.metrics));
        const bool on_device = pa.type == cudaMemoryTypeDevice || pa.type == cudaMemoryTypeManaged;
        double* met = nullptr;
        if ((r = c->mem.alloc(&met, nmet))) return bail(r);
        CKB(cudaMemcpy(met, src.metrics, sizeof(double) * nmet,
                       on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
        B.met = met;
        B.met32 = nullptr;
        if (d->precision == WM_PREC_MIXED) {
            float* p32 = nullptr;
            if ((r = c->mem.alloc(&p32, nmet))) return bail(r);
            CKB(launch_to_f32(met, p32, (long long)nmet, 0));
            B.met32 = p32;
        }
        if ((r = extruded_tables(c, B, d->precision))) return bail(r);
        for (int s = 0; s < 2; ++s) {
            double* w = nullptr;
            if ((r = c->mem.alloc(&w, 5 * (size_t)B.ncell))) return bail(r);
            CKB(cudaMemset(w, 0, sizeof(double) * 5 * B.ncell));
            c->work[s].push_back(w);
        }
    }

    // ---- wall-modelled faces
    for (int w = 0; w < d->nwalls; ++w) {
        const wm_wall& src = d->walls[w];
        BlockDev& B = c->hb[src.block];
        const int ta = src.axis == 0 ? 1 : 0, tb = src.axis == 2 ? 1 : 2;
        WallDev W{};
        W.block = src.block; W.axis = src.axis; W.side = src.side; W.n_match = src.n_match;
        W.isothermal = src.isothermal; W.n_iter = src.n_iter;
        W.nt1 = B.n[ta]; W.nt2 = B.n[tb];
        W.T_wall = src.T_wall; W.kappa = src.kappa; W.B = src.B; W.ekb = std::exp(-src.kappa * src.B);
        const size_t nf = (size_t)W.nt1 * W.nt2;
        double* gm = nullptr;
        if ((r = c->mem.upload(&gm, src.geom, 5 * nf))) return bail(r);
        W.geom = gm;
        if ((r = c->mem.alloc(&W.F, 5 * nf))) return bail(r);
        if ((r = c->mem.alloc(&W.tq, 2 * nf))) return bail(r);
        if (B.wall[2 * src.axis + src.side] >= 0) return bail(fail(WM_E_INVALID, "two walls on one face"));
        B.wall[2 * src.axis + src.side] = w;
        c->hw.push_back(W);
    }

    // ---- ghost programs and BC constants
    if ((r = c->mem.upload(&c->d_bc, d->bc_table, 8 * (size_t)std::max(d->nbc, 1)))) return bail(r);
    if ((r = upload_prog(c, &c->prog_rhs, d->ghost_rhs))) return bail(r);
    if ((r = upload_prog(c, &c->prog_all, d->ghost_all))) return bail(r);
    if ((r = c->mem.alloc(&c->stash, 5 * (size_t)std::max(d->ghost_all.count, 1)))) return bail(r);

    // ---- synthetic inflow
    if (d->inflow) {
        const wm_inflow& I = *d->inflow;
        if (I.block < 0 || I.block >= d->nblocks) return bail(fail(WM_E_INVALID, "inflow block"));
        c->has_inflow = true;
        c->inflow = I;
        c->inflow_block = I.block;
        if ((r = c->mem.upload(&c->d_modes, I.modes, 12 * (size_t)I.n_modes))) return bail(r);
        if ((r = c->mem.upload(&c->d_table, I.table, 7 * (size_t)I.n_tab))) return bail(r);
        const BlockDev& B = c->hb[I.block];
        c->inflow_n = (long long)B.ng * B.plane;
        if ((r = c->mem.alloc(&c->inflow_buf, 5 * (size_t)c->inflow_n))) return bail(r);
        if ((r = c->mem.alloc(&c->inflow_raw, (size_t)IN_PARTS * 3 * c->inflow_n))) return bail(r);
        if ((r = c->mem.alloc(&c->inflow_prof, 6 * (size_t)c->inflow_n))) return bail(r);
        if ((r = c->mem.upload(&c->d_inflow_block, &B, 1))) return bail(r);
        // extruded plane: every ghost row's y constant along k, z the same function of k on
        // every row (then the mode sums factor per row and per k); one component's cos / sin
        // (kz z) table must fit the mode-sum launch's shared memory
        const size_t n = (size_t)c->inflow_n;
        std::vector<double> y(n), z(n);
        CKB(cudaMemcpy(y.data(), B.met + (size_t)WM_MET_XCY * B.ncell, sizeof(double) * n, cudaMemcpyDeviceToHost));
        CKB(cudaMemcpy(z.data(), B.met + (size_t)WM_MET_XCZ * B.ncell, sizeof(double) * n, cudaMemcpyDeviceToHost));
        const int Nk = B.N[2];
        bool extruded = inflow_ext_smem(I.n_modes, Nk) <= inflow_ext_smem_max();
        for (size_t cell = 0; cell < n && extruded; ++cell) {
            const size_t k = cell % Nk;
            extruded = y[cell] == y[cell - k] && z[cell] == z[k];
        }
        InflowArgs IA{};
        IA.block = c->d_inflow_block;
        IA.modes = c->d_modes; IA.table = c->d_table;
        IA.n_modes = I.n_modes; IA.n_tab = I.n_tab;
        IA.U_inf = I.U_inf; IA.L = I.L;
        if (extruded)
            if ((r = c->mem.alloc(&c->inflow_cz, 2 * 3 * (size_t)I.n_modes * Nk))) return bail(r);
        CKB(launch_inflow_setup(IA, B.N[1], Nk, B.ng, c->inflow_prof, c->inflow_cz, 0));
    }

    // ---- sponge means
    c->spmean.assign(d->nblocks, nullptr);
    if (d->sponge.enabled) {
        for (int b = 0; b < d->nblocks; ++b) {
            const BlockDev& B = c->hb[b];
            if ((r = c->mem.alloc(&c->spmean[b], 5 * (size_t)B.N[0] * B.N[1]))) return bail(r);
            // rows outside the sponge are never written (their mean is not needed): keep them 0
            CKB(cudaMemset(c->spmean[b], 0, sizeof(double) * 5 * B.N[0] * B.N[1]));
            const int rows = B.n[0] * B.n[1];
            unsigned char* d_flags = nullptr;
            if ((r = c->mem.alloc(&d_flags, (size_t)rows))) return bail(r);
            CKB(launch_sponge_flags(B.met + (size_t)WM_MET_XCX * B.ncell, B.plane, B.N[2], B.ng, B.n[0], B.n[1],
                                    B.n[2], C.sp_invL, C.sp_xs, C.sp_inv_dx, d_flags, 0));
            std::vector<unsigned char> flags((size_t)rows);
            CKB(cudaMemcpy(flags.data(), d_flags, (size_t)rows, cudaMemcpyDeviceToHost));
            for (int row = 0; row < rows; ++row)
                if (flags[row]) { c->sp_rows.push_back(b); c->sp_rows.push_back(row); }
        }
    }

    c->chunk_req = d->chunk > 0 ? d->chunk : 0;

    // ---- plane-statistics scratch
    int max_nj = 1;
    for (const BlockDev& B : c->hb) max_nj = std::max(max_nj, B.n[1]);
    if ((r = c->mem.alloc(&c->ps_part, (size_t)PS_NQ * max_nj * PS_CHUNKS))) return bail(r);
    if ((r = c->mem.alloc(&c->ps_counter, (size_t)max_nj))) return bail(r);
    CKB(cudaMemset(c->ps_counter, 0, sizeof(unsigned) * max_nj));

    // ---- status word (every view of the case points at it)
    if ((r = c->mem.alloc(&c->d_status, 1))) return bail(r);
    CKB(cudaMemset(c->d_status, 0, sizeof(unsigned)));
    c->hc.status = c->d_status;

    c->self = new View();
    wm_case* self_list[1] = {c};
    if ((r = build_view(c->self, self_list, 1))) return bail(r);
    CKB(cudaDeviceSynchronize());
    *out = c;
    return WM_OK;
#undef CKB
}

int wm_apply_bcs(wm_case* c, double* const* q, double time, void* stream) {
    if (!c) return fail(WM_E_INVALID, "null case");
    if (int r = check_ptrs((const void* const*)q, c->self->nblocks, "q")) return r;
    cudaStream_t s = (cudaStream_t)stream;
    View* v = c->self;
    int r;
    if ((r = fill_inflow(v, &c->prof, &time, 0.0, nullptr, s))) return r;
    GhostArgs G{};
    G.segs = v->d_seg_all; G.nseg = 1; G.total = v->total_all; G.stash = c->stash;
    for (int b = 0; b < v->nblocks; ++b) { G.q[b] = q[b]; G.ncell[b] = v->hb[b].ncell; }
    LaunchScope ls(&c->prof, WM_KIND_GHOST, s, G.total ? 2 : 0);
    CK(launch_ghost(G, s));
    return WM_OK;
}

int wm_rhs(wm_case* c, double* const* q, double* const* rr, double time, void* stream) {
    if (!c) return fail(WM_E_INVALID, "null case");
    if (int r = check_ptrs((const void* const*)q, c->self->nblocks, "q")) return r;
    if (int r = check_ptrs((const void* const*)rr, c->self->nblocks, "r")) return r;
    return run_stage(c->self, &c->prof, 0, q, nullptr, rr, nullptr, &time, 0.0, (cudaStream_t)stream);
}

int wm_max_dt(wm_case* c, const double* const* q, double* dt_dev, void* stream) {
    if (!c || !dt_dev) return fail(WM_E_INVALID, "null argument");
    if (int r = check_ptrs((const void* const*)q, c->self->nblocks, "q")) return r;
    return run_dt(c->self, &c->prof, const_cast<double* const*>(q), false, true, &dt_dev, nullptr,
                  (cudaStream_t)stream);
}

int wm_advance(wm_case* c, double* const* q_in, double* const* q_out, const double* dt_dev, double time,
               void* stream) {
    if (!c || !dt_dev) return fail(WM_E_INVALID, "null argument");
    if (int r = check_ptrs((const void* const*)q_in, c->self->nblocks, "q_in")) return r;
    if (int r = check_ptrs((const void* const*)q_out, c->self->nblocks, "q_out")) return r;
    return run_step(c->self, &c->prof, q_in, q_out, c->work[0].data(), c->work[1].data(), &dt_dev, nullptr, &time,
                    false, (cudaStream_t)stream);
}

int wm_step(wm_case* c, double* const* q_in, double* const* q_out, double* dt_dev, double time, void* stream) {
    int r = wm_max_dt(c, q_in, dt_dev, stream);
    if (r) return r;
    return wm_advance(c, q_in, q_out, dt_dev, time, stream);
}

int wm_step_fused(wm_case* c, double* const* q_in, double* const* q_out, const double* dt_in, double* dt_next,
                  double time, void* stream) {
    if (!c || !dt_in || !dt_next) return fail(WM_E_INVALID, "null argument");
    if (int r = check_ptrs((const void* const*)q_in, c->self->nblocks, "q_in")) return r;
    if (int r = check_ptrs((const void* const*)q_out, c->self->nblocks, "q_out")) return r;
    return run_step(c->self, &c->prof, q_in, q_out, c->work[0].data(), c->work[1].data(), &dt_in, &dt_next, &time,
                    true, (cudaStream_t)stream);
}

int wm_case_status(wm_case* c, unsigned* status, int clear, void* stream) {
    if (!c || !status) return fail(WM_E_INVALID, "null argument");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned st = 0;
    CK(cudaMemcpyAsync(&st, c->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    if (clear) CK(cudaMemsetAsync(c->d_status, 0, sizeof(unsigned), s));
    CK(cudaStreamSynchronize(s));
    *status = st;
    return WM_OK;
}

int wm_check(wm_case* c, void* stream) {
    unsigned st = 0;
    if (int r = wm_case_status(c, &st, 1, stream)) return r;
    if (st & WM_ST_FATAL) return fail(WM_E_NONFINITE, "case status 0x%x: %s", st, status_names(st));
    return WM_OK;
}

int wm_wall_stats(wm_case* c, const double* const* q, double* const* out, void* stream) {
    if (!c) return fail(WM_E_INVALID, "null case");
    if (int r = check_ptrs((const void* const*)q, c->self->nblocks, "q")) return r;
    if (int r = check_ptrs((const void* const*)out, (int)c->self->hw.size(), "out")) return r;
    cudaStream_t s = (cudaStream_t)stream;
    View* v = c->self;
    if (v->hw.empty()) return WM_OK;
    WallArgs W{};
    W.blocks = v->d_blocks; W.cases = v->d_cases; W.walls = v->d_walls;
    W.nwalls = (int)v->hw.size(); W.max_faces = v->max_wall_faces;
    for (int b = 0; b < v->nblocks; ++b) W.q[b] = q[b];
    {
        LaunchScope ls(&c->prof, WM_KIND_WALL, s);
        CK(launch_wall(W, s));
    }
    for (size_t w = 0; w < v->hw.size(); ++w) {
        const size_t nf = (size_t)v->hw[w].nt1 * v->hw[w].nt2;
        CK(cudaMemcpyAsync(out[w], v->hw[w].tq, sizeof(double) * 2 * nf, cudaMemcpyDeviceToDevice, s));
    }
    return WM_OK;
}

int wm_plane_stats(wm_case* c, int block, const double* q, double* sum, void* stream) {
    if (!c || !q || !sum) return fail(WM_E_INVALID, "null argument");
    if (block < 0 || block >= c->self->nblocks) return fail(WM_E_INVALID, "block %d out of range", block);
    PlaneStatsArgs A{};
    A.block = c->self->d_blocks + block;
    A.q = q;
    A.gm1 = c->hc.gm1;
    A.Rg = c->hc.Rg;
    A.nchunks = plane_chunks(c->hb[block].n[0], c->hb[block].n[1]);
    A.part = c->ps_part;
    A.sum = sum;
    A.counter = c->ps_counter;
    CK(launch_plane_stats(A, c->hb[block].n[1], (cudaStream_t)stream));
    return WM_OK;
}

int wm_derived_fields(wm_case* c, const double* const* q, double* const* out, void* stream) {
    if (!c) return fail(WM_E_INVALID, "null case");
    if (int r = check_ptrs((const void* const*)q, c->self->nblocks, "q")) return r;
    if (int r = check_ptrs((const void* const*)out, c->self->nblocks, "out")) return r;
    View* v = c->self;
    for (int b = 0; b < v->nblocks; ++b) {
        DerivedArgs A{};
        A.block = v->d_blocks + b;
        A.cs = v->d_cases;
        A.sgs = c->opts.sgs;
        A.q = q[b];
        A.out = out[b];
        CK(launch_derived(A, v->hb[b].n, (cudaStream_t)stream));
    }
    return WM_OK;
}

int wm_block_geometry(const double* X, const int* N, double* vol, double* xc, double* const* S,
                      double* const* xf, double* met, void* stream) {
    if (!X || !N || !vol || !xc || !S || !xf) return fail(WM_E_INVALID, "null argument");
    GeomArgs A{};
    A.X = X;
    for (int d = 0; d < 3; ++d) {
        if (N[d] < 1) return fail(WM_E_INVALID, "N[%d] = %d: every direction needs a cell", d, N[d]);
        if (!S[d] || !xf[d]) return fail(WM_E_INVALID, "null face array of direction %d", d);
        A.N[d] = N[d];
        A.S[d] = S[d];
        A.xf[d] = xf[d];
    }
    A.vol = vol;
    A.xc = xc;
    A.met = met;
    CK(launch_geometry(A, (cudaStream_t)stream));
    return WM_OK;
}

int wm_batch_create(int ncases, wm_case* const* cases, wm_batch** out) {
    if (!out || !cases) return fail(WM_E_INVALID, "null argument");
    *out = nullptr;
    wm_batch* b = new wm_batch();
    int r = build_view(&b->view, cases, ncases);
    if (r) { delete b; return r; }
    for (int ci = 0; ci < ncases; ++ci)
        for (size_t k = 0; k < cases[ci]->hb.size(); ++k) {
            b->w0.push_back(cases[ci]->work[0][k]);
            b->w1.push_back(cases[ci]->work[1][k]);
        }
    if ((r = b->view.mem.alloc(&b->d_status, (size_t)ncases))) { delete b; return r; }
    *out = b;
    return WM_OK;
}

void wm_batch_destroy(wm_batch* b) { delete b; }

int wm_batch_status(wm_batch* b, unsigned* status, void* stream) {
    if (!b || !status) return fail(WM_E_INVALID, "null argument");
    cudaStream_t s = (cudaStream_t)stream;
    CK(launch_status_gather(b->view.d_cases, b->view.ncases, b->d_status, s));
    CK(cudaMemcpyAsync(status, b->d_status, sizeof(unsigned) * b->view.ncases, cudaMemcpyDeviceToHost, s));
    return WM_OK;
}

int wm_batch_step(wm_batch* b, double* const* q_in, double* const* q_out, const double* const* dt_in,
                  double* const* dt_next, const double* times, void* stream) {
    if (!b || !times) return fail(WM_E_INVALID, "null argument");
    const View& v = b->view;
    if (int r = check_ptrs((const void* const*)q_in, v.nblocks, "q_in")) return r;
    if (int r = check_ptrs((const void* const*)q_out, v.nblocks, "q_out")) return r;
    if (int r = check_ptrs((const void* const*)dt_in, v.ncases, "dt_in")) return r;
    if (int r = check_ptrs((const void* const*)dt_next, v.ncases, "dt_next")) return r;
    return run_step(&b->view, &b->prof, q_in, q_out, b->w0.data(), b->w1.data(), dt_in, dt_next, times, true,
                    (cudaStream_t)stream);
}

int wm_batch_info(wm_batch* b, int* nblocks, int* ntiles, long long* launches_per_step) {
    if (!b) return fail(WM_E_INVALID, "null batch");
    const View& v = b->view;
    int inflow = 0;
    for (wm_case* c : v.members) inflow += c->has_inflow ? 1 : 0;
    const int kinds = (v.work[0].tiles.empty() ? 0 : 1) + (v.work[1].tiles.empty() ? 0 : 1);
    const long long per_stage = IN_LAUNCHES * inflow + ((v.total_rhs || !v.hw.empty() || v.any_sponge) ? 1 : 0) + kinds;
    if (nblocks) *nblocks = v.nblocks;
    if (ntiles) *ntiles = (int)(v.work[0].tiles.size() + v.work[1].tiles.size());
    if (launches_per_step) *launches_per_step = 3 * per_stage + kinds;
    return WM_OK;
}

int wm_profile_enable(wm_case* c, int enable) {
    if (!c) return fail(WM_E_INVALID, "null case");
    c->prof.reset(enable != 0);
    return WM_OK;
}

int wm_profile_read(wm_case* c, int kind, double* ms_total, long long* launches) {
    if (!c || kind < -1 || kind >= WM_NKINDS) return fail(WM_E_INVALID, "bad profile query");
    double ms = 0.0;
    for (auto& r : c->prof.recs) {
        if (kind >= 0 && r.kind != kind) continue;
        CK(cudaEventSynchronize(r.b));
        float t = 0.f;
        CK(cudaEventElapsedTime(&t, r.a, r.b));
        ms += t;
    }
    long long n = 0;
    for (int k = 0; k < WM_NKINDS; ++k)
        if (kind < 0 || k == kind) n += c->prof.nlaunch[k];
    if (ms_total) *ms_total = ms;
    if (launches) *launches = n;
    return WM_OK;
}

}  // extern "C"
