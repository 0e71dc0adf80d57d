// Fused RHS + SSP-RK3 stage kernel.
//
// One CTA owns a tj x tk tile of (j,k) columns of one block and marches along i over a
// chunk of planes [i0, i1).  Shared memory holds
//   pr[4]  primitive records of planes i-1..i+2 (FP64; float form i-2..i+1) on the tile + 2-cell
//          halo (rolling ring)
//   gs     Green-Gauss gradients, mu_eff, k_eff (and the Ducros sensor) of plane i on the
//          tile + 1-cell halo
//   ff     the j- and k-face fluxes of plane i
//   rt     (extruded grids) the metrics of the tile's rows of planes i and i+1
//   qs     (float form) the conservative values of the next plane to convert, by cp.async
//   hp, hg, fr (FP64) per column: plane i-2's primitives, plane i-1's gradient record, the flux
//          divergence being summed
// FP64: two phases per plane, separated by barriers,
//   1. gradient records of plane i; the warps without a record finish plane i-2 (RK epilogue),
//      convert plane i+2 and take the j/k flux differences of plane i-1
//   2. own i-face flux; all j/k faces of plane i (flat loop); the warps without a record also
//      prefetch, and load what they need in the next phase 1 into registers
// Float form: three phases, conversion of plane i+1; gradient records; faces and the RK
// epilogue of plane i-1.
// Each face flux is evaluated once; each conservative value is read from HBM about once
// per stage (halo re-reads hit L2).  Stage 3 also sums rho u V for the constant-mass-flux
// constraint.
//
// Reference: Solver._block_rhs (wmles/solver.py:76-95), green_gauss / viscous_flux /
// ducros (wmles/viscous.py), schemes (wmles/schemes.py), SGS (wmles/sgs.py), SSP-RK3
// (wmles/solver.py:110-121).
#include <algorithm>
#include <cstdio>
#include <type_traits>
#include "physics.cuh"
#include "stage.cuh"

namespace wm {

// A kernel instance holds up to CAP columns; the tile shape tj x tk is a run-time value per
// segment (any shape within the capacities below), so a block's extents are cut into equal
// tiles instead of 32-wide ones with a nearly empty remainder.  The index arithmetic of a
// segment (cell of each record, face, column) is done once, into tables in shared memory.
//
// FP64: 256 columns, one CTA of 512 threads per SM.  16 warps rather than the 8 the columns
// need: they take a share of every flat loop, and more warps hide the FP64 latency, at the price
// of 128 registers a thread.  Float form: 512 columns, one CTA of 640 threads (96 registers),
// or, for the small tile shapes when asked for, 256 columns in two CTAs of 256 threads per SM
// (128 registers).
//
// EXT: the kernel for blocks extruded along k (checked at case creation, capi.cu): their area
// and centre-to-centre vectors depend on (i, j) alone, up to one factor per k on the areas of i
// and j faces.  Their metrics come from a row of 16 values per (i, j), staged for the tile's
// rows one plane ahead, and a pair of values per k; only 1/V and the filter width are read
// per cell.
template <typename R, int SCHEME, int CAP, bool EXT>
struct StageLayout {
    static constexpr int NTH = sizeof(R) == 8 ? 512 : (CAP == 512 ? 640 : 256);     // threads
    static constexpr int MIN_CTAS = sizeof(R) == 4 && CAP == 256 ? 2 : 1;           // per SM
    static constexpr int PN = stage_caps(CAP).pn;      // primitives: tile + 2-cell halo
    static constexpr int GN = stage_caps(CAP).gn;      // gradient records: tile + 1-cell halo
    static constexpr int FN = stage_caps(CAP).fn;      // j faces, then k faces
    static constexpr int RN = EXT ? stage_caps(CAP).rows : 0;      // rows of the tile + 1-row halo + 1
    static constexpr int KN = EXT ? stage_caps(CAP).kn : 0;        // k positions of the tile + 1-cell halo
    // values of a gradient record, and how many of them lie side by side: component v of record c at
    // [v / GV][c][v % GV], so that a face takes a record in 16-byte loads.  General grids, where these
    // loads wait in one queue with those of the metrics: fours (float) or pairs (FP64; the Hybrid form has
    // no room for the 16th value).  Box 160 x 96 x 72, KEP, float 1117 -> 1083 us for two steps, box 75 x
    // 53 x 37, MUSCL, FP64 485 -> 472.  Extruded grids have fewer loads and, in float, no registers
    // to spare: channel, three steps, float 3681 -> 3945, FP64 6411 -> 6461, so one by one there
    static constexpr int GV = EXT ? 1 : sizeof(R) == 4 ? 4 : SCHEME == WM_SCHEME_HYBRID ? 1 : 2;
    static constexpr int NGS = GV == 4 ? 16 : (SCHEME == WM_SCHEME_HYBRID) ? 15 : 14;
    // FP64: plane i+2 is converted while the gradient records of plane i are computed, by the warps that
    // have no record to compute, and a plane takes two barriers instead of three.  It goes into the slot of plane
    // i-2, whose records the columns have copied (hp).  The float form has a record for nearly every thread and
    // keeps three phases.
    static constexpr bool FUSE = sizeof(R) == 8;
    static constexpr int NSLOT = 4;
    static constexpr int HP_N = 6;
    static constexpr size_t qs_off = 0;                                        // float form: double [5][PN]
    static constexpr size_t pr_off = qs_off + (FUSE ? 0 : sizeof(double) * 5 * PN);    // R [NSLOT][PR_N][PN]
    static constexpr size_t gs_off = pr_off + sizeof(R) * NSLOT * PR_N * PN;   // R [NGS][GN]
    // FP64: two planes of gradient records in turn where the shared memory is there (PING), else the
    // columns' last ones copied (hg)
    static constexpr bool PING = FUSE && !(EXT && SCHEME == WM_SCHEME_HYBRID);
    static constexpr size_t ff_off = gs_off + sizeof(R) * NGS * GN * (PING ? 2 : 1);   // R [5][FN]
    // FP64, per tile column: the flux divergence of the output plane; the primitive record (without
    // T) of plane i-2 and (no PING) the gradient record of plane i-1, which would hold 28 registers
    // through the gradient phase
    static constexpr size_t fr_off = ff_off + sizeof(R) * 5 * FN;              // R [5][CAP]
    static constexpr size_t hp_off = fr_off + (FUSE ? sizeof(R) * 5 * CAP : 0);        // R [HP_N][CAP]
    static constexpr size_t hg_off = hp_off + (FUSE ? sizeof(R) * HP_N * CAP : 0);     // R [NGS][CAP]
    static constexpr size_t red_off = (hg_off + (FUSE && !PING ? sizeof(R) * NGS * CAP : 0) + 15) / 16 * 16;
    // mass-flux sums of the warps (three bins each), the bins' rounding constants
    static constexpr size_t cs_off = red_off + (sizeof(double) * 3 * (NTH / 32 + 1) + 15) / 16 * 16;   // float form: double [3][CAP]
    static constexpr size_t rt_off = cs_off + (FUSE ? 0 : sizeof(double) * 3 * CAP);                   // R [2][RN][RT_N]
    static constexpr size_t kt_off = rt_off + sizeof(R) * 2 * RN * RT_N;               // R [KN][2]
    // index tables of the segment
    static constexpr size_t ft_off = kt_off + sizeof(R) * 2 * KN;                      // int [FN]
    static constexpr size_t pt_off = ft_off + 4 * FN;                                  // int [PN]
    static constexpr size_t ct_off = pt_off + 4 * PN;                                  // int [CAP]
    static constexpr size_t ph_off = (ct_off + 4 * CAP + 7) / 8 * 8;                   // Phys<R>
    static constexpr size_t bytes = ph_off + (sizeof(Phys<R>) + 7) / 8 * 8;
    static constexpr int GW = (GN + 31) / 32 * 32;     // threads of the warps with a record, at most
    static_assert(!FUSE || 2 * (NTH - GW) >= CAP, "at most two epilogue columns per thread");
    static_assert(rt_off % 16 == 0, "rows arrive in 16-byte pieces");
    static_assert(GV == 1 || gs_off % 16 == 0, "gradient records are read in 16-byte pieces");
    static_assert(bytes * MIN_CTAS <= 227 * 1024, "shared memory of an SM");
};

// gradient record: g[0..11] = d(u,v,w,T)/d(x,y,z), 12 = mu_eff, 13 = k_eff (all at half
// scale), 14 = theta
enum { GS_MU = 12, GS_K = 13, GS_TH = 14 };

// metric component arrays in the compute precision
template <typename R>
__device__ __forceinline__ const R* metbase(const BlockDev& B) {
    if constexpr (sizeof(R) == 4) return B.met32;
    else return B.met;
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
// a value of a state: not by the read-only path, which wants data that nothing writes during the kernel's
// life, and this kernel may come up while the launch before it still writes (chain_wait)
__device__ __forceinline__ double ld_state(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];\n" ::"l"(p)); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// viscous flux of momentum and energy through one face (times area; to be subtracted),
// wmles/viscous.py:28-51.  gL/gR index a
// gradient record (half scale: the face average of two records is their sum, the same
// value bit for bit as 0.5 (a + b), since scaling by two is exact); pl/pr point at primitive
// records with component stride s; (e0, e1, e2) is the unit vector from the L to the R cell
// centre and idist the inverse distance.
template <int FACE, typename R, class GL, class GR>
__device__ __forceinline__ void viscous_flux(const R* pl, const R* pr, int s, GL gL, GR gR, R Sx, R Sy, R Sz,
                                             R e0, R e1, R e2, R idist, R V[4]) {
    // a record's components one by one, or GW at a time (StageLayout::GV)
    constexpr int GW = sizeof(decltype(gL(0))) / sizeof(R);
    R gf[12], sum[GW > 1 ? 16 : 1];
    if constexpr (GW > 1) {
#pragma unroll
        for (int x = 0; x < (GS_TH + GW - 1) / GW; ++x) {
            const auto l = gL(x), r = gR(x);
#pragma unroll
            for (int y = 0; y < GW; ++y)
                sum[GW * x + y] = reinterpret_cast<const R*>(&l)[y] + reinterpret_cast<const R*>(&r)[y];
        }
    }
    auto add = [&](int v) {
        if constexpr (GW > 1) return sum[v];
        else return gL(v) + gR(v);
    };
    const int pv[4] = {PR_U, PR_V, PR_W, PR_T};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const R b0 = add(3 * a), b1 = add(3 * a + 1), b2 = add(3 * a + 2);
        const R be = FACE == FACE_Z ? b2 : FACE == FACE_XY ? b0 * e0 + b1 * e1 : b0 * e0 + b1 * e1 + b2 * e2;
        const R corr = (pr[pv[a] * s] - pl[pv[a] * s]) * idist - be;
        gf[3 * a] = FACE == FACE_Z ? b0 : b0 + corr * e0;
        gf[3 * a + 1] = FACE == FACE_Z ? b1 : b1 + corr * e1;
        gf[3 * a + 2] = FACE == FACE_Z ? b2 + corr : FACE == FACE_XY ? b2 : b2 + corr * e2;
    }
    const R div = gf[0] + gf[4] + gf[8];
    const R muf = add(GS_MU);
    const R kf = add(GS_K);
    const R d23 = R(2.0 / 3.0) * div;
    const R t00 = muf * (gf[0] + gf[0] - d23), t11 = muf * (gf[4] + gf[4] - d23), t22 = muf * (gf[8] + gf[8] - d23);
    const R t01 = muf * (gf[1] + gf[3]), t02 = muf * (gf[2] + gf[6]), t12 = muf * (gf[5] + gf[7]);
    const R ts0 = dot_s<FACE>(t00, t01, t02, Sx, Sy, Sz);
    const R ts1 = dot_s<FACE>(t01, t11, t12, Sx, Sy, Sz);
    const R ts2 = dot_s<FACE>(t02, t12, t22, Sx, Sy, Sz);
    const R dTdn = dot_s<FACE>(gf[9], gf[10], gf[11], Sx, Sy, Sz);
    const R uf = R(0.5) * (pl[PR_U * s] + pr[PR_U * s]);
    const R vf = R(0.5) * (pl[PR_V * s] + pr[PR_V * s]);
    const R wf = R(0.5) * (pl[PR_W * s] + pr[PR_W * s]);
    V[0] = ts0;
    V[1] = ts1;
    V[2] = ts2;
    V[3] = (uf * ts0 + vf * ts1 + wf * ts2) + kf * dTdn;
}

// MUSCL-HLLC flux.  FP64: one copy of the code for every face of a kernel; inlined per face
// direction, the Hybrid kernel's loop outgrew the instruction cache (5.3 of 17 stall cycles per
// instruction waited for instructions, C-grid, 8 x 32 tiles; stage launch 944 us against 678 with
// one copy).  The float form's code is half as long and runs faster inlined.
template <typename R>
struct Flux5 {
    R f[5];
};
template <typename R>
__device__ __noinline__ Flux5<R> muscl_call(int limiter, const Phys<R>& P, const R* L2, int s2, const R* L, const R* Rr,
                                            const R* R2, int s, R Sx, R Sy, R Sz) {
    Flux5<R> F;
    muscl_hllc_flux<FACE_ANY>(limiter, L2, s2, L, Rr, R2, s, Sx, Sy, Sz, P, F.f);
    return F;
}
template <int FACE, typename R>
__device__ __forceinline__ void muscl_flux(int limiter, const Phys<R>& P, const R* L2, int s2, const R* L, const R* Rr,
                                           const R* R2, int s, R Sx, R Sy, R Sz, R F[5]) {
    if constexpr (sizeof(R) == 8) {
        const Flux5<R> I = muscl_call(limiter, P, L2, s2, L, Rr, R2, s, Sx, Sy, Sz);
#pragma unroll
        for (int v = 0; v < 5; ++v) F[v] = I.f[v];
    } else {
        muscl_hllc_flux<FACE>(limiter, L2, s2, L, Rr, R2, s, Sx, Sy, Sz, P, F);
    }
}

// total face flux (inviscid scheme + viscous), S = face area vector, e / idist = unit
// centre-to-centre vector and its inverse length
template <int FACE, typename R, int SCHEME, class GL, class GR>
__device__ __forceinline__ void face_flux(const StageOpts& o, const Phys<R>& P, const R* L2, int s2, const R* L,
                                          const R* Rr, const R* R2, int s, GL gL, GR gR, R Sx, R Sy,
                                          R Sz, R e0, R e1, R e2, R idist, R F[5]) {
    R V[4];
    if constexpr (SCHEME == WM_SCHEME_KEP) {
        kep_flux<FACE>(o.kep_order, L2, s2, L, Rr, R2, s, Sx, Sy, Sz, F);
        viscous_flux<FACE, R>(L, Rr, s, gL, gR, Sx, Sy, Sz, e0, e1, e2, idist, V);
    } else {
        // the viscous part first: less to keep over the call
        viscous_flux<FACE, R>(L, Rr, s, gL, gR, Sx, Sy, Sz, e0, e1, e2, idist, V);
        if constexpr (SCHEME == WM_SCHEME_MUSCL) {
            muscl_flux<FACE>(o.limiter, P, L2, s2, L, Rr, R2, s, Sx, Sy, Sz, F);
        } else {
            // Ducros-switched blend, wmles/schemes.py:163-166
            R th;
            constexpr int GW = sizeof(decltype(gL(0))) / sizeof(R);
            if constexpr (GW == 4) th = fmax(gL(3).z, gR(3).z);
            else th = fmax(gL(GS_TH), gR(GS_TH));
            const R sw = fmin(fmax((th - P.th0) * P.inv_dth, R(0)), R(1));
            R Fc[5] = {R(0), R(0), R(0), R(0), R(0)}, Fu[5] = {R(0), R(0), R(0), R(0), R(0)};
            if (sw > R(0)) muscl_flux<FACE>(o.limiter, P, L2, s2, L, Rr, R2, s, Sx, Sy, Sz, Fu);
            if (sw < R(1)) kep_flux<FACE>(o.kep_order, L2, s2, L, Rr, R2, s, Sx, Sy, Sz, Fc);
#pragma unroll
            for (int v = 0; v < 5; ++v) F[v] = (sw == R(0)) ? Fc[v] : (sw == R(1)) ? Fu[v] : (R(1) - sw) * Fc[v] + sw * Fu[v];
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) F[1 + v] -= V[v];
}

// Face table: row and k position of the R cell in the tile (row | k << 8) and flags.  Primitive
// and column tables: (j,k) offset in a plane of the block.
enum { FT_K = 1 << 20, FT_WLO = 1 << 21, FT_WHI = 1 << 22 };

// one segment of a CTA's work: tile t (a (j,k) column of one block over planes [t.i0, t.i1))
template <typename R, int SCHEME, int CAP, bool EXT>
__device__ __forceinline__ void stage_segment(const StageArgs& A, const StageOpts& o, const Tile t,
                                              unsigned char* smem_raw) {
    using LY = StageLayout<R, SCHEME, CAP, EXT>;
    constexpr int NTH = LY::NTH, NW = NTH / 32, PN = LY::PN, GN = LY::GN, FN = LY::FN, NGS = LY::NGS;
    constexpr bool FUSE = LY::FUSE;
    double* qs = reinterpret_cast<double*>(smem_raw + LY::qs_off);
    R* pr = reinterpret_cast<R*>(smem_raw + LY::pr_off);
    R* const gs0 = reinterpret_cast<R*>(smem_raw + LY::gs_off);
    R* gs = gs0;                                   // the march's plane
    R* ff = reinterpret_cast<R*>(smem_raw + LY::ff_off);
    R* fr = reinterpret_cast<R*>(smem_raw + LY::fr_off);
    R* hp = reinterpret_cast<R*>(smem_raw + LY::hp_off) + threadIdx.x;
    R* hg = reinterpret_cast<R*>(smem_raw + LY::hg_off) + threadIdx.x;
    double* red = reinterpret_cast<double*>(smem_raw + LY::red_off);
    R* rt = reinterpret_cast<R*>(smem_raw + LY::rt_off);
    R* kt = reinterpret_cast<R*>(smem_raw + LY::kt_off);
    int* ft = reinterpret_cast<int*>(smem_raw + LY::ft_off);
    int* pt = reinterpret_cast<int*>(smem_raw + LY::pt_off);
    int* ct = reinterpret_cast<int*>(smem_raw + LY::ct_off);

    const BlockDev& B = A.blocks[t.blk];
    const CaseDev& C = A.cases[B.case_id];
    // the physical constants: in shared memory, 15 values that would hold 30 registers (FP64) through
    // every phase (general grids in FP64, where shared memory is busiest: left to the compiler; box
    // 192 x 112 x 96, KEP: 2860 -> 2820 us a pass)
    constexpr bool PSH = EXT || !LY::FUSE;
    const Phys<R> Preg(C);
    const Phys<R>& P = PSH ? *reinterpret_cast<const Phys<R>*>(smem_raw + LY::ph_off) : Preg;
    if (PSH && threadIdx.x == 0) *reinterpret_cast<Phys<R>*>(smem_raw + LY::ph_off) = Phys<R>(C);
    const bool sponge = C.sponge != 0, iwall0 = B.wall[0] >= 0, iwall1 = B.wall[1] >= 0;
    const StatePtrs SP = A.p[t.blk];
    const int ng = B.ng, Nk = B.N[2];
    // cell and component offsets fit 32 bits (checked at case creation): one base pointer
    // per cell, 32-bit offsets per component
    const int planei = (int)B.plane, nc = (int)B.ncell;
    const R* MB = metbase<R>(B);
    const int tid = threadIdx.x;
    const int ihi = ng + B.n[0];
    // the tile's own extents (a block's last tiles may be smaller than its shape): every item
    // of the flat loops below is one that counts
    const int TJ = t.tj, TK = t.tk, PK = TK + 4, GK = TK + 2;
    const int ncol = TJ * TK, npr = (TJ + 4) * PK, ngr = (TJ + 2) * GK, nfj = (TJ + 1) * TK, nf = nfj + TJ * (TK + 1);
    // c / GK for record indices (c * GK < 2^20)
    const int gk_mul = (1 << 20) / GK + 1;
    const bool column = tid < ncol;                // this thread owns a tile column
    const int tj = tid / TK, tk = tid - tj * TK;
    const int col_pc = (tj + 2) * PK + (tk + 2), col_gc = (tj + 1) * GK + (tk + 1);
    // j/k faces, shared out so that every warp has about two faces' work per thread: the warps
    // without columns (no i-face flux of their own) come first, once, or twice in the FP64 form of
    // the upwind schemes, whose i-face flux is as long as two rounds of j/k faces
    constexpr int XTRA = NTH > CAP ? NTH - CAP : 0;
    constexpr int XROUNDS = sizeof(R) == 8 && SCHEME != WM_SCHEME_KEP ? 2 : 1;
    // FP64: the warps from thread gw on hold no gradient record; the copies and prefetches are
    // theirs, or of the warps without columns (float form), which have less to do than the others
    const int gw = (ngr + 31) & ~31;
    const int aux = FUSE ? gw : (XTRA ? CAP : 0);
    const int sgs_model = o.sgs;
    const int i0 = t.i0, i1 = t.i1;

    // ---- index tables
    {
        for (int c = tid; c < npr; c += NTH) {
            const int jj = c / PK;
            pt[c] = (t.j0 - 2 + jj) * Nk + t.k0 - 2 + c - jj * PK;
        }
        for (int c = tid; c < ncol; c += NTH) {
            const int jj = c / TK;
            ct[c] = (t.j0 + jj) * Nk + t.k0 + c - jj * TK;
        }
        const int jhi = ng + B.n[1], khi = ng + B.n[2];
        for (int f = tid; f < nf; f += NTH) {
            const bool kf = f >= nfj;
            const int w = kf ? TK + 1 : TK, g = kf ? f - nfj : f;
            const int row = g / w, col = g - row * w;
            int x = row | (col << 8) | (kf ? FT_K : 0);
            const int at = kf ? t.k0 + col : t.j0 + row, lo = kf ? 4 : 2;
            if (at == ng && B.wall[lo] >= 0) x |= FT_WLO;
            else if (at == (kf ? khi : jhi) && B.wall[lo + 1] >= 0) x |= FT_WHI;
            ft[f] = x;
        }
        if constexpr (EXT) {
            const R* src = ktab_of<R>(B) + 2 * (t.k0 - 1);
            for (int c = tid; c < 2 * (TK + 2); c += NTH) kt[c] = src[c];
        }
    }

    using GV = std::conditional_t<LY::GV == 1, R, std::conditional_t<LY::GV == 2, double2, float4>>;
    constexpr int NGV = NGS / LY::GV;
    // ring slot of plane ip + d; `ring` is the slot of the march's plane, stepped with it
    constexpr int SLOT = PR_N * PN, RING = LY::NSLOT * SLOT;
    int ring = 0;
    auto slot = [&](int d) {
        int s = ring + d * SLOT;
        if (d < 0 && s < 0) s += RING;
        if (d > 0 && s >= RING) s -= RING;
        return pr + s;
    };
    // ---- float form: conservative values of plane ip on the tile + 2-cell halo -> staging buffer
    // (async), by the threads from `first` on
    auto stage_plane = [&](int ip, int first) {
        for (int c = tid - first; c < npr; c += NTH - first) {
            const double* src = SP.q_in + (ip * planei + pt[c]);
#pragma unroll
            for (int v = 0; v < 5; ++v) cp_async8(qs + v * PN + c, src + v * nc);
        }
    };
    // ---- (EXT) the rows of metrics of plane ir
    auto stage_rows = [&](int ir, int first) {
        if constexpr (EXT) {
            constexpr int E16 = 16 / (int)sizeof(R);
            const R* src = rows_of<R>(B) + ((long long)ir * B.N[1] + t.j0 - 1) * RT_N;
            R* dst = rt + (ir & 1) * LY::RN * RT_N;
            for (int c = (tid - first) * E16; c < (TJ + 3) * RT_N; c += (NTH - first) * E16) cp_async16(dst + c, src + c);
        }
    };
    // ---- conservative values -> primitive record c of the plane d ahead of the march's
    auto convert = [&](int d, int c, const double q[5]) {
        R* dst = slot(d) + c;
        R rec[PR_N];
        cons_to_rec(q, P, rec);
#pragma unroll
        for (int v = 0; v < PR_N; ++v) dst[v * PN] = rec[v];
    };
    auto convert_staged = [&](int d) {
        for (int c = tid; c < npr; c += NTH) {
            double q[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) q[v] = qs[v * PN + c];
            convert(d, c, q);
        }
    };

    // ---- gradient record c of the march's plane ip on the tile + 1-cell halo
    auto grad_cell = [&](int ip, int c) {
        const R* Pm = slot(-1);
        const R* P0 = slot(0);
        const R* Pp = slot(1);
        const int jj = (c * gk_mul) >> 20, kk = c - jj * GK, pc = (jj + 1) * PK + kk + 1;
        const int pv[4] = {PR_U, PR_V, PR_W, PR_T};
        // FP64: the offset computed (a table look-up would delay the first load); float, bound by its
        // instructions: from the table
        const R* m = MB + (ip * planei + (FUSE ? (t.j0 - 1 + jj) * Nk + t.k0 - 1 + kk : pt[pc]));
        // a quarter of 1/V: the face values below are sums of two cells, twice the face
        // averages (scaling by two is exact, so the products and sums are the averages'
        // bit for bit, doubled), and the record holds half the gradient (faces average two
        // records by adding them); the SGS models are homogeneous of degree one in the
        // gradient and the Ducros sensor of degree zero, so they take the half gradient
        const R qivol = R(0.25) * __ldg(m + WM_MET_IVOL * nc);
        const R delta = sgs_model != WM_SGS_NONE ? __ldg(m + WM_MET_DELTA * nc) : R(0);
        R acc[12];
        if constexpr (EXT) {
            const R* row = rt + (ip & 1) * LY::RN * RT_N + jj * RT_N;
            const R Six = row[RT_SI], Siy = row[RT_SI + 1], Hix = row[RT_HI], Hiy = row[RT_HI + 1];
            const R Sjx = row[RT_SJ], Sjy = row[RT_SJ + 1], Hjx = row[RT_N + RT_SJ], Hjy = row[RT_N + RT_SJ + 1];
            const R Skz = row[RT_SK], qxy = qivol * kt[2 * kk];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const R c0 = P0[pv[a] * PN + pc];
                const R li = Pm[pv[a] * PN + pc] + c0, hi = c0 + Pp[pv[a] * PN + pc];
                const R lj = P0[pv[a] * PN + pc - PK] + c0, hj = c0 + P0[pv[a] * PN + pc + PK];
                const R lk = P0[pv[a] * PN + pc - 1] + c0, hk = c0 + P0[pv[a] * PN + pc + 1];
                acc[3 * a] = (hi * Hix - li * Six) + (hj * Hjx - lj * Sjx);
                acc[3 * a + 1] = (hi * Hiy - li * Siy) + (hj * Hjy - lj * Sjy);
                acc[3 * a + 2] = hk * Skz - lk * Skz;
            }
#pragma unroll
            for (int q = 0; q < 12; ++q) acc[q] *= q % 3 == 2 ? qivol : qxy;
        } else {
            const R* mi = m + planei;
            const R* mj = m + Nk;
            const R* mk = m + 1;
            const R Six = __ldg(m + WM_MET_SIX * nc), Siy = __ldg(m + WM_MET_SIY * nc), Siz = __ldg(m + WM_MET_SIZ * nc);
            const R Hix = __ldg(mi + WM_MET_SIX * nc), Hiy = __ldg(mi + WM_MET_SIY * nc), Hiz = __ldg(mi + WM_MET_SIZ * nc);
            const R Sjx = __ldg(m + WM_MET_SJX * nc), Sjy = __ldg(m + WM_MET_SJY * nc), Sjz = __ldg(m + WM_MET_SJZ * nc);
            const R Hjx = __ldg(mj + WM_MET_SJX * nc), Hjy = __ldg(mj + WM_MET_SJY * nc), Hjz = __ldg(mj + WM_MET_SJZ * nc);
            const R Skx = __ldg(m + WM_MET_SKX * nc), Sky = __ldg(m + WM_MET_SKY * nc), Skz = __ldg(m + WM_MET_SKZ * nc);
            const R Hkx = __ldg(mk + WM_MET_SKX * nc), Hky = __ldg(mk + WM_MET_SKY * nc), Hkz = __ldg(mk + WM_MET_SKZ * nc);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const R c0 = P0[pv[a] * PN + pc];
                const R li = Pm[pv[a] * PN + pc] + c0, hi = c0 + Pp[pv[a] * PN + pc];
                const R lj = P0[pv[a] * PN + pc - PK] + c0, hj = c0 + P0[pv[a] * PN + pc + PK];
                const R lk = P0[pv[a] * PN + pc - 1] + c0, hk = c0 + P0[pv[a] * PN + pc + 1];
                acc[3 * a] = ((hi * Hix - li * Six) + (hj * Hjx - lj * Sjx)) + (hk * Hkx - lk * Skx);
                acc[3 * a + 1] = ((hi * Hiy - li * Siy) + (hj * Hjy - lj * Sjy)) + (hk * Hky - lk * Sky);
                acc[3 * a + 2] = ((hi * Hiz - li * Siz) + (hj * Hjz - lj * Sjz)) + (hk * Hkz - lk * Skz);
            }
#pragma unroll
            for (int q = 0; q < 12; ++q) acc[q] *= qivol;
        }
        const R T = P0[PR_T * PN + pc];
        const R muh = R(0.5) * sutherland(T, P);              // half the molecular viscosity
        R muth = R(0);                                        // half the eddy viscosity
        if (sgs_model != WM_SGS_NONE) {
            const R rho = P0[PR_RHO * PN + pc];
            muth = rho * sgs_nut(sgs_model, acc, delta, P.sgs_c);
        }
        const R mu = muh + muth, kc = P.cp * (muh * P.inv_Pr + muth * P.inv_Prt);
        R th = R(0);
        if constexpr (SCHEME == WM_SCHEME_HYBRID) th = ducros(acc);
        if constexpr (LY::GV == 1) {
#pragma unroll
            for (int q = 0; q < 12; ++q) gs[q * GN + c] = acc[q];
            gs[GS_MU * GN + c] = mu;
            gs[GS_K * GN + c] = kc;
            if constexpr (NGS > 14) gs[GS_TH * GN + c] = th;
        } else {
            R rec[16] = {acc[0], acc[1], acc[2], acc[3], acc[4], acc[5], acc[6], acc[7], acc[8], acc[9], acc[10], acc[11], mu, kc, th, R(0)};
            GV* g = reinterpret_cast<GV*>(gs) + c;
#pragma unroll
            for (int x = 0; x < NGV; ++x) {
                GV y;
#pragma unroll
                for (int w = 0; w < LY::GV; ++w) reinterpret_cast<R*>(&y)[w] = rec[LY::GV * x + w];
                g[x * GN] = y;
            }
        }
    };

    // wall-model flux override of a wall-modelled face (axis, side) at its position (a, b); EXT, i and j
    // faces: over the factor per k that their flux differences are multiplied by (kk: k position in kt)
    auto wall_flux = [&](int face, int a, int b, int kk, R F[5]) {
        const WallDev& W = A.walls[B.wall[face]];
        const long long f = (long long)a * W.nt2 + b;
        const long long nw = (long long)W.nt1 * W.nt2;
        const double scale = EXT && face < 4 ? 1.0 / double(kt[2 * kk]) : 1.0;
#pragma unroll
        for (int v = 0; v < 5; ++v) F[v] = R(EXT ? W.F[v * nw + f] * scale : W.F[v * nw + f]);
    };

    // ---- i-face flux between planes ip-1 and ip for this thread's column
    // float form: gradient record of plane ip-1 at this column
    GV gsp[FUSE ? 1 : NGV];
    auto save_gs = [&]() {
        if constexpr (!FUSE) {
            if (!column) return;
#pragma unroll
            for (int v = 0; v < NGV; ++v) gsp[v] = reinterpret_cast<const GV*>(gs)[v * GN + col_gc];
        }
    };
    // record c + off of the march's plane: its components or, GV > 1, groups of them
    auto grad_at = [&](int c, int off) {
        const GV* g = reinterpret_cast<const GV*>(gs) + c;
        return [g, off](int v) { return g[v * GN + off]; };
    };
    auto iface_flux = [&](int ip, R F[5]) {
        if ((ip == ng && iwall0) || (ip == ihi && iwall1)) {
            wall_flux(ip == ng ? 0 : 1, t.j0 + tj - ng, t.k0 + tk - ng, tk + 1, F);
            return;
        }
        // FP64: plane ip-2's record from the column's own copy
        const R* L2 = FUSE ? hp : slot(-2) + col_pc;
        constexpr int S2 = FUSE ? CAP : PN;
        const R* L = slot(-1) + col_pc;
        const R* Rr = slot(0) + col_pc;
        const R* R2 = slot(1) + col_pc;
        const GV* gl = LY::PING ? reinterpret_cast<const GV*>(gs0 + (gs == gs0 ? NGS * GN : 0)) + col_gc
                                : reinterpret_cast<const GV*>(hg);
        auto gL = [&](int v) {
            if constexpr (FUSE) return gl[v * (LY::PING ? GN : CAP)];
            else return gsp[v];
        };
        auto gR = grad_at(col_gc, 0);
        if constexpr (EXT) {
            const R* row = rt + (ip & 1) * LY::RN * RT_N + (tj + 1) * RT_N;
            face_flux<FACE_XY, R, SCHEME>(o, P, L2, S2, L, Rr, R2, PN, gL, gR, row[RT_SI], row[RT_SI + 1], R(0), row[RT_EI],
                                          row[RT_EI + 1], R(0), row[RT_IDI], F);
        } else {
            const R* m = MB + (ip * planei + (FUSE ? (t.j0 + tj) * Nk + t.k0 + tk : ct[tid]));
            const R Sx = __ldg(m + WM_MET_SIX * nc), Sy = __ldg(m + WM_MET_SIY * nc), Sz = __ldg(m + WM_MET_SIZ * nc);
            const R e0 = __ldg(m + WM_MET_EIX * nc), e1 = __ldg(m + WM_MET_EIY * nc), e2 = __ldg(m + WM_MET_EIZ * nc);
            const R id = __ldg(m + WM_MET_IDI * nc);
            face_flux<FACE_ANY, R, SCHEME>(o, P, L2, S2, L, Rr, R2, PN, gL, gR, Sx, Sy, Sz, e0, e1, e2, id, F);
        }
    };

    // ---- one j- or k-face flux of plane ip (entry f of the face table) into shared memory
    auto jk_face = [&](int ip, int f) {
        const int at = ft[f], row = at & 255, col = (at >> 8) & 255;
        R F[5];
        const bool kf = at & FT_K;
        if (at & (FT_WLO | FT_WHI)) {
            // j face: (i, k) along the wall; k face: (i, j)
            wall_flux((kf ? 4 : 2) + (at & FT_WHI ? 1 : 0), ip - ng, kf ? t.j0 - ng + row : t.k0 - ng + col, col + 1, F);
        } else {
            const int pc = (row + 2) * PK + col + 2;
            const R* p = slot(0) + pc;
            const int gc = (row + 1) * GK + col + 1;
            auto gR = grad_at(gc, 0);
            if constexpr (EXT) {
                const R* mr = rt + (ip & 1) * LY::RN * RT_N + (row + 1) * RT_N;
                if (kf) {
                    face_flux<FACE_Z, R, SCHEME>(o, P, p - 2, PN, p - 1, p, p + 1, PN, grad_at(gc, -1), gR,
                                                 R(0), R(0), mr[RT_SK], R(0), R(0), R(1), kt[2 * col + 3], F);
                } else {
                    face_flux<FACE_XY, R, SCHEME>(o, P, p - 2 * PK, PN, p - PK, p, p + PK, PN,
                                                  grad_at(gc, -GK), gR, mr[RT_SJ], mr[RT_SJ + 1],
                                                  R(0), mr[RT_EJ], mr[RT_EJ + 1], R(0), mr[RT_IDJ], F);
                }
            } else {
                const int ps = kf ? 1 : PK, gp = kf ? 1 : GK;                // step to the next cell across the face
                const R* m = MB + (ip * planei + (FUSE ? (t.j0 + row) * Nk + t.k0 + col : pt[pc])) + (kf ? WM_MET_SKX : WM_MET_SJX) * nc;
                const R Sx = __ldg(m), Sy = __ldg(m + nc), Sz = __ldg(m + 2 * nc);
                m += (kf ? WM_MET_EKX - WM_MET_SKX : WM_MET_EJX - WM_MET_SJX) * nc;
                const R e0 = __ldg(m), e1 = __ldg(m + nc), e2 = __ldg(m + 2 * nc), id = __ldg(m + 3 * nc);
                face_flux<FACE_ANY, R, SCHEME>(o, P, p - 2 * ps, PN, p - ps, p, p + ps, PN,
                                               grad_at(gc, -gp), gR, Sx, Sy, Sz, e0, e1, e2, id, F);
            }
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) ff[v * FN + f] = F[v];
    };

    // ---- cache-line prefetch of what the next plane reads from global memory.  General grids: the
    // metrics of plane ip+1 and the i-face areas of plane ip+2; extruded: 1/V and the filter width.
    // Each warp from `first` on takes components, its lanes the lines of the tile's rows (FP64, general:
    // with the halo of the gradient records; else the halo's lines are left to the CTAs that own
    // them, as all march in step: half the lines to ask for, box 192 x 112 x 96 float 1827 -> 1671 us
    // a pass, but FP64, which has the L1 for fewer of them, 2928 -> 3128).
    constexpr int PH = sizeof(R) == 8 && !EXT ? 1 : 0;
    const int pf_nl = ((TK + 3 * PH) * (int)sizeof(R) + 127) / 128 + 1, pf_n = (TJ + 3 * PH) * pf_nl;
    const int pf_mul = 65536 / pf_nl + 1;                      // x / pf_nl for the x below
    auto prefetch_next = [&](int ip, int first) {
        // S (0..8), delta, 1/V, e/idist (13..26) of plane ip+1 (23), then S_i of plane ip+2 (planes up to
        // ihi + 1 exist: ip < i1 here)
        constexpr int NPF = EXT ? 2 : PH ? 26 : 23;
        for (int comp = (tid - first) >> 5; comp < NPF; comp += (NTH - first) >> 5) {
            const int cc = EXT ? WM_MET_DELTA + comp : comp < 9 ? comp : comp < 23 ? comp + 4 : comp - 23;
            const R* base = MB + cc * nc + (ip + (comp < 23 ? 1 : 2)) * planei + (t.j0 - PH) * Nk + t.k0 - PH;
            for (int x = tid & 31; x < pf_n; x += 32) {
                const int row = (x * pf_mul) >> 16, line = x - row * pf_nl;
                const R* rowp = base + row * Nk;
                const uintptr_t a = (reinterpret_cast<uintptr_t>(rowp) & ~uintptr_t(127)) + 128u * line;
                if (a <= reinterpret_cast<uintptr_t>(rowp + TK - 1 + 3 * PH)) prefetch_l1(reinterpret_cast<const void*>(a));
            }
        }
    };
    auto prefetch_q0 = [&](int ip, int first) {                // tile columns of the step-start state
        const int nl = (TK + 30) >> 4, mul = (1 << 16) / nl + 1;   // lines of a row, at most
        const double* base = SP.q0 + ip * planei + t.j0 * Nk + t.k0;
        for (int x = tid - first; x < TJ * nl; x += NTH - first) {
            const int r = (x * mul) >> 16, k = min(16 * (x - r * nl), TK - 1);
#pragma unroll
            for (int v = 0; v < 5; ++v) prefetch_l2(base + v * nc + r * Nk + k);
        }
    };

    const double dt = A.stage ? *A.dt[B.case_id] : 0.0;
    // constant mass flux (stage 3): sum of rho u_dir V over the case, exact in three bins of fixed
    // exponent (cmf_bins, capi.cu), so that its bits depend neither on the tiles' shape nor on the order
    // in which threads, CTAs and launches add.  The sums wait in shared memory (in registers they cost some
    // 50 B of spills): a column's in the float form, a warp's in FP64, which has no room for the columns'
    // (float form with a warp's: 30 shuffles for every warp and plane, channel 256 x 128 x 128 1188 us a step
    // against 1158).
    const bool cmf_on = A.stage == 3 && A.cmf_sum != nullptr && C.cmf_dir >= 0;
    const int cmf_dir = C.cmf_dir;
    double* cmf_bin = red + 3 * NW;
    if (cmf_on && tid < 3 * NW + 3) red[tid] = tid < 3 * NW ? 0.0 : C.cmf_bin[tid - 3 * NW];
    double* cmf_col = reinterpret_cast<double*>(smem_raw + LY::cs_off) + threadIdx.x;
    if (!FUSE && cmf_on && tid < CAP)
#pragma unroll
        for (int m = 0; m < 3; ++m) cmf_col[m * CAP] = 0.0;

    // ---- RK epilogue of one cell: its operands, loaded ahead of use (from issue to use some 2000
    // cycles under load), then r = -(div F)/V (+ source) from the flux divergence dv (times -1,
    // not yet divided by V) and the stage update
    struct Epi {
        double q[5], q0[5], vol;
        R ivol;
    };
    auto epi_load = [&](int io, int c, Epi& e) {
        const int idx = io * planei + ct[c];
        e.ivol = __ldg(MB + WM_MET_IVOL * nc + idx);
#pragma unroll
        for (int v = 0; v < 5; ++v) e.q[v] = ld_state(SP.q_in + v * nc + idx);
        if (A.stage >= 2) {
#pragma unroll
            for (int v = 0; v < 5; ++v) e.q0[v] = ld_state(SP.q0 + v * nc + idx);
        }
        if (cmf_on) e.vol = __ldg(B.met + WM_MET_VOL * nc + idx);
    };
    // returns rho u_dir V of stage 3 with constant mass flux, else 0
    auto output = [&](int io, int c, const Epi& e, const R dv[5]) -> double {
        const int jk = ct[c], idx = io * planei + jk;
        R r[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) r[v] = dv[v] * e.ivol;
        double rq[5];
        if (sponge) {
            // -sigma(x) (q - spanwise mean), wmles/smooth_ramp.py:212-221
            const double xl = __ldg(B.met + WM_MET_XCX * nc + idx) * C.sp_invL;
            const double eta = fmin(fmax((xl - C.sp_xs) * C.sp_inv_dx, 0.0), 1.0);
            const double sig = C.sp_sigma0 * (eta * eta * eta * (10.0 + eta * (-15.0 + 6.0 * eta)));
            const long long mi = (long long)io * B.N[1] + jk / Nk;
            const long long mn = (long long)B.N[0] * B.N[1];
#pragma unroll
            for (int v = 0; v < 5; ++v) rq[v] = double(r[v]) - sig * (e.q[v] - SP.spmean[v * mn + mi]);
        } else {
#pragma unroll
            for (int v = 0; v < 5; ++v) rq[v] = double(r[v]);
        }
        double* out = SP.q_out + idx;
        if (A.stage == 0) {
#pragma unroll
            for (int v = 0; v < 5; ++v) out[v * nc] = rq[v];
        } else if (A.stage == 1) {
#pragma unroll
            for (int v = 0; v < 5; ++v) out[v * nc] = e.q[v] + dt * rq[v];
        } else if (A.stage == 2) {
#pragma unroll
            for (int v = 0; v < 5; ++v) out[v * nc] = 0.75 * e.q0[v] + 0.25 * (e.q[v] + dt * rq[v]);
        } else {
            double qn[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) {
                qn[v] = (1.0 / 3.0) * e.q0[v] + (2.0 / 3.0) * (e.q[v] + dt * rq[v]);
                out[v * nc] = qn[v];
            }
            // rounded by itself: contracted with a bin's constant, it would depend on the instance
            if (cmf_on) return __dmul_rn(cmf_dir == 0 ? qn[1] : cmf_dir == 1 ? qn[2] : qn[3], e.vol);
        }
        return 0.0;
    };
    // a value's part in bin m; x: what it leaves for the next
    auto cmf_part = [&](int m, double& x) {
        const double c = cmf_bin[m], h = __dsub_rn(__dadd_rn(x, c), c);
        x = __dsub_rn(x, h);
        return h;
    };
    auto cmf_warp_sum = [&](int m, double h) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) h = __dadd_rn(h, __shfl_down_sync(0xffffffffu, h, off));
        if ((tid & 31) == 0) red[3 * (tid >> 5) + m] = __dadd_rn(red[3 * (tid >> 5) + m], h);
    };
    // FP64: a warp's cells of a plane (up to two a lane)
    auto cmf_add = [&](double x0, double x1) {
        constexpr int UNR = SCHEME == WM_SCHEME_HYBRID ? 3 : 1;      // fewest spills
#pragma unroll UNR
        for (int m = 0; m < 3; ++m) {
            const double h = cmf_part(m, x0);
            cmf_warp_sum(m, __dadd_rn(h, cmf_part(m, x1)));
        }
    };
    // the segment's sums into the case's, at its end
    auto cmf_flush = [&]() {
        if (!cmf_on) return;
        if constexpr (!FUSE)
            for (int m = 0; m < 3; ++m) cmf_warp_sum(m, tid < CAP ? cmf_col[m * CAP] : 0.0);
        __syncthreads();
        if (tid < 3) {
            double sum = 0.0;
            for (int w = 0; w < NW; ++w) sum = __dadd_rn(sum, red[3 * w + tid]);
            atomicAdd(A.cmf_sum + 3 * B.case_id + tid, sum);
        }
    };
    // ---- prologue: primitives of planes i0-2, i0-1 (FP64: i0) straight from global memory, the
    // next plane staged
    __syncthreads();                         // index tables
    constexpr int PRE = FUSE ? 3 : 2;
    if constexpr (!FUSE) stage_plane(i0 - 2 + PRE, 0);
    stage_rows(i0 - 1, 0);
    for (int c = tid; c < npr; c += NTH) {
        const double* src = SP.q_in + ((i0 - 2) * planei + pt[c]);
        double q[PRE][5];
#pragma unroll
        for (int d = 0; d < PRE; ++d)
#pragma unroll
            for (int v = 0; v < 5; ++v) q[d][v] = ld_state(src + d * planei + v * nc);
#pragma unroll
        for (int d = 0; d < PRE; ++d) {
            R rec[PR_N];
            cons_to_rec(q[d], P, rec);
#pragma unroll
            for (int v = 0; v < PR_N; ++v) pr[d * SLOT + v * PN + c] = rec[v];
        }
    }
    cp_async_wait_all();
    __syncthreads();

    // ---- march: gradient records of plane ip, faces of plane ip (from i0 on)
    auto next_plane = [&]() {
        ring = ring + SLOT == RING ? 0 : ring + SLOT;
        if constexpr (LY::PING) gs = gs == gs0 ? gs0 + NGS * GN : gs0;
    };
    auto faces = [&](int ip) {
        // in two rounds, the threads without columns take faces [0, 2 XTRA), the others the CAP after those
        static_assert(XROUNDS == 1 || FN <= NTH + XTRA, "the strides below leave out faces beyond the first rounds");
        if (ip < i0 || ip >= i1) return;
        const int f0 = tid < CAP ? tid + XROUNDS * XTRA : tid - CAP;
        const int step0 = tid < CAP || XROUNDS == 1 ? NTH + (XROUNDS - 1) * XTRA : XTRA;
#pragma unroll 1
        for (int f = f0, step = step0; f < nf; f += step) {
            jk_face(ip, f);
            if (XROUNDS == 2 && f >= XTRA) step = NTH + XTRA;
        }
    };
    if constexpr (FUSE) {
        // The warps that hold a gradient record, and the warps left over: those finish plane ip-2 for
        // up to two columns a thread, convert up to three cells of plane ip+2 and take the flux
        // differences of plane ip-1.  The values they need from global memory are loaded into
        // registers at the end of the face phase, where these warps wait for the column threads:
        // some 2000 cycles of latency under load, and no register held through a compute phase.
        constexpr int NCV = (PN + NTH - LY::GW - 1) / (NTH - LY::GW);
        const int ac = tid - gw, as = NTH - gw;
        const int tk_mul = (1 << 20) / TK + 1;                   // c / TK for column indices
        R Flo[5];
        Epi e[2];
        double cq[NCV][5];
        // Every value is set on every path: otherwise the compiler would have to keep the last ones
        // through the phases.
        auto load_aux = [&](int ip) {                            // for the gradient phase of plane ip + 1
            if (tid < gw) {
#pragma unroll
                for (int r = 0; r < NCV; ++r)
#pragma unroll
                    for (int v = 0; v < 5; ++v) cq[r][v] = 0.0;
#pragma unroll
                for (int r = 0; r < 2; ++r) e[r] = Epi{};
                return;
            }
#pragma unroll
            for (int r = 0; r < NCV; ++r) {
                const int c = ac + r * as;
                const bool ok = c < npr && ip + 3 <= i1 + 1;
                const double* src = SP.q_in + (ok ? (ip + 3) * planei + pt[c] : 0);
#pragma unroll
                for (int v = 0; v < 5; ++v) cq[r][v] = ok ? ld_state(src + v * nc) : 0.0;
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int c = ac + r * as;
                const bool ok = c < ncol && ip - 1 >= i0;
                const int idx = ok ? (ip - 1) * planei + ct[c] : 0;
                e[r].ivol = ok ? __ldg(MB + WM_MET_IVOL * nc + idx) : R(0);
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    e[r].q[v] = ok ? ld_state(SP.q_in + v * nc + idx) : 0.0;
                    e[r].q0[v] = ok && A.stage >= 2 ? ld_state(SP.q0 + v * nc + idx) : 0.0;
                }
                e[r].vol = ok && cmf_on ? __ldg(B.met + WM_MET_VOL * nc + idx) : 0.0;
            }
        };
        auto finish = [&](int io) {
            double x[2] = {0.0, 0.0};
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int c = ac + r * as;
                if (c >= ncol) break;
                R d[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) d[v] = fr[v * CAP + c];
                x[r] = output(io, c, e[r], d);
            }
            if (cmf_on) cmf_add(x[0], x[1]);
        };
        load_aux(i0 - 2);
#pragma unroll 1
        for (int ip = i0 - 1; ip <= i1; ++ip) {
            next_plane();
            if (tid < gw) {
                if (tid < ngr) grad_cell(ip, tid);
            } else {
                if (ip - 2 >= i0) finish(ip - 2);
                if (ip < i1) {
#pragma unroll
                    for (int r = 0; r < NCV; ++r)
                        if (ac + r * as < npr) convert(2, ac + r * as, cq[r]);
                }
                if (ip - 1 >= i0)
                    for (int c = ac; c < ncol; c += as) {
                        const int row = (c * tk_mul) >> 20;
                        const R* pj = ff + c;                                // row of the j faces
                        const R* pk = ff + nfj + c + row;                    // row of the k faces, one longer
                        const R rk = EXT ? kt[2 * (c - row * TK) + 2] : R(1);
#pragma unroll
                        for (int v = 0; v < 5; ++v)
                            fr[v * CAP + c] = (pj[v * FN] - pj[v * FN + TK]) * rk - (pk[v * FN + 1] - pk[v * FN]);
                    }
            }
            __syncthreads();
            if (!EXT && tid >= CAP && ip < i1) prefetch_next(ip, CAP);
            if (tid >= gw && ip < i1) {
                stage_rows(ip + 1, gw);
                if (EXT) prefetch_next(ip, gw);
                // the step-start state of the plane after the next epilogue's, from HBM
                if (A.stage >= 2) prefetch_q0(ip, gw);
            }
            if (column) {
                if (ip >= i0) {
                    R Fhi[5];
                    iface_flux(ip, Fhi);
                    if (ip > i0) {
                        const R rk = EXT ? kt[2 * tk + 2] : R(1);
#pragma unroll
                        for (int v = 0; v < 5; ++v) fr[v * CAP + tid] -= (Fhi[v] - Flo[v]) * rk;
                    }
#pragma unroll
                    for (int v = 0; v < 5; ++v) Flo[v] = Fhi[v];
                }
                // what the next plane's i face needs of this one's
                const R* L = slot(-1) + col_pc;
#pragma unroll
                for (int v = 0; v < LY::HP_N; ++v) hp[v * CAP] = L[v * PN];
                if constexpr (!LY::PING) {   // EXT: components one by one
#pragma unroll
                    for (int v = 0; v < NGS; ++v) hg[v * CAP] = gs[v * GN + col_gc];
                }
            }
            faces(ip);
            load_aux(ip);
            cp_async_wait_all();
            __syncthreads();
        }
        if (tid >= gw) finish(i1 - 1);               // the segment's last plane
        cmf_flush();
    } else {
        R Flo[5], dv[5];
        Epi e;                                       // operands of the next epilogue
#pragma unroll 1
        for (int ip = i0 - 1; ip <= i1; ++ip) {
            next_plane();
            R dFj[5], dFk[5];
            if (column && ip - 1 >= i0) {
                const R* pj = ff + tid;                              // row tj of the j faces
                const R* pk = ff + nfj + tid + tj;                   // row tj of the k faces, one longer
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    dFj[v] = pj[v * FN + TK] - pj[v * FN];
                    dFk[v] = pk[v * FN + 1] - pk[v * FN];
                }
            }
            if (ip >= i0) save_gs();
            convert_staged(1);
            __syncthreads();
            for (int c = tid; c < ngr; c += NTH) grad_cell(ip, c);
            __syncthreads();
            if (tid >= aux) {
                if (ip + 2 <= i1 + 1) stage_plane(ip + 2, aux);
                // the step-start state of the plane after the next epilogue's, from HBM
                if (A.stage >= 2 && ip < i1) prefetch_q0(ip, aux);
                if (ip < i1) {
                    stage_rows(ip + 1, aux);
                    prefetch_next(ip, aux);
                }
            }
            if (column && ip >= i0) {
                R Fhi[5];
                iface_flux(ip, Fhi);
                if (ip > i0) {
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        if constexpr (EXT) dv[v] = (-(Fhi[v] - Flo[v]) - dFj[v]) * kt[2 * tk + 2] - dFk[v];
                        else dv[v] = (-(Fhi[v] - Flo[v]) - dFj[v]) - dFk[v];
                    }
                }
#pragma unroll
                for (int v = 0; v < 5; ++v) Flo[v] = Fhi[v];
            }
            if (column && ip - 1 >= i0) epi_load(ip - 1, tid, e);
            faces(ip);
            if (column && ip - 1 >= i0) {
                double x = output(ip - 1, tid, e, dv);
                if (cmf_on)
#pragma unroll
                    for (int m = 0; m < 3; ++m) cmf_col[m * CAP] = __dadd_rn(cmf_col[m * CAP], cmf_part(m, x));
            }
            cp_async_wait_all();
            __syncthreads();
        }
        cmf_flush();
    }
}

template <typename R, int SCHEME, int CAP, bool EXT>
__global__ void __launch_bounds__(StageLayout<R, SCHEME, CAP, EXT>::NTH, StageLayout<R, SCHEME, CAP, EXT>::MIN_CTAS)
    stage_kernel(const __grid_constant__ StageArgs A, const StageOpts o) {
    using LY = StageLayout<R, SCHEME, CAP, EXT>;
    chain_wait();
    constexpr int NTH = LY::NTH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    // this CTA's segments: one tile, or a balanced range of tiles (consecutive column pieces)
    const int first = A.cta_first ? A.cta_first[blockIdx.x] : blockIdx.x;
    const int last = A.cta_first ? A.cta_first[blockIdx.x + 1] : blockIdx.x + 1;
#pragma unroll 1
    for (int ti = first; ti < last; ++ti) {
        stage_segment<R, SCHEME, CAP, EXT>(A, o, A.tiles[ti], smem_raw);
        __syncthreads();                 // shared memory is reused by the next segment
    }

    if (A.stage == 3 && A.cmf_sum != nullptr) {
        // every CTA of the stage's launches signals; the last one turns each case's sums into the shift
        // delta = target - sum(rho u V) / sum(V), wmles/solver.py:24-29
        __shared__ bool last_cta;
        if (tid < 3) __threadfence();
        __syncthreads();
        if (tid == 0) last_cta = atomicAdd(A.cmf_counter, 1u) == unsigned(A.cmf_ctas - 1);
        __syncthreads();
        if (last_cta) {
            __threadfence();
            for (int c = tid; c < A.ncases; c += NTH) {
                const CaseDev& Cc = A.cases[c];
                if (Cc.cmf_dir < 0) continue;
                double* sum = A.cmf_sum + 3 * c;
                const double hi = __ldcg(sum);
                // an infinite value leaves NaN in the lower bins
                const double tot = isfinite(hi) ? hi + (__ldcg(sum + 1) + __ldcg(sum + 2)) : hi;
                A.cmf_delta[c] = Cc.cmf_target - tot / Cc.cmf_volume;
#pragma unroll
                for (int m = 0; m < 3; ++m) sum[m] = 0.0;
            }
            if (tid == 0) *A.cmf_counter = 0u;
        }
    }
}

template <typename R, int SCHEME, int CAP, bool EXT>
static cudaError_t configure_one() {
    using LY = StageLayout<R, SCHEME, CAP, EXT>;
    static std::atomic<unsigned long long> done{0};     // per instantiation, one bit per device
    return once_per_device(done, [] {
        return cudaFuncSetAttribute(stage_kernel<R, SCHEME, CAP, EXT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)LY::bytes);
    });
}

template <typename R, int SCHEME, int CAP, bool EXT>
static cudaError_t launch_one(const StageArgs& A, const StageOpts& o, cudaStream_t s) {
    using LY = StageLayout<R, SCHEME, CAP, EXT>;
    cudaError_t e = configure_one<R, SCHEME, CAP, EXT>();
    if (e != cudaSuccess) return e;
    return launch_chained(stage_kernel<R, SCHEME, CAP, EXT>, A.nctas, LY::NTH, LY::bytes, s, A, o);
}

template <typename R, int SCHEME, int CAP, bool EXT>
static int occupancy_one() {
    using LY = StageLayout<R, SCHEME, CAP, EXT>;
    if (configure_one<R, SCHEME, CAP, EXT>() != cudaSuccess) return 1;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, stage_kernel<R, SCHEME, CAP, EXT>, LY::NTH, LY::bytes) !=
        cudaSuccess)
        return 1;
    return n;
}

// kernel variants: 256 columns (FP64; float form: two CTAs per SM), 512 columns (float form)
template <typename R, int SCHEME>
static cudaError_t launch_cap(const StageArgs& A, const StageOpts& o, cudaStream_t s) {
    if constexpr (sizeof(R) == 4)
        if (stage_cap(o) == 512)
            return A.ext ? launch_one<R, SCHEME, 512, true>(A, o, s) : launch_one<R, SCHEME, 512, false>(A, o, s);
    return A.ext ? launch_one<R, SCHEME, 256, true>(A, o, s) : launch_one<R, SCHEME, 256, false>(A, o, s);
}

template <typename R, int SCHEME>
static int occupancy_cap(const StageOpts& o) {
    if constexpr (sizeof(R) == 4)
        if (stage_cap(o) == 512) return occupancy_one<R, SCHEME, 512, false>();
    return occupancy_one<R, SCHEME, 256, false>();
}

int stage_ctas_per_sm(const StageOpts& o) {
    if (o.precision == WM_PREC_MIXED) {
        switch (o.scheme) {
            case WM_SCHEME_KEP: return occupancy_cap<float, WM_SCHEME_KEP>(o);
            case WM_SCHEME_MUSCL: return occupancy_cap<float, WM_SCHEME_MUSCL>(o);
            default: return occupancy_cap<float, WM_SCHEME_HYBRID>(o);
        }
    }
    switch (o.scheme) {
        case WM_SCHEME_KEP: return occupancy_cap<double, WM_SCHEME_KEP>(o);
        case WM_SCHEME_MUSCL: return occupancy_cap<double, WM_SCHEME_MUSCL>(o);
        default: return occupancy_cap<double, WM_SCHEME_HYBRID>(o);
    }
}

cudaError_t launch_stage(const StageArgs& A, const StageOpts& o, cudaStream_t s) {
    if (o.precision == WM_PREC_MIXED) {
        switch (o.scheme) {
            case WM_SCHEME_KEP: return launch_cap<float, WM_SCHEME_KEP>(A, o, s);
            case WM_SCHEME_MUSCL: return launch_cap<float, WM_SCHEME_MUSCL>(A, o, s);
            default: return launch_cap<float, WM_SCHEME_HYBRID>(A, o, s);
        }
    }
    switch (o.scheme) {
        case WM_SCHEME_KEP: return launch_cap<double, WM_SCHEME_KEP>(A, o, s);
        case WM_SCHEME_MUSCL: return launch_cap<double, WM_SCHEME_MUSCL>(A, o, s);
        default: return launch_cap<double, WM_SCHEME_HYBRID>(A, o, s);
    }
}

int stage_cap(const StageOpts& o) { return o.precision == WM_PREC_MIXED && (o.tile < 0 || o.tile == 3) ? 512 : 256; }

double split_planes(long long cols, int n0, int slots, int* chunk, int* tail) {
    if (chunk) *chunk = n0;
    if (tail) *tail = 0;
    double best = 1e300;
    for (int ic = 1, m; ic <= n0; ic = m > 1 ? (n0 + m - 2) / (m - 1) : n0 + 1) {    // the shortest for each number of chunks
        m = (n0 + ic - 1) / ic;
        const double cost = double((cols * m + slots - 1) / slots) * (ic + SEG_PLANES);
        if (cost < best - 1e-9) { best = cost; if (chunk) *chunk = ic; }
    }
    const long long q = slots / cols, r = slots - q * cols;
    if (q < 1 || r < 1) return best;
    const long long m = (cols + r - 1) / r;            // tail segments of the busiest tail CTA
    for (int x = 8; x < n0 / 2 && m * (x + SEG_PLANES) < best; ++x) {      // tail segments of at least 8 planes
        const double cost = std::max((n0 - x + q - 1) / q + SEG_PLANES, m * (x + SEG_PLANES));
        if (cost < best - 1e-9) { best = cost; if (tail) *tail = x; }
    }
    return best;
}

// Tile shape of `count` blocks of n cells that may use `slots` resident CTAs together.  tile >= 0: the requested
// shape.  Else the cheapest split of its j-k plane into equal tiles within the kernel's capacities:
// estimated time of the launch = planes the busiest CTA marches (split_planes) x time of a
// plane.  That time has a part that does not shrink with the tile, one thread's chain of work and
// the barriers, and one in proportion to its items, weighted by their instructions; narrow rows
// cost some more (whole 128-byte lines).  Fitted to stage times (us per launch) on the channel
// 256 x 128 x 128: FP64 8x32 663, 16x16 712, 6x32 749, 4x32 1010; float 16x32 371, 12x32 413,
// 6x64 415, 8x32 512; on the C-grid (40 cells along k): FP64 6x40 554, 12x20 571, 5x40 600,
// 16x16 724, 8x32 944; float 11x40 261, 8x40 265, 16x22 278, 16x32 339.  Looked at on 120 batches of 3 to 96
// channels of 8^3 to 192 x 96 x 96, both forms and kinds: 0.74-1.01 of the fixed shape's time where both were timed.
void tile_shape(const StageOpts& o, const int n[3], int count, int slots, int* tj, int* tk) {
    switch (o.tile) {
        case 0: *tj = 8; *tk = 32; return;
        case 1: *tj = 16; *tk = 16; return;
        case 2: *tj = 4; *tk = 32; return;
        case 3: *tj = 16; *tk = 32; return;
        default: break;
    }
    const int cap = stage_cap(o);
    const StageCaps L = stage_caps(cap);
    auto items = [](int a, int b) {
        return 730.0 * (a + 2) * (b + 2) + 350.0 * ((a + 1) * b + a * (b + 1) + a * b) + 100.0 * (a + 4) * (b + 4) +
               110.0 * a * b;
    };
    const double full = items(cap / 32, 32), fixed = cap == 512 ? 0.4 : 0.55;
    if (slots < 1) slots = 1;
    double best = 1e300;
    *tj = 1; *tk = std::min(n[2], 32);
    for (int mk = 1; mk <= n[2]; ++mk) {
        const int k = (n[2] + mk - 1) / mk;
        if ((n[2] + k - 1) / k != mk) continue;              // the same width as a smaller mk
        for (int mj = 1; mj <= n[1]; ++mj) {
            const int j = (n[1] + mj - 1) / mj;
            if ((n[1] + j - 1) / j != mj) continue;
            if (j * k > cap || (j + 4) * (k + 4) > L.pn || (j + 2) * (k + 2) > L.gn ||
                (j + 1) * k + j * (k + 1) > L.fn || j + 3 > L.rows || k + 2 > L.kn)
                continue;
            const double plane = fixed * full + (1.0 - fixed) * items(j, k) * (1.0 + 4.0 / k);
            const double cost = split_planes((long long)count * mj * mk, n[0], slots, nullptr, nullptr) * plane;
            if (cost < best * (1.0 - 1e-9)) { best = cost; *tj = j; *tk = k; }
        }
    }
}

}  // namespace wm
