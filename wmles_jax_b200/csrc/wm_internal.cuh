// Device-side descriptors shared by the kernels of libwmles_cuda.so.
//
// Every launch works on a *view*: a set of one or more independent cases whose blocks,
// per-case constants, wall faces and stage tiles are concatenated into device tables.
// Blocks carry a global index (into the view's block table) and their case's index.
#pragma once
#include <atomic>
#include <cstdint>
#include <cuda_runtime.h>
#include "../../include/wmles_cuda.h"

namespace wm {

// runs `set` (a kernel attribute set-up, which holds for the current device only) once per
// device: `done` keeps one bit per device ordinal below 64 (others set it on every call); two
// threads racing on a device both set the same value
template <class F>
inline cudaError_t once_per_device(std::atomic<unsigned long long>& done, F set) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    e = set();
    if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_acq_rel);
    return e;
}

// A step is a chain of some seven dependent launches, and on a small case the gaps between them are a good
// part of it.  Its kernels are launched with programmatic stream serialisation: the next one's CTAs come up as
// the last CTAs of this one leave, instead of after its memory is flushed and the launch is processed.
// chain_wait() is every thread's first statement in such a kernel: it returns when the kernels before it in
// the stream have completed and their writes are visible.  As no CTA goes on (or returns) before that,
// completion stays in stream order along the chain.  (Letting the next kernel up early, while this one runs,
// was slower: channel 256 x 128 x 128 FP64 6.65 ms for three steps against 6.46, 6.51 without the chain.)
__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }

template <class... P, class... T>
inline cudaError_t launch_chained(void (*kernel)(P...), unsigned ctas, unsigned threads, size_t smem, cudaStream_t s,
                                  const T&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

constexpr int MAX_CASES = WM_MAX_BLOCKS;   // a case has at least one block

// SMs of a B200: the constant where a rule for spreading work (or the order of a sum) must not depend on the device
constexpr int CHIP_SMS = 148;

// x / d of a divisor known at set-up, for 0 <= x < 2^31: (x mul) >> shift with mul = ceil(2^shift / d),
// shift = 31 + ceil(log2 d) (mul < 2^33 x 2^31 fits 64 bits; exact for 31-bit x)
struct FastDiv {
    unsigned long long mul;
    int shift;
    __host__ void set(unsigned d) {
        int l = 0;
        while ((1u << l) < d) ++l;
        shift = 31 + l;
        mul = ((1ull << shift) + d - 1) / d;
    }
    __host__ __device__ int operator()(unsigned x) const { return (int)((x * mul) >> shift); }
};

// one structured block, resident in device memory
struct BlockDev {
    int n[3];          // interior cells
    int N[3];          // ghosted extents
    int ng;
    int case_id;       // index of the block's case in the view
    long long ncell;   // Ni*Nj*Nk
    long long plane;   // Nj*Nk
    const double* met;     // WM_NMET x ncell (float64)
    const float* met32;    // WM_NMET x ncell (float32 copy for the mixed form), may be null
    int wall[6];       // view wall index of face (axis*2 + side), -1 if not wall-modelled
    int tj, tk;        // shape of its stage tiles in this view
    FastDiv div_nj, div_nk;   // by n[1], n[2]
    // blocks extruded along k (ext_check in geom.cu): metrics per (i, j) row and per k; else null
    const double* rows;    // N[0] x N[1] x RT_N
    const double* ktab;    // N[2] x 2: area factor of i and j faces, inverse centre distance to k - 1
    const float *rows32, *ktab32;   // rounded copies (mixed form)
};

// entries of a row of an extruded block (x, y components unless noted)
enum { RT_SI = 0, RT_HI = 2 /* lower, upper i face */, RT_SJ = 4, RT_SK = 6 /* z */, RT_EI = 7, RT_IDI = 9,
       RT_EJ = 10, RT_IDJ = 12,
       RT_MI = 13, RT_MJ = 14 /* lengths of the means of the lower and upper i and j face vectors */, RT_N = 16 };

template <typename R>
__device__ __forceinline__ const R* rows_of(const BlockDev& B) {
    if constexpr (sizeof(R) == 4) return B.rows32;
    else return B.rows;
}
template <typename R>
__device__ __forceinline__ const R* ktab_of(const BlockDev& B) {
    if constexpr (sizeof(R) == 4) return B.ktab32;
    else return B.ktab;
}

// per-case physical constants, precomputed where the kernels only need a derived value
struct CaseDev {
    double gamma, Rg, Pr, Prt, mu_ref, T_ref, S_suth;
    double cp, gm1, inv_gm1, inv_Rg, inv_Tref, TrefS, inv_Pr, inv_Prt;
    double th0, inv_dth;   // Hybrid: s = clip((theta - th0) * inv_dth, 0, 1)
    double sgs_c;          // model coefficient
    double cfl, nu_fac;    // nu_fac = max(4/3, gamma/Pr)
    double c_ref;          // speed of sound at T_ref
    double Pr13, Pr3, kader_beta;   // Pr^(1/3), Pr^3, (3.85 Pr^(1/3) - 1.3)^2 + 2.12 ln Pr
    int cmf_dir;
    double cmf_target, cmf_volume;
    double cmf_bin[3];     // roundings of the mass-flux sum (cmf_bins in capi.cu)
    int sponge;
    double sp_xs, sp_inv_dx, sp_sigma0, sp_invL;   // sigma = sigma0 * ramp(eta)
    unsigned int* status;  // the case's status word (WM_ST_* bits, set with atomicOr)
};

struct WallDev {
    int block, axis, side, n_match;   // block: view block index
    int isothermal, n_iter;
    int nt1, nt2;              // tangential interior extents (axes in increasing order)
    double T_wall, kappa, B, ekb;
    const double* geom;        // 5 x nf
    double* F;                 // 5 x nf flux override (written by the wall kernel)
    double* tq;                // 2 x nf (tau_w, q_w)
};

// stage-kernel work item: one (j,k) tile of one block over planes [i0, i1)
struct Tile {
    int blk, j0, k0, i0, i1;   // blk: view block index
    int tj, tk;                // extents of this tile (the block's last ones may be smaller)
};

// one case's ghost-cell program inside a view-wide gather launch
struct GhostSeg {
    const int* dst;
    const int* src;
    const int* ops;
    const int* op_code;
    const double* op_nrm;
    const double* bc;          // the case's BC table (8 per BC)
    const double* inflow;      // 5 x inflow_n (or null)
    long long inflow_n;
    int start, count;          // entries [start, start + count) of the launch
    int block0;                // view index of the case's first block
    double gamma, gm1, Rg;
};

struct StatePtrs {
    const double* q_in;    // stage input (ghosts filled)
    const double* q0;      // Q at the start of the step (RK stages 2, 3)
    double* q_out;         // stage output (interior written)
    const double* spmean;  // sponge spanwise mean of q_in, 5 x Ni x Nj (or null)
};

// records the calling thread's error text (read by wm_last_error) and returns `code`
int set_error(int code, const char* msg);

struct StageArgs {
    const BlockDev* blocks;
    const CaseDev* cases;
    const WallDev* walls;
    const Tile* tiles;
    const int* cta_first;         // CTA c runs tiles [cta_first[c], cta_first[c+1]); null: tile c
    int nctas;                    // grid size
    int stage;                    // 0: q_out = RHS; 1,2,3: SSP-RK3 stage
    int ncases;
    double* cmf_sum;              // stage 3 with constant mass flux: per case the sum of rho u V in three bins
                                  // (zero between steps: reset by the last CTA); else null
    unsigned int* cmf_counter;    // last-CTA-done counter (the last CTA resets it)
    int cmf_ctas;                 // CTAs of the stage's launches
    int ext;                      // the tiles' blocks are extruded along k
    double* cmf_delta;            // per case: constant-mass-flux shift, written by the last CTA
    const double* dt[MAX_CASES];  // per case: device time step
    StatePtrs p[WM_MAX_BLOCKS];
};

}  // namespace wm
