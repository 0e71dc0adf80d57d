// Launch interface of the fused stage kernel (stage.cu).
#pragma once
#include "wm_internal.cuh"

namespace wm {

struct StageOpts {
    int precision;   // WM_PREC_*
    int scheme;      // WM_SCHEME_*
    int kep_order;   // 2 or 4
    int limiter;     // WM_LIMITER_*
    int sgs;         // WM_SGS_*
    int tile;        // tile shape id (-1: a shape per block, see tile_shape)
};

// shared-memory capacities of a kernel variant with `cap` tile columns: primitive cells (tile +
// 2-cell halo), gradient records (tile + 1-cell halo), j and k faces, rows (tile + 3) and k
// positions (tile + 2)
struct StageCaps {
    int pn, gn, fn, rows, kn;
};
constexpr StageCaps stage_caps(int cap) {
    return cap == 512 ? StageCaps{736, 640, 1072, 28, 144} : StageCaps{440, 342, 552, 20, 84};
}

// cost of a segment beyond its planes, in planes: its prologue and the gradient and i-face planes
// at its ends
constexpr double SEG_PLANES = 2.0;
// Cheapest way to share `cols` columns of n0 planes among `slots` CTAs, in planes of the slowest
// CTA: either chunks of *chunk planes, one CTA each, or (*tail > 0) the lockstep wave split
// (build_waves, capi.cu) that leaves the last *tail planes to the CTAs left over.
double split_planes(long long cols, int n0, int slots, int* chunk, int* tail);

// tile columns of the kernel variant the options select
int stage_cap(const StageOpts& o);
cudaError_t launch_stage(const StageArgs& A, const StageOpts& o, cudaStream_t s);
void tile_shape(const StageOpts& o, const int n[3], int count, int slots, int* tj, int* tk);
int stage_ctas_per_sm(const StageOpts& o);

}  // namespace wm
