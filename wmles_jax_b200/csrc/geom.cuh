// Block geometry and packed metric table on the device (geom.cu).
#pragma once
#include <cuda_runtime.h>

namespace wm {

struct GeomArgs {
    const double* X;             // 3 x (N0+1) x (N1+1) x (N2+1) nodes, ghost nodes filled
    int N[3];                    // cells per direction including ghosts
    double* vol;                 // N0 x N1 x N2
    double* xc;                  // 3 x N0 x N1 x N2
    double* S[3];                // 3 x (N0 + (d==0)) x (N1 + (d==1)) x (N2 + (d==2))
    double* xf[3];               // same extents as S[d]
    double* met;                 // WM_NMET x N0 x N1 x N2, or null
};

cudaError_t launch_geometry(const GeomArgs& A, cudaStream_t s);

// A block extruded along k: in every cell the stage kernels read, S_i, S_j, e_i and e_j have no z
// component and S_k = (0, 0, Skz), e_k = (0, 0, 1) exactly; Skz, e and 1/|dx| of i and j faces
// do not depend on k, S_i and S_j only through one factor per k (ktab[2 k]), and 1/|dx| of k
// faces only on k (ktab[2 k + 1]), to `tol`.  Clears *flag where that does not hold.  met: WM_NMET x
// N0 x N1 x N2; k0: the reference k (factor 1).
cudaError_t launch_ext_check(const double* met, const int N[3], int ng, int k0, const double* ktab, double tol, int* flag,
                             cudaStream_t s);
// rows of such a block (N0 x N1 x RT_N) from its metrics at k0
cudaError_t launch_ext_rows(const double* met, const int N[3], int k0, double* rows, cudaStream_t s);

// dst[i] = (float)src[i] (round to nearest), i < n
cudaError_t launch_to_f32(const double* src, float* dst, long long n, cudaStream_t s);

}  // namespace wm
