// Plane statistics of a channel block (PlaneStats.accumulate, wmles/channel5200.py:121-152):
// per interior j-plane, the means over interior (i, k) of rho, u, v, w, uu, vv, ww, uv, uw,
// vw, T, p, added to a device accumulator, so a driver samples the flow every few steps
// without copying the state to the host.
//
// One CTA per (i-chunk, plane): each thread walks its cells of the chunk and keeps the 12
// FP64 sums in registers; a block reduction writes one partial per quantity; the last CTA of
// a plane adds, per quantity, the plane's chunk partials in chunk order divided by its cell count (a
// fixed order: the result does not depend on scheduling).
//
// What bounds it: the state is read once (40 B per cell), so HBM if enough loads are in flight
// and the arithmetic is short: one reciprocal per cell instead of four divisions, two cells
// per thread at a time, as many chunks as one wave of CTAs holds (plane_chunks), and a last CTA
// per plane (one for all planes took 11 us by itself).  192 x 96 x 96: 59 -> 23 us.
#include <algorithm>
#include <cfloat>
#include "wm_internal.cuh"
#include "stats.cuh"

namespace wm {

constexpr int PS_NT = 128, PS_CPS = 8;       // threads per CTA, CTAs resident per SM

__global__ void __launch_bounds__(PS_NT, PS_CPS) plane_stats_kernel(const __grid_constant__ PlaneStatsArgs A) {
    __shared__ double red[PS_NQ][PS_NT / 32];
    __shared__ bool last;
    const BlockDev& B = *A.block;
    const int ng = B.ng, ni = B.n[0], nk = B.n[2], Nk = B.N[2], plane = (int)B.plane;
    const int chunk = blockIdx.x, jj = blockIdx.y;          // jj: interior plane index
    const int i0 = (int)((long long)chunk * ni / A.nchunks), i1 = (int)((long long)(chunk + 1) * ni / A.nchunks);
    const long long N = B.ncell;
    const FastDiv div_nk = B.div_nk;
    const double* q = A.q;
    const double iRg = 1.0 / A.Rg;
    double acc[PS_NQ];
#pragma unroll
    for (int x = 0; x < PS_NQ; ++x) acc[x] = 0.0;
    const int cells = (i1 - i0) * nk, base = (i0 + ng) * plane + (jj + ng) * Nk + ng;
    auto load = [&](int c, double w[5]) {
        const int i = div_nk(c);
        const int idx = base + i * plane + (c - i * nk);
#pragma unroll
        for (int v = 0; v < 5; ++v) w[v] = __ldg(q + v * N + idx);
    };
    auto add = [&](const double w[5]) {
        // gas.cons_to_prim (wmles/gas.py:28-33)
        const double rho = w[0], ir = 1.0 / rho;
        const double u = w[1] * ir, v = w[2] * ir, ww = w[3] * ir;
        const double p = A.gm1 * (w[4] - (0.5 * rho) * ((u * u + v * v) + ww * ww));
        const double x[PS_NQ] = {rho, u, v, ww, u * u, v * v, ww * ww, u * v, u * ww, v * ww, p * ir * iRg, p};
#pragma unroll
        for (int y = 0; y < PS_NQ; ++y) acc[y] += x[y];
    };
    int c = threadIdx.x;
    for (; c + PS_NT < cells; c += 2 * PS_NT) {
        double wa[5], wb[5];
        load(c, wa);
        load(c + PS_NT, wb);
        add(wa);
        add(wb);
    }
    if (c < cells) {
        double wa[5];
        load(c, wa);
        add(wa);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < PS_NQ; ++q) {
        double s = acc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) red[q][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x < PS_NQ) {
        double s = 0.0;
        for (int wv = 0; wv < PS_NT / 32; ++wv) s += red[threadIdx.x][wv];
        A.part[((long long)threadIdx.x * B.n[1] + jj) * A.nchunks + chunk] = s;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(A.counter + jj, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < PS_NQ) {
        const long long e = (long long)threadIdx.x * B.n[1] + jj;
        double s = 0.0;
#pragma unroll 8
        for (int ch = 0; ch < A.nchunks; ++ch) s += __ldcg(A.part + e * A.nchunks + ch);
        A.sum[e] += s * (1.0 / ((double)ni * nk));
    }
    if (threadIdx.x == 0) A.counter[jj] = 0u;
}

// chunks per plane: one wave of CTAs on CHIP_SMS (a constant, so that the order of the sums does
// not depend on the device), at most PS_CHUNKS and one plane of cells each
int plane_chunks(int ni, int nj) {
    return std::max(1, std::min({PS_CHUNKS, ni, CHIP_SMS * PS_CPS / std::max(1, nj)}));
}

cudaError_t launch_plane_stats(const PlaneStatsArgs& A, int nj, cudaStream_t s) {
    dim3 grid(A.nchunks, nj);
    plane_stats_kernel<<<grid, PS_NT, 0, s>>>(A);
    return cudaGetLastError();
}

}  // namespace wm
