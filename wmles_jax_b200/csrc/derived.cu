// Derived output fields on the device (derived_fields, wmles/io_vtk.py:269-293): per interior
// cell rho, velocity, pressure, temperature, Mach number, SGS viscosity mu_t, molecular
// viscosity, vorticity magnitude and Q-criterion, from a state whose first ghost layer is
// filled, so output needs no copy of the state to the host.
//
// FP64.  The velocity gradient is the Green-Gauss gradient of wmles/viscous.py:6-19 (face values =
// means of the two cells, times the face area vector, over the volume), the SGS viscosity the
// case's model (wmles/sgs.py:14-50).
#include <algorithm>
#include "physics.cuh"
#include "aux.cuh"
#include "derived.cuh"

namespace wm {

// What bounds it: HBM (40 B of state and 88 B of metrics in, 88 B of fields out per cell) once divisions
// and latency are out of the way.  A CTA marches along i over a (j, k) tile, one column per thread: the
// velocities of a plane and its halo are divided once, kept in registers for the i neighbours and in shared
// memory for the j and k ones, and the next plane's state is loaded while the current one is computed.
// Blocks extruded along k read their face areas from the (i, j) row (B.rows) instead of 18 values per cell.
// 192 x 96 x 96: 229 -> 120 us (one reciprocal per neighbour and no march: 157; three CTAs' worth of threads
// at 80 registers: 156).  What is left is the latency of the roots and divisions of a cell at 16 warps per SM.
constexpr int DV_NT = 128, DV_CPS = 4;
constexpr int DV_SLOTS = 204;        // (tj + 2) (tk + 2) of the largest tiles, 32 x 4 and 4 x 32

// fields of one cell: um, u0, up velocities of its i neighbours and itself, vs the plane's velocities at it
__device__ __forceinline__ void derived_cell(const DerivedArgs& A, const BlockDev& B, const CaseDev& C, const double um[3],
                                             const double u0[3], const double up[3], const double* vs, int pitch,
                                             double rho, double E, int i, int j, int k, double kt, const double* rows,
                                             const double* met, long long c, long long ni_cells, long long N, int plane,
                                             int Nk, int Nj) {
    const int idx = i * plane + j * Nk + k;
    const double iv = __ldg(met + WM_MET_IVOL * N + idx);
    const double* row = rows ? rows + ((long long)i * Nj + j) * RT_N : nullptr;
    double acc[3][3] = {};       // acc[a][x]: sum over the faces of u_a S_x
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int off = d == 0 ? plane : d == 1 ? Nk : 1, soff = d == 1 ? pitch : 1;
        double sl[3] = {}, sh[3] = {};
        if (row) {
            if (d == 2) {
                sl[2] = sh[2] = __ldg(row + RT_SK);
            } else {
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    sl[x] = __ldg(row + (d ? RT_SJ : RT_SI) + x) * kt;
                    sh[x] = __ldg(row + (d ? RT_N + RT_SJ : RT_HI) + x) * kt;
                }
            }
        } else {
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                sl[x] = __ldg(met + (3 * d + x) * N + idx);
                sh[x] = __ldg(met + (3 * d + x) * N + idx + off);
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double ul = d == 0 ? um[a] : vs[a * DV_SLOTS - soff], uh = d == 0 ? up[a] : vs[a * DV_SLOTS + soff];
            const double lo = 0.5 * (ul + u0[a]), hi = 0.5 * (u0[a] + uh);
#pragma unroll
            for (int x = 0; x < 3; ++x) acc[a][x] += hi * sh[x] - lo * sl[x];
        }
    }
    // g[3 a + d] = d u_a / d x_d
    double g[9];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int x = 0; x < 3; ++x) g[3 * a + x] = acc[a][x] * iv;
    const double ke = (u0[0] * u0[0] + u0[1] * u0[1]) + u0[2] * u0[2];
    const double p = C.gm1 * (E - (0.5 * rho) * ke);
    const double T = p / (rho * C.Rg);
    const double mu = sutherland_d(T, C);
    const double mut = A.sgs != WM_SGS_NONE ? rho * sgs_nut<double>(A.sgs, g, __ldg(met + WM_MET_DELTA * N + idx), C.sgs_c) : 0.0;
    const double wxy = g[3] - g[1], wxz = g[6] - g[2], wyz = g[7] - g[5];
    const double om = sqrt((wxy * wxy + wxz * wxz) + wyz * wyz);
    double s2 = 0.0, o2 = 0.0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const double s = 0.5 * (g[3 * a + b] + g[3 * b + a]), o = 0.5 * (g[3 * a + b] - g[3 * b + a]);
            s2 += s * s;
            o2 += o * o;
        }
    const double qc = 0.5 * (o2 - s2);
    const double mach = sqrt(ke) / sqrt(C.gamma * C.Rg * T);
    const double out[WM_NDERIVED] = {rho, u0[0], u0[1], u0[2], p, T, mach, mut, mu, om, qc};
#pragma unroll
    for (int v = 0; v < WM_NDERIVED; ++v) A.out[(long long)v * ni_cells + c] = out[v];
}

__global__ void __launch_bounds__(DV_NT, DV_CPS) derived_kernel(const __grid_constant__ DerivedArgs A) {
    __shared__ double vs[2][3][DV_SLOTS];
    const BlockDev& B = *A.block;
    const CaseDev& C = *A.cs;
    const int ng = B.ng, nj = B.n[1], nk = B.n[2], Nk = B.N[2], plane = (int)B.plane, Nj = B.N[1];
    const long long N = B.ncell;
    const long long ni_cells = (long long)B.n[0] * nj * nk;
    const int tk = 1 << A.lt, tj = DV_NT >> A.lt, pitch = tk + 2;
    const int j0 = int(blockIdx.x) / A.ktiles * tj, k0 = int(blockIdx.x) % A.ktiles * tk;
    const int jn = min(tj, nj - j0), kn = min(tk, nk - k0);          // the tile's columns
    const int ia = ng + blockIdx.y * A.planes, ib = min(ia + A.planes, ng + B.n[0]);
    const int tx = threadIdx.x & (tk - 1), ty = threadIdx.x >> A.lt;
    const bool act = tx < kn && ty < jn;
    const int j = j0 + ty + ng, k = k0 + tx + ng;
    const int col = j * Nk + k, slot = (ty + 1) * pitch + tx + 1;
    // halo column of this thread: below and above the tile in j (tk each), then in k (tj each)
    int hcol = 0, hslot = -1;
    {
        const int h = threadIdx.x, e = h - 2 * tk;
        int hj = -1, hk = -1;
        if (h < 2 * tk) {
            hk = (h & (tk - 1)) + 1;
            hj = h < tk ? 0 : jn + 1;
            if (hk > kn) hk = -1;
        } else if (e < 2 * tj) {
            hj = (e < tj ? e : e - tj) + 1;
            hk = e < tj ? 0 : kn + 1;
            if (hj > jn) hk = -1;
        }
        if (hk >= 0) {
            hslot = hj * pitch + hk;
            hcol = (j0 + hj - 1 + ng) * Nk + (k0 + hk - 1 + ng);
        }
    }
    const double* q = A.q;
    const double* met = B.met;
    const double* rows = B.rows;
    const double kt = rows && act ? __ldg(B.ktab + 2 * k) : 1.0;
    auto load = [&](double w[5], int i, int c, int nv) {
#pragma unroll
        for (int v = 0; v < 5; ++v)
            if (v < nv) w[v] = __ldg(q + v * N + (i * plane + c));
    };
    double um[3] = {}, u0[3] = {}, w0[5] = {}, wn[5] = {}, hn[4] = {};
    if (act) {
        load(wn, ia - 1, col, 4);
        load(w0, ia, col, 5);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            um[a] = wn[1 + a] / wn[0];
            vs[ia & 1][a][slot] = u0[a] = w0[1 + a] / w0[0];
        }
        load(wn, ia + 1, col, 5);
    }
    if (hslot >= 0) {
        load(hn, ia, hcol, 4);
#pragma unroll
        for (int a = 0; a < 3; ++a) vs[ia & 1][a][hslot] = hn[1 + a] / hn[0];
        if (ia + 1 < ib) load(hn, ia + 1, hcol, 4);
    }
    __syncthreads();
    for (int i = ia; i < ib; ++i) {
        // plane i + 1 to shared memory (read after this plane's barrier), plane i + 2 under way
        const double rho = w0[0], E = w0[4];
        double up[3] = {};
        if (act) {
#pragma unroll
            for (int a = 0; a < 3; ++a) vs[(i + 1) & 1][a][slot] = up[a] = wn[1 + a] / wn[0];
#pragma unroll
            for (int v = 0; v < 5; ++v) w0[v] = wn[v];
            if (i + 1 < ib) load(wn, i + 2, col, 5);
        }
        if (hslot >= 0 && i + 1 < ib) {
#pragma unroll
            for (int a = 0; a < 3; ++a) vs[(i + 1) & 1][a][hslot] = hn[1 + a] / hn[0];
            if (i + 2 < ib) load(hn, i + 2, hcol, 4);
        }
        if (act) derived_cell(A, B, C, um, u0, up, &vs[i & 1][0][slot], pitch, rho, E, i, j, k, kt, rows, met,
                              ((long long)(i - ng) * nj + (j - ng)) * nk + (k - ng), ni_cells, N, plane, Nk, Nj);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            um[a] = u0[a];
            u0[a] = up[a];
        }
        __syncthreads();
    }
}

cudaError_t launch_derived(DerivedArgs A, const int n[3], cudaStream_t s) {
    if (n[0] <= 0 || n[1] <= 0 || n[2] <= 0) return cudaSuccess;
    // tile: as wide in k as the block, in powers of two from 4 to 32; planes per CTA: one wave of CTAs
    A.lt = 2;
    while (A.lt < 5 && (1 << A.lt) < n[2]) ++A.lt;
    const int tk = 1 << A.lt, tj = DV_NT >> A.lt;
    A.ktiles = (n[2] + tk - 1) / tk;
    const int tiles = (n[1] + tj - 1) / tj * A.ktiles;
    const int chunks = std::min(n[0], std::max((n[0] + 31) / 32, CHIP_SMS * DV_CPS / tiles));
    A.planes = (n[0] + chunks - 1) / chunks;
    derived_kernel<<<dim3(tiles, (n[0] + A.planes - 1) / A.planes), DV_NT, 0, s>>>(A);
    return cudaGetLastError();
}

}  // namespace wm
