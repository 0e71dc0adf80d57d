// Per-cell and per-face physics of the wmles RHS, templated on the compute type R
// (double for the FP64 form, float for the mixed form).  Each function cites the
// reference formula it evaluates (EduardoMolina/wmles_jax).
#pragma once
#include <cuda_runtime.h>
#include "wm_internal.cuh"

namespace wm {

template <typename R>
struct Phys {
    R gamma, gm1, inv_gm1, Rg, inv_Rg, cp, inv_Pr, inv_Prt;
    R mu_ref, inv_Tref, TrefS, S_suth;
    R th0, inv_dth, sgs_c;
    __device__ explicit Phys(const CaseDev& c)
        : gamma(R(c.gamma)), gm1(R(c.gm1)), inv_gm1(R(c.inv_gm1)), Rg(R(c.Rg)), inv_Rg(R(c.inv_Rg)),
          cp(R(c.cp)), inv_Pr(R(c.inv_Pr)), inv_Prt(R(c.inv_Prt)), mu_ref(R(c.mu_ref)),
          inv_Tref(R(c.inv_Tref)), TrefS(R(c.TrefS)), S_suth(R(c.S_suth)), th0(R(c.th0)),
          inv_dth(R(c.inv_dth)), sgs_c(R(c.sgs_c)) {}
};

__device__ __forceinline__ double wm_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float wm_sqrt(float x) { return sqrtf(x); }

// primitive record kept per cell in shared memory: rho, u, v, w, p, e = p/((g-1)rho) + |u|^2/2, T
enum { PR_RHO = 0, PR_U, PR_V, PR_W, PR_P, PR_E, PR_T, PR_N };

// conservative -> primitive record, wmles/gas.py:28-33
template <typename R>
__device__ __forceinline__ void cons_to_rec(const double q[5], const Phys<R>& P, R out[PR_N]) {
    const R rho = R(q[0]);
    const R ir = R(1) / rho;
    const R u = R(q[1]) * ir, v = R(q[2]) * ir, w = R(q[3]) * ir;
    const R ke = R(0.5) * (u * u + v * v + w * w);
    const R p = P.gm1 * (R(q[4]) - rho * ke);
    out[PR_RHO] = rho; out[PR_U] = u; out[PR_V] = v; out[PR_W] = w; out[PR_P] = p;
    out[PR_T] = p * ir * P.inv_Rg;
    out[PR_E] = p * ir * P.inv_gm1 + ke;
}

// Sutherland viscosity, wmles/gas.py:24-26 ((T/T_ref)^1.5 as x sqrt(x))
template <typename R>
__device__ __forceinline__ R sutherland(R T, const Phys<R>& P) {
    const R x = T * P.inv_Tref;
    return P.mu_ref * (x * wm_sqrt(x)) * P.TrefS / (T + P.S_suth);
}

// Orientation of a face's area vector S and centre-to-centre vector e, known at compile time on
// grids extruded along k: FACE_XY (S and e in the x-y plane) leaves out the products with
// their zero z components, FACE_Z (S = (0, 0, Sz), e = (0, 0, 1)) those with x and y.  The terms
// left out are exact zeros, so finite results do not change; where the general form adds such a
// zero to a product, prod() keeps the product rounded by itself in the float form (the same bits
// as the general form).
enum { FACE_ANY = 0, FACE_XY = 1, FACE_Z = 2 };
__device__ __forceinline__ float prod(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double prod(double a, double b) { return a * b; }

// (x, y, z) . S
template <int FACE, typename R>
__device__ __forceinline__ R dot_s(R x, R y, R z, R Sx, R Sy, R Sz) {
    if constexpr (FACE == FACE_XY) return x * Sx + y * Sy;
    else if constexpr (FACE == FACE_Z) return prod(z, Sz);
    else return x * Sx + y * Sy + z * Sz;
}
// a * b + c * S, where S is the x (A = 0), y or z (A = 2) component.  The float form's contraction is
// spelled out, or it would be the compiler's choice by what surrounds it and differ by orientation
template <int FACE, int A>
__device__ __forceinline__ double madd_s(double a, double b, double c, double S) {
    if constexpr ((FACE == FACE_XY && A == 2) || (FACE == FACE_Z && A < 2)) return a * b;
    else return a * b + c * S;
}
template <int FACE, int A>
__device__ __forceinline__ float madd_s(float a, float b, float c, float S) {
    if constexpr ((FACE == FACE_XY && A == 2) || (FACE == FACE_Z && A < 2)) return __fmul_rn(a, b);
    else return __fmaf_rn(c, S, __fmul_rn(a, b));
}

// Kennedy-Gruber two-point flux (already times the face area), wmles/schemes.py:15-23
template <int FACE, typename R>
__device__ __forceinline__ void kg_flux(const R* a, int sa, const R* b, int s, R Sx, R Sy, R Sz, R F[5]) {
    const R rho = R(0.5) * (a[PR_RHO * sa] + b[PR_RHO * s]);
    const R u = R(0.5) * (a[PR_U * sa] + b[PR_U * s]);
    const R v = R(0.5) * (a[PR_V * sa] + b[PR_V * s]);
    const R w = R(0.5) * (a[PR_W * sa] + b[PR_W * s]);
    const R p = R(0.5) * (a[PR_P * sa] + b[PR_P * s]);
    const R ea = R(0.5) * (a[PR_E * sa] + b[PR_E * s]);
    const R un = dot_s<FACE>(u, v, w, Sx, Sy, Sz);
    const R m = rho * un;
    F[0] = m;
    F[1] = madd_s<FACE, 0>(m, u, p, Sx);
    F[2] = madd_s<FACE, 1>(m, v, p, Sy);
    F[3] = madd_s<FACE, 2>(m, w, p, Sz);
    F[4] = m * ea + p * un;
}

// KEP order 2 / 4, wmles/schemes.py:57-70: 2 [(2/3) F(L,R) - (1/12) (F(L,R2) + F(L2,R))],
// written (4/3) F(L,R) - (1/6) (...) (the outer factor 2 moved into the constants: exact)
template <int FACE, typename R>
__device__ __forceinline__ void kep_flux(int order, const R* L2, int s2, const R* L, const R* Rr,
                                         const R* R2, int s, R Sx, R Sy, R Sz, R F[5]) {
    kg_flux<FACE>(L, s, Rr, s, Sx, Sy, Sz, F);
    if (order == 4) {
        R Fa[5], Fb[5];
        kg_flux<FACE>(L, s, R2, s, Sx, Sy, Sz, Fa);
        kg_flux<FACE>(L2, s2, Rr, s, Sx, Sy, Sz, Fb);
#pragma unroll
        for (int v = 0; v < 5; ++v)
            F[v] = R(4.0 / 3.0) * F[v] - R(1.0 / 6.0) * (Fa[v] + Fb[v]);
    }
}

// limiters, wmles/schemes.py:100-105
template <typename R>
__device__ __forceinline__ R albada(R a, R b) {
    const R eps = R(1e-12);
    return (a * (b * b + eps) + b * (a * a + eps)) / (a * a + b * b + R(2) * eps);
}
template <typename R>
__device__ __forceinline__ R sgn(R a) { return R((a > R(0)) - (a < R(0))); }
template <typename R>
__device__ __forceinline__ R minmod(R a, R b) {
    return R(0.5) * (sgn(a) + sgn(b)) * fmin(fabs(a), fabs(b));
}

// both limited slopes of one variable at a face, albada(a, b) and albada(b, c).  FP64: the two
// quotients from one division (1 / (d1 d2) times the other denominator; the denominators are at
// least 2e-12), as a division is some 30 instructions and a face takes ten
template <typename R>
__device__ __forceinline__ void albada2(R a, R b, R c, R& l, R& r) {
    if constexpr (sizeof(R) == 8) {
        const R eps = R(1e-12);
        const R a2 = a * a, b2 = b * b, c2 = c * c;
        const R d1 = a2 + b2 + R(2) * eps, d2 = b2 + c2 + R(2) * eps;
        const R q = R(1) / (d1 * d2);
        l = (a * (b2 + eps) + b * (a2 + eps)) * (d2 * q);
        r = (b * (c2 + eps) + c * (b2 + eps)) * (d1 * q);
    } else {
        l = albada(a, b);
        r = albada(b, c);
    }
}

// a / b from inv, 1 / b to a few units in the last place: one correction by the remainder, so that the quotient
// is rounded about as a division rounds it
__device__ __forceinline__ double quotient(double a, double b, double inv) {
    const double q = a * inv;
    return fma(fma(-q, b, a), inv, q);
}

// HLLC flux times |S|, wmles/schemes.py:108-137
template <int FACE, typename R>
__device__ __forceinline__ void hllc_flux(const R wl[5], const R wr[5], R Sx, R Sy, R Sz, R gamma,
                                          R inv_gm1, R F[5]) {
    const R Sm = wm_sqrt(dot_s<FACE>(Sx, Sy, Sz, Sx, Sy, Sz));
    const R iS = R(1) / Sm;
    const R nx = Sx * iS, ny = Sy * iS, nz = Sz * iS;
    constexpr bool D = sizeof(R) == 8;           // FP64: quotients that share a division (below)
    const R rl = wl[0], ul = wl[1], vl = wl[2], wlz = wl[3], pl = wl[4];
    const R rr = wr[0], ur = wr[1], vr = wr[2], wrz = wr[3], pr = wr[4];
    const R unl = dot_s<FACE>(ul, vl, wlz, nx, ny, nz);
    const R unr = dot_s<FACE>(ur, vr, wrz, nx, ny, nz);
    // FP64: 1 / rl and 1 / rr from 1 / (rl rr), later 1 / (s - un) and 1 / (s - ss) from their
    // product's: four divisions a face instead of seven, of some 30 instructions each.  The two quotients
    // that the flux is proportional to are corrected (uncorrected, the residual's error against extended precision
    // was 14-20 % larger than with divisions; the other two, under a root and beside a larger term,
    // make no difference to it)
    const R irr = D ? R(1) / (rl * rr) : R(0), il = rr * irr, ir = rl * irr;
    const R cl = wm_sqrt(D ? gamma * pl * il : gamma * pl / rl), cr = wm_sqrt(D ? gamma * pr * ir : gamma * pr / rr);
    const R sL = fmin(unl - cl, unr - cr), sR = fmax(unl + cl, unr + cr);
    const R ss = (pr - pl + rl * unl * (sL - unl) - rr * unr * (sR - unr)) /
                 (rl * (sL - unl) - rr * (sR - unr));
    // choose the side, then evaluate only that branch
    const bool left = (sL >= R(0)) || (ss >= R(0));
    const R r = left ? rl : rr, u = left ? ul : ur, v = left ? vl : vr, w = left ? wlz : wrz;
    const R p = left ? pl : pr, un = left ? unl : unr;
    const R E = p * inv_gm1 + R(0.5) * r * (u * u + v * v + w * w);
    R Fp[5];
    Fp[0] = r * un;
    Fp[1] = madd_s<FACE, 0>(r * un, u, p, nx);
    Fp[2] = madd_s<FACE, 1>(r * un, v, p, ny);
    Fp[3] = madd_s<FACE, 2>(r * un, w, p, nz);
    Fp[4] = (E + p) * un;
    const bool star = left ? !(sL >= R(0)) : (sR > R(0));
    if (star) {
        const R s = left ? sL : sR;
        R f, e;
        if constexpr (D) {
            const R a = s - un, b = s - ss, q = R(1) / (a * b), ra = r * a;
            const R iro = left ? il : ir;
            f = quotient(ra, b, a * q);
            e = quotient(E, r, iro) + (ss - un) * (ss + p * (iro * (b * q)));
        } else {
            f = r * (s - un) / (s - ss);
            e = E / r + (ss - un) * (ss + p / (r * (s - un)));
        }
        const R d = ss - un;
        Fp[0] += s * (f - r);
        Fp[1] += s * (f * (FACE == FACE_Z ? u : u + d * nx) - r * u);
        Fp[2] += s * (f * (FACE == FACE_Z ? v : v + d * ny) - r * v);
        Fp[3] += s * (f * (FACE == FACE_XY ? w : w + d * nz) - r * w);
        Fp[4] += s * (f * e - E);
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) F[q] = Fp[q] * Sm;
}

// MUSCL reconstruction with positivity fallback + HLLC, wmles/schemes.py:140-152
template <int FACE, typename R>
__device__ __forceinline__ void muscl_hllc_flux(int limiter, const R* L2, int s2, const R* L, const R* Rr,
                                                const R* R2, int s, R Sx, R Sy, R Sz,
                                                const Phys<R>& P, R F[5]) {
    R wl[5], wr[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
        const R a = L[v * s] - L2[v * s2], b = Rr[v * s] - L[v * s], c = R2[v * s] - Rr[v * s];
        if (limiter == WM_LIMITER_MINMOD) {
            wl[v] = L[v * s] + R(0.5) * minmod(a, b);
            wr[v] = Rr[v * s] - R(0.5) * minmod(b, c);
        } else {
            R sl, sr;
            albada2(a, b, c, sl, sr);
            wl[v] = L[v * s] + R(0.5) * sl;
            wr[v] = Rr[v * s] - R(0.5) * sr;
        }
    }
    if (wl[0] <= R(0) || wl[4] <= R(0) || wr[0] <= R(0) || wr[4] <= R(0)) {
#pragma unroll
        for (int v = 0; v < 5; ++v) { wl[v] = L[v * s]; wr[v] = Rr[v * s]; }
    }
    hllc_flux<FACE>(wl, wr, Sx, Sy, Sz, P.gamma, P.inv_gm1, F);
}

// SGS eddy viscosity nu_t from g[i][j] = du_i/dx_j, wmles/sgs.py:14-42
template <typename R>
__device__ __forceinline__ R sgs_nut(int model, const R g[9], R delta, R c) {
    if (model == WM_SGS_SMAGORINSKY) {
        R ss = R(0);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const R s = R(0.5) * (g[3 * i + j] + g[3 * j + i]);
                ss += s * s;
            }
        const R cd = c * delta;
        return cd * cd * wm_sqrt(R(2) * ss);
    }
    if (model == WM_SGS_WALE) {
        // S_ij S_ij and S^d_ij S^d_ij from the six distinct entries of each symmetric tensor
        // (off-diagonal squares counted twice, an exact doubling), summed as trees: the
        // reference's contractions up to the order of the additions, with dependency chains
        // of four additions instead of nine
        R g2[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                g2[3 * i + j] = g[3 * i] * g[j] + g[3 * i + 1] * g[3 + j] + g[3 * i + 2] * g[6 + j];
        const R s01 = R(0.5) * (g[1] + g[3]), s02 = R(0.5) * (g[2] + g[6]), s12 = R(0.5) * (g[5] + g[7]);
        const R ss = ((g[0] * g[0] + g[4] * g[4]) + g[8] * g[8]) + R(2) * ((s01 * s01 + s02 * s02) + s12 * s12);
        const R tr = (g2[0] + g2[4] + g2[8]) * R(1.0 / 3.0);
        const R d0 = g2[0] - tr, d1 = g2[4] - tr, d2 = g2[8] - tr;
        const R q01 = R(0.5) * (g2[1] + g2[3]), q02 = R(0.5) * (g2[2] + g2[6]), q12 = R(0.5) * (g2[5] + g2[7]);
        const R sdsd = ((d0 * d0 + d1 * d1) + d2 * d2) + R(2) * ((q01 * q01 + q02 * q02) + q12 * q12);
        const R cd = c * delta;
        const R rsd = wm_sqrt(sdsd), rss = wm_sqrt(ss);
        return cd * cd * (sdsd * rsd) / (ss * ss * rss + sdsd * wm_sqrt(rsd) + R(1e-30));
    }
    if (model == WM_SGS_VREMAN) {
        const R d2 = delta * delta;
        R b[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                b[3 * i + j] = d2 * (g[3 * i] * g[3 * j] + g[3 * i + 1] * g[3 * j + 1] + g[3 * i + 2] * g[3 * j + 2]);
        const R Bb = b[0] * b[4] - b[1] * b[1] + b[0] * b[8] - b[2] * b[2] + b[4] * b[8] - b[5] * b[5];
        R aa = R(0);
#pragma unroll
        for (int i = 0; i < 9; ++i) aa += g[i] * g[i];
        return R(2.5) * c * c * wm_sqrt(fmax(Bb, R(0)) / (aa + R(1e-30)));
    }
    return R(0);
}

// Ducros sensor, wmles/viscous.py:22-25
template <typename R>
__device__ __forceinline__ R ducros(const R g[9]) {
    const R div = g[0] + g[4] + g[8];
    const R a = g[7] - g[5], b = g[2] - g[6], c = g[3] - g[1];
    const R w2 = a * a + b * b + c * c;
    return div * div / (div * div + w2 + R(1e-30));
}

// ------------------------------------------------------------------ wall model (FP64)
// Spalding's law solved for u+ by safeguarded Newton, wmles/wall_model.py:19-40
// *moving is set when the iteration ends with an update larger than 1e-8 of the iterate
// (not settled within n_iter; the reference returns that iterate all the same)
__device__ __forceinline__ double spalding_utau(double kappa, double ekb, int n_iter, double h, double U,
                                                double rho_w, double mu_w, bool* moving) {
    const double Reh = h * U * rho_w / mu_w;
    // F has one root (dF > 0 everywhere), so that every start that settles ends at the same u+.  Over
    // Reh = 625, where the reference starts from 25 whatever the root, the logarithmic layer's estimate
    // (Reh = u+ y+ with u+ = 18) saves about four iterations.  Only where the reference's own start
    // settles, as its last iterate is the answer otherwise: from above the root an iteration lowers
    // kappa u+ by at most one, from 25 or, after an overshoot, 50 to 100, some 50 kappa iterations in all (29
    // at kappa = 0.6, counted over B and Reh); and where rounding leaves both starts at one u+ (ekb, the size
    // of F's terms over their sum near the wall, at most 100: B above -11 at kappa = 0.41)
    double up = fmin(fmax(sqrt(Reh), 1.0), 25.0);
    if (n_iter >= 30 && kappa > 0.0 && kappa <= 0.6 && ekb <= 100.0 && Reh > 625.0 && Reh < 1e12)
        up = fmin(fmax(log(Reh / (18.0 * ekb)) / kappa, 1.0), 100.0);
    double last = 0.0;
    *moving = false;
    for (int it = 0; it < n_iter; ++it) {
        const double ku = kappa * up;
        const double ex = exp(ku);
        const double g = ex - 1.0 - ku - 0.5 * ku * ku;
        // F / dF with both multiplied by u+^2: one division instead of three
        const double num = (up + ekb * (g - ku * ku * ku * (1.0 / 6.0))) * up - Reh;
        const double den = (1.0 + ekb * kappa * g) * (up * up) + Reh;
        const double next = fmin(fmax(up - num * up / den, 0.5 * up), 100.0);
        last = next - up;
        up = next;
        // settled: the iteration converges quadratically, so that after an update of 1e-9 the iterate is
        // the root to the last places (the relative error left is below (kappa u+ / 2) 1e-18); going on
        // would only move it among neighbouring doubles, for up to n_iter iterations of the whole warp
        if (fabs(last) <= 1e-9 * up) return U / up;
    }
    *moving = !(fabs(last) <= 1e-8 * up);
    return U / up;
}

}  // namespace wm
