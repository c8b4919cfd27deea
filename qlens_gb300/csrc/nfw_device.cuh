// nfw_device.cuh -- elliptical NFW deflection on the device by QLens's
// adaptive Gauss-Patterson quadrature, in FP64.
//
//   NFW::kappa_rsq, lens_function_xsq, kapavg_spherical_rsq   models.cpp:978-1010
//   q == 1: LensProfile::deflection_spherical_default         profile.cpp:1515-1518, 2281-2290
//   q <  1: LensProfile::deflection_numerical                 profile.cpp:2359-2375
//           alpha_x = x J_0, alpha_y = y J_1,
//           J_n = sqrt(1-eps) int_0^1 2w kappa(u (x^2 + y^2/(1-eps u)) q) / (1-eps u)^(n+1/2) dw,
//           u = w^2, eps = 1 - q^2 (LensIntegral, profile.h:441-449; profile.cpp:2703-2733, 2778-2783)
//   LensIntegral::PattersonIntegrate                          profile.cpp:3830-3876
//           levels of 1, 3, ..., 511 nested nodes; stop after level 2 once
//           |I_L - I_{L-1}| < 1e-3 |I_L| (QLens's default integral_tolerance)
//
// Both integrals share their nodes: each node's kappa is evaluated once and
// feeds J_0 and J_1, each of which keeps its own convergence test, so every
// level sum is the one the reference forms for that integral alone.  The sum
// of a level runs over the new nodes first, then the old ones, both in
// ascending order, as in the reference.  Node values of levels <= 5 (63
// nodes) are kept per thread; the rare rays that need levels 6-8 recompute
// the older values they lack, which gives the same bits (the arithmetic of a
// node is spelled out, so that no build contracts it otherwise).
//
// FP64 runs at 2 FMA a clock and SM and bounds this: a node's square roots,
// arc functions, logarithm and six divisions were ~190 operations.  kappa / ks is
// now a polynomial on the sixteenth of an octave that s = (xi/rs)^2 lies in
// (nfw_kappa_table.h: six FP64 terms, the rest below 1e-9 of the value in FP32;
// within 2.1e-16 of the exact value, where the closed form lost up to 1e-11 near
// s = 1 and 3e-16 elsewhere), and what depends on the lens only is tabulated by
// the kernels whose rays share it (NfwTab): 11 operations a node, 26 without the
// table (eight evaluations with a halo 30.6 -> 16.0 ms; 655,000 samples at 1e-10
// for the surrogate 95 -> 29).  Close to s = 1 and below 1e-6, where QLens switches to its own
// expansions, and outside the table the closed form is evaluated as before.
#pragma once
#include "qlpix_internal.h"
#include "patterson_rule.h"
#include "nfw_kappa_table.h"

namespace qlpix {

static __constant__ double c_pat_points[QLP_PAT_N] = QLP_PAT_POINTS_INIT;
static __constant__ double c_pat_weights[QLP_PAT_NW] = QLP_PAT_WEIGHTS_INIT;
static __device__ const __align__(16) double c_nfwk[QLP_NFWK_N * 6] = QLP_NFWK_C_INIT;
static __device__ const __align__(16) float c_nfwk32[QLP_NFWK_N * 4] = QLP_NFWK_F_INIT;

#define NFW_PAT_TOL 1e-3                 // QLens's default integral_tolerance (LensRec::tol)
#define NFW_KEEP_LEVELS 6            // levels 0..5 keep their node values
#define NFW_KEEP ((2 << (NFW_KEEP_LEVELS - 1)) - 1)   // 63

__device__ __forceinline__ double nfw_lens_function_xsq(double xsq)
{
    return ((xsq > 1.0) ? (atan(sqrt(xsq - 1)) / sqrt(xsq - 1))
                        : (xsq < 1.0) ? (atanh(sqrt(1 - xsq)) / sqrt(1 - xsq)) : 1.0);
}

__device__ __forceinline__ double nfw_kappa_rsq(double ks, double rs, double rsq)
{
    double xsq = rsq / (rs * rs);
    if (xsq < 1e-6) return -ks * (2 + log(xsq / 4));
    else if (fabs(xsq - 1) < 1e-5) return 2 * ks * (0.3333333333333333 - (xsq - 1) / 5.0);
    else return 2 * ks * (1 - nfw_lens_function_xsq(xsq)) / (xsq - 1);
}

__device__ __forceinline__ double nfw_kapavg_spherical_rsq(double ks, double rs, double rsq)
{
    double xsq = rsq / (rs * rs);
    if (xsq > 1e-5) return 2 * ks * (2 * nfw_lens_function_xsq(xsq) + log(xsq / 4)) / xsq;
    else return -ks * (1 + log(xsq / 4));
}

static __device__ __noinline__ double nfw_kappa_closed(double s) { return nfw_kappa_rsq(1.0, 1.0, s); }

// kappa / ks at s = (xi/rs)^2: interval and offset from the bits of s
__device__ __forceinline__ double nfw_kappa(double s)
{
    const int hi = __double2hiint(s);
    const unsigned lo = (unsigned)__double2loint(s);
    const unsigned k = (unsigned)(hi - ((1023 + QLP_NFWK_E0) << 20)) >> 16;
    // |s - 1| < 1e-5 lies in these high words; the first interval reaches below 1e-6
    if (k >= QLP_NFWK_N || (unsigned)(hi - 0x3fefffe8) <= 0x28u || (k == 0 && s < 1e-6)) return nfw_kappa_closed(s);
    const double t = __hiloint2double(0x3ff00000 | ((hi << 4) & 0xfffff) | (int)(lo >> 28), (int)(lo << 4)) - 1.5;
    const float tf = (float)(int)((((unsigned)hi << 16) | (lo >> 16)) ^ 0x80000000u) * 2.3283064365386963e-10f;
    const float4 f = __ldg(reinterpret_cast<const float4*>(c_nfwk32) + k);
    const double2* c = reinterpret_cast<const double2*>(c_nfwk) + 3 * k;
    const double2 c45 = __ldg(c + 2), c23 = __ldg(c + 1), c01 = __ldg(c);
    // to double by its bits (a zero becomes 2^-127)
    const int r = __float_as_int(__fmaf_rn(__fmaf_rn(f.z, tf, f.y), tf, f.x));
    double v = __hiloint2double((r & 0x80000000) | (((r & 0x7fffffff) >> 3) + (896 << 20)), r << 29);
    v = __fma_rn(v, t, c45.y);
    v = __fma_rn(v, t, c45.x);
    v = __fma_rn(v, t, c23.y);
    v = __fma_rn(v, t, c23.x);
    v = __fma_rn(v, t, c01.y);
    return __fma_rn(v, t, c01.x);
}

// What the integrands need of node i of the 511-point set: u q / rs^2,
// 1 / (1 - eps u) and 2 w / sqrt(1 - eps u).
__device__ __forceinline__ void nfw_node_lens(const LensRec& L, int i, double& uq, double& rq, double& c0)
{
    const double w = __fma_rn(0.5, c_pat_points[i], 0.5);
    const double u = __dmul_rn(w, w);
    const double qfac = __fma_rn(-L.epsilon, u, 1.0);
    const double y = rsqrt(qfac);
    const double r = __dmul_rn(y, y);
    rq = __fma_rn(r, __fma_rn(-qfac, r, 1.0), r);
    c0 = __dmul_rn(__dmul_rn(2.0, w), y);
    uq = __dmul_rn(u, __ddiv_rn(L.q, __dmul_rn(L.rs, L.rs)));
}

// The two integrands over ks at a node with these constants.
__device__ __forceinline__ void nfw_node(double xsq, double ysq, double uq, double rq, double c0, double& f0, double& f1)
{
    f0 = __dmul_rn(c0, nfw_kappa(__dmul_rn(__fma_rn(ysq, rq, xsq), uq)));
    f1 = __dmul_rn(f0, rq);
}

// nfw_node_lens of the nodes of levels <= 5 for one lens, by slot (i+1)/8 - 1
struct NfwTab { double uq[NFW_KEEP], rq[NFW_KEEP], c0[NFW_KEEP]; };

// Tables of a model's NFW lenses (any threads; a barrier before use).
__device__ __forceinline__ void nfw_tables(const LensModel& lm, NfwTab* tab)
{
    for (int e = threadIdx.x; e < lm.nlens * NFW_KEEP; e += blockDim.x) {
        const int k = e / NFW_KEEP, i = e - k * NFW_KEEP;
        const LensRec& L = lm.lens[k];
        if (L.type != QLP_LENS_SPLE && L.type != QLP_LENS_SHEAR && L.q != 1.0)
            nfw_node_lens(L, 8 * i + 7, tab[k].uq[i], tab[k].rq[i], tab[k].c0[i]);
    }
}

// The two Patterson integrals of LensIntegral::j_integral for lens-frame
// (x^2, y^2): I_n = 0.5 * sum_level(w_j f_n(node_j)) at the level where that
// integral converged to `tol` (QLens: 1e-3).  The deflection is
// alpha_x = x sqrt(1-eps) I_0, alpha_y = y sqrt(1-eps) I_1.  tab: the lens's
// table, or null.
static __device__ void nfw_integrals(const LensRec& L, double xsq, double ysq, double tol, double& I0, double& I1,
                                     const NfwTab* tab = nullptr)
{
    double keep0[NFW_KEEP], keep1[NFW_KEEP];   // values at nodes of levels <= 5, slot (i+1)/8 - 1
    double r0 = 0, r1 = 0, old0, old1;
    bool done0 = false, done1 = false;
    int level = 0;
    do {
        const double* wt = c_pat_weights + ((2 << level) - level - 2);   // levels 0..L-1 hold 2^(L+1)-2-L weights
        const int order = (2 << level) - 1;
        const int istep0 = (QLP_PAT_N + 1) / (order + 1);
        const int istep = 2 * istep0;
        old0 = r0; old1 = r1;
        double s0 = 0, s1 = 0;
        // new nodes (even j)
        for (int j = 0, i = istep0 - 1; j < order; j += 2, i += istep) {
            double f0, f1, uq, rq, c0;
            const int slot = ((i + 1) >> 3) - 1;
            if (tab && level < NFW_KEEP_LEVELS) { uq = tab->uq[slot]; rq = tab->rq[slot]; c0 = tab->c0[slot]; }
            else nfw_node_lens(L, i, uq, rq, c0);
            nfw_node(xsq, ysq, uq, rq, c0, f0, f1);
            if (level < NFW_KEEP_LEVELS) { keep0[slot] = f0; keep1[slot] = f1; }
            s0 = __fma_rn(wt[j], f0, s0);
            s1 = __fma_rn(wt[j], f1, s1);
        }
        // old nodes (odd j)
        for (int j = 1, i = istep - 1; j < order; j += 2, i += istep) {
            double f0, f1;
            if (((i + 1) & 7) == 0) { f0 = keep0[((i + 1) >> 3) - 1]; f1 = keep1[((i + 1) >> 3) - 1]; }
            else {
                double uq, rq, c0;
                nfw_node_lens(L, i, uq, rq, c0);
                nfw_node(xsq, ysq, uq, rq, c0, f0, f1);
            }
            s0 = __fma_rn(wt[j], f0, s0);
            s1 = __fma_rn(wt[j], f1, s1);
        }
        if (!done0) {
            r0 = s0;
            if ((level > 1) && (fabs(r0 - old0) < tol * fabs(r0))) done0 = true;
        }
        if (!done1) {
            r1 = s1;
            if ((level > 1) && (fabs(r1 - old1) < tol * fabs(r1))) done1 = true;
        }
    } while (++level < QLP_PAT_LEVELS && !(done0 && done1));
    I0 = L.ks * (0.5 * r0);
    I1 = L.ks * (0.5 * r1);
}

// The same two integrals for one ray per warp (all 32 lanes call it with the
// same arguments, converged): the lanes evaluate a level's new nodes in
// parallel into the warp's buffers v0, v1 (QLP_PAT_N doubles each, by node
// index), then every lane forms the level sums from the buffers in
// nfw_integrals' order.  The node values come from the same function and
// are added in the same order, so the result has nfw_integrals' bits, after
// about one node's latency per level instead of 2^level of them.
static __device__ void nfw_integrals_warp(const LensRec& L, double xsq, double ysq, double tol, double& I0,
                                          double& I1, double* v0, double* v1)
{
    const int lane = threadIdx.x & 31;
    double r0 = 0, r1 = 0, old0, old1;
    bool done0 = false, done1 = false;
    int level = 0;
    do {
        const double* wt = c_pat_weights + ((2 << level) - level - 2);
        const int order = (2 << level) - 1;
        const int istep0 = (QLP_PAT_N + 1) / (order + 1);
        const int istep = 2 * istep0;
        old0 = r0; old1 = r1;
        for (int q = lane; 2 * q < order; q += 32) {
            const int i = istep0 - 1 + q * istep;
            double f0, f1, uq, rq, c0;
            nfw_node_lens(L, i, uq, rq, c0);
            nfw_node(xsq, ysq, uq, rq, c0, f0, f1);
            v0[i] = f0;
            v1[i] = f1;
        }
        __syncwarp();
        double s0 = 0, s1 = 0;
        for (int j = 0, i = istep0 - 1; j < order; j += 2, i += istep) {
            s0 = __fma_rn(wt[j], v0[i], s0);
            s1 = __fma_rn(wt[j], v1[i], s1);
        }
        for (int j = 1, i = istep - 1; j < order; j += 2, i += istep) {
            s0 = __fma_rn(wt[j], v0[i], s0);
            s1 = __fma_rn(wt[j], v1[i], s1);
        }
        if (!done0) {
            r0 = s0;
            if ((level > 1) && (fabs(r0 - old0) < tol * fabs(r0))) done0 = true;
        }
        if (!done1) {
            r1 = s1;
            if ((level > 1) && (fabs(r1 - old1) < tol * fabs(r1))) done1 = true;
        }
        __syncwarp();
    } while (++level < QLP_PAT_LEVELS && !(done0 && done1));
    I0 = L.ks * (0.5 * r0);
    I1 = L.ks * (0.5 * r1);
}

// wbuf: null, or the calling warp's 2 QLP_PAT_N doubles for
// nfw_integrals_warp (then all 32 lanes call with the same arguments); tab:
// the lens's table, or null
static __device__ void nfw_deflection(const LensRec& L, double x, double y, double& dx, double& dy,
                                      double* wbuf = nullptr, const NfwTab* tab = nullptr)
{
    if (L.q == 1.0) {
        double kapavg = nfw_kapavg_spherical_rsq(L.ks, L.rs, x * x + y * y);
        dx = kapavg * x;
        dy = kapavg * y;
        return;
    }
    if ((fabs(x) < 1e-14) && (fabs(y) < 1e-14)) {
        dx = 0;
        dy = 0;
        return;
    }
    double I0, I1;
    if (wbuf) nfw_integrals_warp(L, x * x, y * y, L.tol, I0, I1, wbuf, wbuf + QLP_PAT_N);
    else nfw_integrals(L, x * x, y * y, L.tol, I0, I1, tab);
    const double sqe = sqrt(1 - L.epsilon);
    dx = x * (sqe * I0);
    dy = y * (sqe * I1);
}

}  // namespace qlpix
