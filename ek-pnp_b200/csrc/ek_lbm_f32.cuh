// ek_lbm_f32.cuh -- node update of the shifted-storage forms (FP32 and FP16
// populations, FP32 arithmetic).  Included by the single-channel kernels
// (ek_lbm_f32.cu) and the batched persistent kernel (ek_batch.cu).
//
// Storage: d_i = f_i - w_i*R with R = R_s(y) a per-row reference density of
// species s (fluid, c+, c-) at the row where the value is stored.  R_s(y) =
// 36 K 2^-q for integers K, so the change of frame when a population is pulled
// from row y' to row y, d += w_i (R_s(y') - R_s(y)) = (16|4|1) (K' - K) 2^-q, is
// exact in FP32; the profiles follow the fields' row means (set at
// initialisation, re-based on request).  Every quantity of the collision is
// rewritten in deviations so that FP32 keeps the small departures:
//   dens = R + sum_i d_i,  j = sum_i c_i d_i  (sum_i w_i c_i = 0)
//   deq_i = w_i*(d_dens + dens*A_i),  A_i = cu_i*(1 + cu_i/2) - u^2/(2 cs2)
//   TRT:  s = (d_i + d_ibar)/2, a = (d_i - d_ibar)/2,
//         out_i = d_i - w+ (s - seq) - w- (a - aeq), out_ibar = d_ibar - w+(..) + w-(..)
//   Guo source (LBM.cu:556-756) split as F+_i = w_i(-u.F/cs2 + cu_i cF_i),
//         F-_i = w_i cF_i,  cF_i = (c_i.F)/(cfl cs2),  src_i = sp F+_i + sm F-_i
// The physics, wall treatment and step order are those of the FP64 form
// (ek_lbm_f64.cu, which cites the reference lines); only the number format
// and the algebraic form of the collision differ.
//
// Arithmetic: FP32 throughout the collision.  Two places where plain FP32
// would keep a systematic error, and what this form does there:
//  * In the double layer the y-force is 1e3-1e4 times the x-force and the
//    diagonal populations carry both.  Sums such as g_x + g_y, or the
//    momentum (t5 + t8) - (t6 + t7), round the x-part at the scale of the
//    y-part, with the same rounding every step (a bias, not noise: u_x off by
//    3e-5 of its max and the plug velocity by 20% after 10,000 steps of the
//    4096 x 1024 channel).  So the diagonals collide in x/y-separated moments:
//    X = (t5 - t6) + (t8 - t7) (the two differences of values streamed from
//    one row are exact by Sterbenz), Y, the diagonal mass S and the xy-moment
//    Q relax separately and the x-force enters X alone; only the final
//    populations round at the scale of the y-part, once, as a store would.
//  * The ion anti-bounce-back wall (gpu_bc_charge, LBM.cu:908-1024) makes each
//    wall node an undamped period-2 oscillator: its density alternates
//    between rho_0 and 2 c_w - rho_0 (1 and 108 from the noisy start at
//    zeta = -4), so deviations from any fixed reference are large and their
//    rounding never decays.  The wall nodes' ion populations are therefore
//    kept against a per-x frame that alternates with the ping-pong buffer,
//    F_a ~ rho_0 and F_b ~ 2 c_w - F_a (both on the species' dyadic grid):
//    in these frames the anti-bounce-back is an exact reflection of the
//    deviations plus w_i (2 c_w - F_a - F_b), a sub-grid constant.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "ek_internal.h"

namespace ek {

// FP32 constants of one channel.
struct ChanF {
    int nx, ny, nxp, flags;
    size_t plane;                    // population and field plane size (elements)
    float wp, wm, wcp, wcm, wtp, wtm, sp, sm;
    float kcu;                       // 1/(cs2*cfl): cu_i = (c_i.u)*kcu
    float hinvcs2;                   // 0.5/cs2
    float inv_cfl, half_dt, dt;
    float gF;                        // 1/(cfl*cs2)
    float inv_cs2;
    float rho0, c0;
    float mob_p, mob_n;
    float ms, md;                    // moving top wall terms
    float f_chargef, ext_xf, exff;   // force F = f_charge (c+ - c-) (E + ext_x) + exf, FP32
    float cfl_hdt;                   // cfl dt/2: population momentum of the half force
    float srcF;                      // sm cfl dt: population momentum of the Guo source per unit F
    float half_inv_dxf, half_inv_dyf;  // E = (psi[-] - psi[+]) * (1/(2 dx))
    float rhs_qf;                    // -f_charge / eps: right-hand side per unit c+ - c-
    // FP64 set-up constants (initialisation; the zero mode of E_y)
    double f_charge, eps, ext_x, exf, dx, dy;
    double half_inv_dx, half_inv_dy;
    const double *zlo, *zhi, *cplo, *cphi, *cnlo, *cnhi;
    // field planes of the step (PoissonPlan::rhsf, psif, psim)
    float *rhsf;
    const float *psif;
    const double *psim;
    const float *lift;               // wall lifting's x-fluctuation (Chan::lift)
    const float *kref;               // per-row references / 36 (see Chan::kref)
    // Ion frames of the wall nodes (/36), per population buffer b (the
    // frame of the values stored in pops[b]), species s (0 c+, 1 c-), wall w
    // (0 lower, 1 upper): kwall[((b*2 + s)*2 + w)*nx + x]; and half the frame
    // defect (2 c_w - F_0 - F_1)/2 per (s, w, x): wdelta[(s*2 + w)*nx + x].
    const float *kwall;
    const float *wdelta;
    int keep_l2;                     // right-hand side stores ask L2 to keep the plane
};

__device__ __forceinline__ float kwall_at(const ChanF &k, int buf, int s, int w, int x) {
    return __ldg(k.kwall + ((size_t)((buf * 2 + s) * 2 + w)) * k.nx + x);
}
__device__ __forceinline__ float wdelta_at(const ChanF &k, int s, int w, int x) {
    return __ldg(k.wdelta + ((size_t)(s * 2 + w)) * k.nx + x);
}

template <typename S> __device__ __forceinline__ float ld_pop(const S *p);
template <> __device__ __forceinline__ float ld_pop<float>(const float *p) { return __ldg(p); }
template <> __device__ __forceinline__ float ld_pop<__half>(const __half *p) { return __half2float(__ldg(p)); }
template <typename S> __device__ __forceinline__ void st_pop(S *p, float v);
template <> __device__ __forceinline__ void st_pop<float>(float *p, float v) { *p = v; }
template <> __device__ __forceinline__ void st_pop<__half>(__half *p, float v) { *p = __float2half_rn(v); }

constexpr float W0F = 4.0f / 9.0f, WSF = 1.0f / 9.0f, WDF = 1.0f / 36.0f;

// ---- arithmetic of one node or of two neighbouring nodes -------------------
// V = float updates one node a thread, V = float2 the nodes x and x + 1 (x
// even) with the packed FP32 instructions of sm_100 (one issue slot for both).
// Every operation is an explicit round-to-nearest intrinsic, so that nothing
// is left to the compiler's choice of fused multiply-adds: the forms of the
// step (two nodes a thread, the batch, the TMA-fed one) give the same bits.
// No inexact product is an operand of vadd (vfma instead): packed, the sum of a
// product was seen to round once (ptxas 12.9), where the scalar one rounds twice.
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <typename V> __device__ __forceinline__ V bc(float v);
template <> __device__ __forceinline__ float bc<float>(float v) { return v; }
template <> __device__ __forceinline__ float2 bc<float2>(float v) { return make_float2(v, v); }
__device__ __forceinline__ float vrcp(float a) { return 1.0f / a; }
__device__ __forceinline__ float2 vrcp(float2 a) { return make_float2(1.0f / a.x, 1.0f / a.y); }
// a + k b, a k for a scalar k
template <typename V> __device__ __forceinline__ V vaxpy(float k, V b, V a) { return vfma(bc<V>(k), b, a); }
template <typename V> __device__ __forceinline__ V vscale(float k, V a) { return vmul(bc<V>(k), a); }

// Columns of a thread's nodes: x, and where its pulls and differences look --
// xm left of the first node, xr right of the first (the second node itself,
// or 0 where the second lies past the last column), xp right of the last.
struct Cols {
    int x, xm, xr, xp;
    bool two;  // the second node exists (nx odd: the last thread of a row has one)
};
template <typename V> __device__ __forceinline__ Cols make_cols(int x, int nx);
template <> __device__ __forceinline__ Cols make_cols<float>(int x, int nx) {
    const int xp = x + 1 == nx ? 0 : x + 1;
    return {x, x == 0 ? nx - 1 : x - 1, xp, xp, false};
}
template <> __device__ __forceinline__ Cols make_cols<float2>(int x, int nx) {
    return {x, x == 0 ? nx - 1 : x - 1, x + 1 == nx ? 0 : x + 1, x + 2 >= nx ? x + 2 - nx : x + 2, x + 1 < nx};
}

// Addresses: a plane's base pointer is the same for the whole block, and an
// element's byte offset inside a plane fits 32 bits for every channel this
// library takes (at most 8192 x 65535 elements of 8 bytes), so an access is a
// uniform 64-bit base plus a 32-bit offset.  Offsets of the four columns in a row:
struct RowAt {
    uint32_t x, xm, xr, xp;  // elements
};
__device__ __forceinline__ RowAt row_at(const Cols &c, int y, int nxp) {
    const uint32_t r = (uint32_t)y * (uint32_t)nxp;
    return {r + (uint32_t)c.x, r + (uint32_t)c.xm, r + (uint32_t)c.xr, r + (uint32_t)c.xp};
}
template <typename T> __device__ __forceinline__ T *at(T *base, uint32_t e) {
    return (T *)((char *)base + (size_t)(e * (uint32_t)sizeof(T)));
}
template <typename T> __device__ __forceinline__ const T *at(const T *base, uint32_t e) {
    return (const T *)((const char *)base + (size_t)(e * (uint32_t)sizeof(T)));
}

// Values of a plane's row at the thread's own columns (rows are
// padded to 16 or to a multiple of 32 elements and start 32-byte aligned, so the pair is one
// access), at their left neighbours and at their right ones.
template <typename V, typename S> struct Row;
template <typename S> struct Row<float, S> {
    static __device__ __forceinline__ float own(const S *p, const RowAt &r) { return ld_pop<S>(at(p, r.x)); }
    static __device__ __forceinline__ float left(const S *p, const RowAt &r) { return ld_pop<S>(at(p, r.xm)); }
    static __device__ __forceinline__ float right(const S *p, const RowAt &r) { return ld_pop<S>(at(p, r.xp)); }
    static __device__ __forceinline__ void put(S *p, const RowAt &r, float v) { st_pop<S>(at(p, r.x), v); }
};
__device__ __forceinline__ float2 ld_pair(const float *p) { return __ldg((const float2 *)p); }
__device__ __forceinline__ float2 ld_pair(const __half *p) { return __half22float2(__ldg((const __half2 *)p)); }
__device__ __forceinline__ void st_pair(float *p, float2 v) { *(float2 *)p = v; }
__device__ __forceinline__ void st_pair(__half *p, float2 v) { *(__half2 *)p = __float22half2_rn(v); }
template <typename S> struct Row<float2, S> {
    static __device__ __forceinline__ float2 own(const S *p, const RowAt &r) { return ld_pair(at(p, r.x)); }
    static __device__ __forceinline__ float2 left(const S *p, const RowAt &r) {
        return make_float2(ld_pop<S>(at(p, r.xm)), ld_pop<S>(at(p, r.x)));
    }
    static __device__ __forceinline__ float2 right(const S *p, const RowAt &r) {
        return make_float2(ld_pop<S>(at(p, r.xr)), ld_pop<S>(at(p, r.xp)));
    }
    static __device__ __forceinline__ void put(S *p, const RowAt &r, float2 v) { st_pair(at(p, r.x), v); }
};
// The same of psi's fluctuation plane, which the kernel before writes (ld_fresh).
template <typename V> struct PsiRow;
template <> struct PsiRow<float> {
    static __device__ __forceinline__ float own(const float *p, const RowAt &r) { return ld_fresh(at(p, r.x)); }
    static __device__ __forceinline__ float left(const float *p, const RowAt &r) { return ld_fresh(at(p, r.xm)); }
    static __device__ __forceinline__ float right(const float *p, const RowAt &r) { return ld_fresh(at(p, r.xp)); }
};
template <> struct PsiRow<float2> {
    static __device__ __forceinline__ float2 own(const float *p, const RowAt &r) { return ld_fresh((const float2 *)at(p, r.x)); }
    static __device__ __forceinline__ float2 left(const float *p, const RowAt &r) {
        return make_float2(ld_fresh(at(p, r.xm)), ld_fresh(at(p, r.x)));
    }
    static __device__ __forceinline__ float2 right(const float *p, const RowAt &r) {
        return make_float2(ld_fresh(at(p, r.xr)), ld_fresh(at(p, r.xp)));
    }
};
// Per-x arrays without padding (wall frames, lifting): element by element.
template <typename V> struct PerX;
template <> struct PerX<float> {
    static __device__ __forceinline__ float own(const float *a, const Cols &c) { return __ldg(a + c.x); }
    static __device__ __forceinline__ float left(const float *a, const Cols &c) { return __ldg(a + c.xm); }
    static __device__ __forceinline__ float right(const float *a, const Cols &c) { return __ldg(a + c.xp); }
};
template <> struct PerX<float2> {
    static __device__ __forceinline__ float2 own(const float *a, const Cols &c) {
        return make_float2(__ldg(a + c.x), __ldg(a + (c.two ? c.x + 1 : c.x)));
    }
    static __device__ __forceinline__ float2 left(const float *a, const Cols &c) {
        return make_float2(__ldg(a + c.xm), __ldg(a + c.x));
    }
    static __device__ __forceinline__ float2 right(const float *a, const Cols &c) {
        return make_float2(__ldg(a + c.xr), __ldg(a + c.xp));
    }
};
// Moments to a plane of doubles; ref: a reference density added in FP64.
__device__ __forceinline__ void st_moment(double *p, const Cols &, const RowAt &r, float ref, float v) {
    *at(p, r.x) = (double)ref + (double)v;
}
__device__ __forceinline__ void st_moment(double *p, const Cols &c, const RowAt &r, float2 ref, float2 v) {
    *at(p, r.x) = (double)ref.x + (double)v.x;
    if (c.two) *at(p, r.x + 1) = (double)ref.y + (double)v.y;
}
__device__ __forceinline__ float ld_f64(const double *p, const Cols &, const RowAt &r, float) { return (float)*at(p, r.x); }
__device__ __forceinline__ float2 ld_f64(const double *p, const Cols &c, const RowAt &r, float2) {
    return make_float2((float)*at(p, r.x), (float)*at(p, r.x + (c.two ? 1u : 0u)));
}
__device__ __forceinline__ void st_rhs(float *p, const RowAt &r, float v, bool keep) { st_field_f(at(p, r.x), v, keep); }
__device__ __forceinline__ void st_rhs(float *p, const RowAt &r, float2 v, bool keep) { st_field_f2(at(p, r.x), v, keep); }

template <typename V, typename S>
__device__ __forceinline__ void own9s(const S *__restrict__ b, size_t pl, const RowAt &r, V p[9]) {
#pragma unroll
    for (int d = 0; d < 9; ++d) p[d] = Row<V, S>::own(b + d * pl, r);
}

// Pull: direction d arrives from (x - cx_d, y - cy_d); r0, rm, rp: the row
// itself, the one below and the one above.
template <typename V, typename S>
__device__ __forceinline__ void pull9s(const S *__restrict__ b, size_t pl, const RowAt &r0, const RowAt &rm,
                                       const RowAt &rp, V p[9]) {
    using R = Row<V, S>;
    p[0] = R::own(b, r0);
    p[1] = R::left(b + 1 * pl, r0);
    p[2] = R::own(b + 2 * pl, rm);
    p[3] = R::right(b + 3 * pl, r0);
    p[4] = R::own(b + 4 * pl, rp);
    p[5] = R::left(b + 5 * pl, rm);
    p[6] = R::right(b + 6 * pl, rm);
    p[7] = R::right(b + 7 * pl, rp);
    p[8] = R::left(b + 8 * pl, rp);
}

// Change of frame of pulled populations to the puller's row reference:
// directions 2, 5, 6 came from row y-1 (dm = kref[y-1] - kref[y]), 4, 7, 8
// from row y+1 (dp = kref[y+1] - kref[y]); 36 w = 4 (straight), 1 (diagonal).
template <typename V> __device__ __forceinline__ void reframe_dn(V p[9], float dm) {
    p[2] = vadd(p[2], bc<V>(4.0f * dm));
    p[5] = vadd(p[5], bc<V>(dm));
    p[6] = vadd(p[6], bc<V>(dm));
}
template <typename V> __device__ __forceinline__ void reframe_up(V p[9], float dp) {
    p[4] = vadd(p[4], bc<V>(4.0f * dp));
    p[7] = vadd(p[7], bc<V>(dp));
    p[8] = vadd(p[8], bc<V>(dp));
}
template <typename V> __device__ __forceinline__ void reframe(V p[9], float dm, float dp) {
    reframe_dn(p, dm);
    reframe_up(p, dp);
}
// Pulls from a wall row, whose ion values sit in per-x frames kw(x'):
// lower wall (puller y = 1): 2 from x, 5 from x-1, 6 from x+1;
// upper wall (puller y = ny-2): 4 from x, 7 from x+1, 8 from x-1.
template <typename V> __device__ __forceinline__ void reframe_dn_wall(V p[9], const float *kw, const Cols &c, V k0) {
    p[2] = vaxpy(4.0f, vsub(PerX<V>::own(kw, c), k0), p[2]);
    p[5] = vadd(p[5], vsub(PerX<V>::left(kw, c), k0));
    p[6] = vadd(p[6], vsub(PerX<V>::right(kw, c), k0));
}
template <typename V> __device__ __forceinline__ void reframe_up_wall(V p[9], const float *kw, const Cols &c, V k0) {
    p[4] = vaxpy(4.0f, vsub(PerX<V>::own(kw, c), k0), p[4]);
    p[7] = vadd(p[7], vsub(PerX<V>::right(kw, c), k0));
    p[8] = vadd(p[8], vsub(PerX<V>::left(kw, c), k0));
}

// Ion anti-bounce-back in deviations: d_ibar = -q_i + 2 w_i (c_wall - R).
template <typename V> __device__ __forceinline__ V wall_reflect(float w2, V dcw, V q) {
    return vaxpy(w2, dcw, vscale(-1.0f, q));
}
template <typename V> __device__ __forceinline__ void ion_wall_dev(const V q[9], V dcw, V p[9]) {
    p[0] = wall_reflect(2.0f * W0F, dcw, q[0]);
    p[3] = wall_reflect(2.0f * WSF, dcw, q[1]);
    p[4] = wall_reflect(2.0f * WSF, dcw, q[2]);
    p[1] = wall_reflect(2.0f * WSF, dcw, q[3]);
    p[2] = wall_reflect(2.0f * WSF, dcw, q[4]);
    p[7] = wall_reflect(2.0f * WDF, dcw, q[5]);
    p[8] = wall_reflect(2.0f * WDF, dcw, q[6]);
    p[5] = wall_reflect(2.0f * WDF, dcw, q[7]);
    p[6] = wall_reflect(2.0f * WDF, dcw, q[8]);
}

// Moments with opposite directions paired first.  In the double layer the
// y-opposite populations carry large, nearly opposite parts (the force-
// balanced y-flux); adding those partners first cancels them exactly
// (Sterbenz), so the small remaining sums round at their own scale.
template <typename V> __device__ __forceinline__ V sum9f(const V t[9]) {
    return vadd(vadd(t[0], vadd(t[1], t[3])), vadd(vadd(t[2], t[4]), vadd(vadd(t[5], t[7]), vadd(t[6], t[8]))));
}
// x-momentum: t5 - t6 and t8 - t7 pair values streamed from one row (same
// y-part), so each difference is exact when the y-part dominates.
template <typename V> __device__ __forceinline__ V momx(const V t[9]) {
    return vadd(vsub(t[1], t[3]), vadd(vsub(t[5], t[6]), vsub(t[8], t[7])));
}
template <typename V> __device__ __forceinline__ V momy(const V t[9]) {
    return vadd(vsub(t[2], t[4]), vsub(vadd(t[5], t[6]), vadd(t[7], t[8])));
}

// v/36 by multiplication with the rounded 1/36: the momentum-carrying parts
// of the equilibria and of the force are built from these units times the
// exact integers 36 w = 4 (straight) or 1 (diagonal), so their momentum is
// dens*u (or F) up to the rounding of the unit; with the weights rounded to
// FP32 it would be off by a relative 7.4e-9 that the fluid, whose momentum is
// conserved, would gain step after step.
__device__ __forceinline__ float div36(float v) { return v * (1.0f / 36.0f); }

// TRT of one species in deviations, in place, FP32.  ux, uy: the species'
// advection velocity; usq_rest: u^2 of the rest equilibrium (the c- quirk of
// LBM.cu:493 passes the fluid's); FORCE adds the Guo source of (fx, fy) to the
// post-collision values (add_guo's split, LBM.cu:554-756).
// The diagonal pairs (5,7), (6,8) collide in the moments
//   S = d5 + d6 + d7 + d8  (mass)        Q = d5 - d6 + d7 - d8  (xy)
//   X = d5 - d6 - d7 + d8  (x-momentum)  Y = d5 + d6 - d7 - d8  (y-momentum)
// which the pair form's TRT maps linearly: S, Q relax with w+ to
//   S_eq = (base + dens (cx^2 + cy^2)/2)/9,  Q_eq = dens cx cy/9,
// X, Y with w- to their antisymmetric equilibria.
// Conserved quantities are split exactly rather than rebuilt from rounded
// weights: an equilibrium off by a fixed factor 1 + e (the rounding of 1/36,
// or of rho * (m / rho)) is what the relaxation restores every step, so the
// quantity would grow like (1 + e)^t (3e-5 of u_x after 10,000 steps).
//  * mass: the rest equilibrium is the remainder d_dens - sum of the others
//    (plus, for the c- quirk, its extra term), so the equilibria carry d_dens;
//  * fluid momentum (FLUID, P = the population momentum with the half force,
//    cfl rho u): the straight pair takes round(P/3) and the diagonal moment
//    the exact rest P - 2 round(P/3) (Sterbenz), summing to P exactly; the
//    force source sm cfl dt F is split the same way.
// Ions (not FLUID) relax their flux to 4 dens c/36 per pair unit: the ion
// flux is not conserved, so no factor accumulates.
// Pairs are carried doubled (d1 + d3, d1 - d3), which is exact.  Which sums take
// a product unrounded (vfma) is part of the form: runs repeat earlier ones bit
// for bit, FP16 storage too, whose rounding any other choice would scatter.
template <bool FORCE, bool FLUID, typename V>
__device__ __forceinline__ void trt_f32(V d[9], V ddens, V dens, V ux, V uy, bool rest_fluid, V usq_fluid, float wp,
                                        float wm, const ChanF &k, V fx, V fy, V px, V py) {
    const V vsq = vfma(ux, ux, vmul(uy, uy));
    const V base = vfma(vscale(-k.hinvcs2, vsq), dens, ddens);
    const V cx = vscale(k.kcu, ux), cy = vscale(k.kcu, uy);
    // symmetric equilibria: straight pairs, diagonal mass (z / 9) and xy (q9 / 9)
    // moments, rest remainder
    const V seq13 = vscale(WSF, vfma(dens, vmul(vscale(0.5f, cx), cx), base));
    const V seq24 = vscale(WSF, vfma(dens, vmul(vscale(0.5f, cy), cy), base));
    const V z = vfma(dens, vscale(0.5f, vfma(cx, cx, vmul(cy, cy))), base);
    const V q9 = vmul(dens, vmul(cx, cy));
    V e0 = vsub(ddens, vaxpy(1.0f / 9.0f, z, vaxpy(2.0f, seq13, vscale(2.0f, seq24))));
    if (rest_fluid) e0 = vfma(vscale(W0F, dens), vscale(k.hinvcs2, vsub(vsq, usq_fluid)), e0);
    // antisymmetric equilibria (half-pair units: a13 = (d1 - d3)/2, X = d5 - d6 - d7 + d8)
    V aq13, aqx, aq24, aqy;
    if (FLUID) {
        aq13 = vscale(1.0f / 3.0f, px);
        aqx = vaxpy(-2.0f, aq13, px);
        aq24 = vscale(1.0f / 3.0f, py);
        aqy = vaxpy(-2.0f, aq24, py);
    } else {
        aq13 = aqx = vscale(1.0f / 9.0f, vmul(dens, cx));
        aq24 = aqy = vscale(1.0f / 9.0f, vmul(dens, cy));
    }
    const V nwp = bc<V>(-wp), nwm = bc<V>(-wm);
    V d0 = vfma(nwp, vsub(d[0], e0), d[0]);
    V s13 = vadd(d[1], d[3]), a13 = vsub(d[1], d[3]);
    V s24 = vadd(d[2], d[4]), a24 = vsub(d[2], d[4]);
    s13 = vfma(nwp, vaxpy(-2.0f, seq13, s13), s13);
    a13 = vfma(nwm, vaxpy(-2.0f, aq13, a13), a13);
    s24 = vfma(nwp, vaxpy(-2.0f, seq24, s24), s24);
    a24 = vfma(nwm, vaxpy(-2.0f, aq24, a24), a24);
    const V A = vsub(d[5], d[6]), B = vsub(d[8], d[7]);  // x-differences of values from one row
    const V C = vadd(d[5], d[6]), D = vadd(d[7], d[8]);
    V X = vadd(A, B), Q = vsub(A, B), Y = vsub(C, D), S = vadd(C, D);
    S = vfma(nwp, vaxpy(-1.0f / 9.0f, z, S), S);
    Q = vfma(nwp, vaxpy(-1.0f / 9.0f, q9, Q), Q);
    X = vfma(nwm, vsub(X, aqx), X);
    Y = vfma(nwm, vsub(Y, aqy), Y);
    if (FORCE) {
        const V uF = vscale(k.inv_cs2, vfma(ux, fx, vmul(uy, fy)));
        const V cfx = vscale(k.gF, fx), cfy = vscale(k.gF, fy);
        const float sp = k.sp * k.dt;
        // symmetric (mass-free) part: the rest takes the remainder
        const V g13 = vscale(sp, vscale(WSF, vfma(cx, cfx, vscale(-1.0f, uF))));
        const V g24 = vscale(sp, vscale(WSF, vfma(cy, cfy, vscale(-1.0f, uF))));
        const V ws = vscale(1.0f / 9.0f, vsub(vfma(cx, cfx, vmul(cy, cfy)), uF));
        const V wq = vscale(1.0f / 9.0f, vfma(cx, cfy, vmul(cy, cfx)));
        d0 = vsub(d0, vaxpy(sp, ws, vaxpy(2.0f, g13, vscale(2.0f, g24))));
        s13 = vaxpy(2.0f, g13, s13);
        s24 = vaxpy(2.0f, g24, s24);
        S = vaxpy(sp, ws, S);
        Q = vaxpy(sp, wq, Q);
        // momentum: sm cfl dt F, a third to each straight half-pair unit
        const V fsx = vscale(k.srcF, fx), fsy = vscale(k.srcF, fy);
        const V q13 = vscale(1.0f / 3.0f, fsx), q24 = vscale(1.0f / 3.0f, fsy);
        a13 = vaxpy(2.0f, q13, a13);
        a24 = vaxpy(2.0f, q24, a24);
        X = vadd(X, vaxpy(-2.0f, q13, fsx));
        Y = vadd(Y, vaxpy(-2.0f, q24, fsy));
    }
    const V h13 = vscale(0.5f, s13), h24 = vscale(0.5f, s24);
    const V P = vscale(0.25f, vadd(S, Y)), M = vscale(0.25f, vsub(S, Y)), U = vadd(Q, X), W = vsub(Q, X);
    d[0] = d0;
    d[1] = vaxpy(0.5f, a13, h13);
    d[3] = vaxpy(-0.5f, a13, h13);
    d[2] = vaxpy(0.5f, a24, h24);
    d[4] = vaxpy(-0.5f, a24, h24);
    d[5] = vaxpy(0.25f, U, P);
    d[6] = vaxpy(-0.25f, U, P);
    d[7] = vaxpy(0.25f, W, M);
    d[8] = vaxpy(-0.25f, W, M);
}

// Central-difference E of the shifted forms (the stencil of gpu_efield and
// gpu_bc, poisson.cu:145-174: wall rows take the adjacent row's Ey), with
// the 1/(2 dx), 1/(2 dy) factors precomputed: a multiply in place of an
// FP64 division per component.
__device__ __forceinline__ void efield_shifted(const ChanF &k, const double *__restrict__ psi, int x, int y, int xm,
                                               int xp, double *ex, double *ey) {
    const size_t r = (size_t)y * k.nxp;
    *ex = (__ldg(psi + r + xm) - __ldg(psi + r + xp)) * k.half_inv_dx;
    const int yc = y == 0 ? 1 : (y == k.ny - 1 ? k.ny - 2 : y);
    *ey = (__ldg(psi + (size_t)(yc - 1) * k.nxp + x) - __ldg(psi + (size_t)(yc + 1) * k.nxp + x)) * k.half_inv_dy;
}

// E of the step from psi = psim (row means, FP64) + psif (FP32): Ex from the
// FP32 fluctuations alone, Ey from the FP64 difference of the two row means
// (the zero mode, rounded once) plus that of the fluctuations.  Stencil of
// gpu_efield / gpu_bc (poisson.cu:145-174).
template <typename V>
__device__ __forceinline__ void efield_f32(const ChanF &k, const Cols &c, int y, V *ex, V *ex_tot, V *ey) {
    using R = PsiRow<V>;
    const RowAt r = row_at(c, y, k.nxp);
    const V dx = vsub(R::left(k.psif, r), R::right(k.psif, r));
    *ex = vscale(k.half_inv_dxf, dx);
    *ex_tot = vaxpy(k.half_inv_dxf, dx, bc<V>(k.ext_xf));
    const int yc = y == 0 ? 1 : (y == k.ny - 1 ? k.ny - 2 : y);
    const float eym = (float)((ld_fresh(k.psim + yc - 1) - ld_fresh(k.psim + yc + 1)) * k.half_inv_dy);
    const V dn = R::own(k.psif, row_at(c, yc - 1, k.nxp)), up = R::own(k.psif, row_at(c, yc + 1, k.nxp));
    *ey = vaxpy(k.half_inv_dyf, vsub(dn, up), bc<V>(eym));
}

// One step of a thread's node or pair of nodes.  src/dst: 27 population
// planes (species-major); fields: the channel's 9 FP64 field planes.
// Raw populations, as stored: FIRST -> the nodes' own (pre-collision) values;
// otherwise the fluid pulled from the neighbours and the ions pulled (interior
// rows) or the nodes' own values (wall rows).
template <typename S, bool FIRST, typename V>
__device__ __forceinline__ void gather_global(const ChanF &k, const S *__restrict__ src, const Cols &c, int y, V f[9],
                                              V h[9], V t[9]) {
    const size_t pl = k.plane;
    const RowAt r0 = row_at(c, y, k.nxp);
    const S *sf = src, *sh = src + 9 * pl, *st = src + 18 * pl;
    if (FIRST) {
        own9s<V, S>(sf, pl, r0, f);
        own9s<V, S>(sh, pl, r0, h);
        own9s<V, S>(st, pl, r0, t);
    } else {
        const RowAt rm = row_at(c, y == 0 ? k.ny - 1 : y - 1, k.nxp), rp = row_at(c, y + 1 == k.ny ? 0 : y + 1, k.nxp);
        pull9s<V, S>(sf, pl, r0, rm, rp, f);
        if (y == 0 || y == k.ny - 1) {
            own9s<V, S>(sh, pl, r0, h);
            own9s<V, S>(st, pl, r0, t);
        } else {
            pull9s<V, S>(sh, pl, r0, rm, rp, h);
            pull9s<V, S>(st, pl, r0, rm, rp, t);
        }
    }
}

// Collision, walls and stores of a thread's nodes from their raw populations
// (see gather_global); src is read only for the lower wall's row-1 pull.
// sbuf: index (0/1) of the population buffer that src is, which names the wall
// nodes' ion frames of the values read (sbuf) and written (sbuf ^ 1).
// `moments` is a run-time flag, so that every step's arithmetic is independent
// of how the steps are split into calls.
template <typename S, bool FIRST, bool EXPLICIT_E, typename V>
__device__ __forceinline__ void collide_shifted(const ChanF &k, V f[9], V h[9], V t[9], const S *__restrict__ src,
                                                S *__restrict__ dst, double *__restrict__ fields, const Cols &c, int y,
                                                bool moments, int sbuf) {
    using R = Row<V, S>;
    const size_t pl = k.plane;
    const int nxp = k.nxp, ny = k.ny;
    const RowAt r0 = row_at(c, y, nxp);
    const bool lo = y == 0, hi = y == ny - 1, wall = lo || hi;
    const int ym = y == 0 ? ny - 1 : y - 1, yp = y + 1 == ny ? 0 : y + 1;
    const int nx = k.nx;
    // frames (/36) of these nodes' values: the fluid and interior ions use the
    // row references, the wall nodes' ions the per-x frame of the output buffer
    const float kf0 = __ldg(k.kref + y);
    auto kw = [&](int buf, int s, int w) { return k.kwall + (size_t)((buf * 2 + s) * 2 + w) * nx; };
    V kh0, kt0;
    if (wall) {
        const int w = lo ? 0 : 1;
        kh0 = PerX<V>::own(kw(sbuf ^ 1, 0, w), c);
        kt0 = PerX<V>::own(kw(sbuf ^ 1, 1, w), c);
    } else {
        kh0 = bc<V>(__ldg(k.kref + ny + y));
        kt0 = bc<V>(__ldg(k.kref + 2 * ny + y));
    }
    const float Rf = 36.0f * kf0;
    const V Rh = vscale(36.0f, kh0), Rt = vscale(36.0f, kt0);  // exact: 36 K 2^-q < 2^22 2^-q
    if (!FIRST) reframe(f, __ldg(k.kref + ym) - kf0, __ldg(k.kref + yp) - kf0);
    if (wall) {
        // anti-bounce-back (gpu_bc_charge) from the stored frame into the
        // other: an exact reflection plus w_i times the frame defect; the
        // first step too, whose stored values init_node_shifted reflected
        const int w = lo ? 0 : 1;
        V q[9];
#pragma unroll
        for (int d = 0; d < 9; ++d) q[d] = h[d];
        ion_wall_dev(q, PerX<V>::own(k.wdelta + (size_t)w * nx, c), h);
#pragma unroll
        for (int d = 0; d < 9; ++d) q[d] = t[d];
        ion_wall_dev(q, PerX<V>::own(k.wdelta + (size_t)(2 + w) * nx, c), t);
    } else if (!FIRST) {
        if (y == 1) {
            reframe_dn_wall(h, kw(sbuf, 0, 0), c, kh0);
            reframe_dn_wall(t, kw(sbuf, 1, 0), c, kt0);
        } else {
            reframe_dn(h, __ldg(k.kref + ny + ym) - __ldg(k.kref + ny + y));
            reframe_dn(t, __ldg(k.kref + 2 * ny + ym) - __ldg(k.kref + 2 * ny + y));
        }
        if (y == ny - 2) {
            reframe_up_wall(h, kw(sbuf, 0, 1), c, kh0);
            reframe_up_wall(t, kw(sbuf, 1, 1), c, kt0);
        } else {
            reframe_up(h, __ldg(k.kref + ny + yp) - __ldg(k.kref + ny + y));
            reframe_up(t, __ldg(k.kref + 2 * ny + yp) - __ldg(k.kref + 2 * ny + y));
        }
    }
    const V drho = sum9f(f), dcp = sum9f(h), dcn = sum9f(t);
    const V rho = vadd(bc<V>(Rf), drho);
    V ex, ex_tot, ey;  // ex_tot: with the applied field
    if (EXPLICIT_E) {
        ex = ld_f64(fields + F_EX * pl, c, r0, V{});
        ey = ld_f64(fields + F_EY * pl, c, r0, V{});
        ex_tot = vadd(ex, bc<V>(k.ext_xf));
    } else {
        efield_f32<V>(k, c, y, &ex, &ex_tot, &ey);
    }
    V fx = bc<V>(0.0f), fy = bc<V>(0.0f);
    const V dq = vsub(dcp, dcn);
    const bool force = (k.flags & EK_FLAG_FORCE) != 0;
    if (force) {
        const V q = vscale(k.f_chargef, vadd(vsub(Rh, Rt), dq));  // f_charge (c+ - c-)
        fx = vfma(q, ex_tot, bc<V>(k.exff));
        fy = vmul(q, ey);
    }
    const V rrho = vrcp(rho);
    const V mx = momx(f), my = momy(f);
    V ux = vmul(vaxpy(k.half_dt, fx, vscale(k.inv_cfl, mx)), rrho);
    V uy = vmul(vaxpy(k.half_dt, fy, vscale(k.inv_cfl, my)), rrho);
    if (lo) {
        V m[9];
        const float kf1 = __ldg(k.kref + 1);
        if (FIRST) {
            own9s<V, S>(src, pl, row_at(c, 1, nxp), m);
        } else {
            pull9s<V, S>(src, pl, row_at(c, 1, nxp), r0, row_at(c, 2, nxp), m);
            reframe(m, __ldg(k.kref + 0) - kf1, __ldg(k.kref + 2) - kf1);
        }
        const V rrho1 = vrcp(vadd(bc<V>(36.0f * kf1), sum9f(m)));
        ux = vmul(vaxpy(-k.half_dt, fx, vscale(-k.inv_cfl, momx(m))), rrho1);
        uy = vmul(vaxpy(-k.half_dt, fy, vscale(-k.inv_cfl, momy(m))), rrho1);
    }
    if (moments) {
        const V none = bc<V>(0.0f);
        st_moment(fields + F_RHO * pl, c, r0, bc<V>(Rf), drho);
        st_moment(fields + F_UX * pl, c, r0, none, ux);
        st_moment(fields + F_UY * pl, c, r0, none, uy);
        st_moment(fields + F_CP * pl, c, r0, Rh, dcp);
        st_moment(fields + F_CN * pl, c, r0, Rt, dcn);
    }
    // right-hand side without its FP64 row constant (rhs_q (R+ - R-) and the
    // lifting's x-mean, added by the row pass), with the lifting's x-fluctuation
    if (!wall) {
        V v = vscale(k.rhs_qf, dq);
        if (y == 1) v = vsub(v, PerX<V>::own(k.lift, c));
        if (y == ny - 2) v = vsub(v, PerX<V>::own(k.lift + nx, c));
        st_rhs(k.rhsf, r0, v, k.keep_l2);
    }
    // ions: FP32 TRT, moment form (trt_f32)
    const V zero = bc<V>(0.0f);
    const V usq = vfma(ux, ux, vmul(uy, uy));
    trt_f32<false, false>(h, dcp, vadd(Rh, dcp), vaxpy(k.mob_p, ex, ux), vaxpy(k.mob_p, ey, uy), false, usq, k.wcp, k.wcm,
                          k, zero, zero, zero, zero);
#pragma unroll
    for (int d = 0; d < 9; ++d) R::put(dst + (9 + d) * pl, r0, h[d]);
    // c-: the quirk of LBM.cu:493, its rest equilibrium with the fluid's u^2
    trt_f32<false, false>(t, dcn, vadd(Rt, dcn), vaxpy(k.mob_n, ex, ux), vaxpy(k.mob_n, ey, uy),
                          (k.flags & EK_FLAG_REST_QUIRK) != 0, usq, k.wtp, k.wtm, k, zero, zero, zero, zero);
#pragma unroll
    for (int d = 0; d < 9; ++d) R::put(dst + (18 + d) * pl, r0, t[d]);
    S *df = dst;
    if (lo) {
        R::put(df, r0, f[0]);
#pragma unroll
        for (int d = 1; d < 9; ++d) R::put(df + oppd(d) * pl, r0, f[d]);
        return;
    }
    if (hi) {
        const V ms = bc<V>(k.ms), md = bc<V>(k.md);
        R::put(df, r0, f[0]);
        R::put(df + 3 * pl, r0, vsub(f[1], ms));
        R::put(df + 4 * pl, r0, f[2]);
        R::put(df + 1 * pl, r0, vadd(f[3], ms));
        R::put(df + 2 * pl, r0, f[4]);
        R::put(df + 7 * pl, r0, vsub(f[5], md));
        R::put(df + 8 * pl, r0, vadd(f[6], md));
        R::put(df + 5 * pl, r0, vadd(f[7], md));
        R::put(df + 6 * pl, r0, vsub(f[8], md));
        return;
    }
    // fluid: FP32 TRT with the Guo source, moment form (trt_f32); the
    // population momentum with the half force, cfl rho u
    const V px = vaxpy(k.cfl_hdt, fx, mx), py = vaxpy(k.cfl_hdt, fy, my);
    if (force)
        trt_f32<true, true>(f, drho, rho, ux, uy, false, usq, k.wp, k.wm, k, fx, fy, px, py);
    else
        trt_f32<false, true>(f, drho, rho, ux, uy, false, usq, k.wp, k.wm, k, zero, zero, px, py);
#pragma unroll
    for (int d = 0; d < 9; ++d) R::put(df + d * pl, r0, f[d]);
}

// The step of the node x, or of the nodes x and x + 1 (V = float2, x even).
template <typename S, bool FIRST, bool EXPLICIT_E, typename V>
__device__ __forceinline__ void node_shifted(const ChanF &k, const S *__restrict__ src, S *__restrict__ dst,
                                             double *__restrict__ fields, int x, int y, bool moments, int sbuf,
                                             bool wait) {
    const Cols c = make_cols<V>(x, k.nx);
    V f[9], h[9], t[9];
    gather_global<S, FIRST, V>(k, src, c, y, f, h, t);
    if (wait) pdl_wait();  // the populations are in flight; psi comes from the kernel before (StepChain)
    collide_shifted<S, FIRST, EXPLICIT_E, V>(k, f, h, t, src, dst, fields, c, y, moments, sbuf);
}

// Equilibrium deviations from the fields (pre-collision layout), written to
// population buffer `buf`.  The wall nodes' ions are stored reflected
// (anti-bounce-back from their frame in buf ^ 1 into the one of buf), since
// every step, the first included, reflects them on load.
template <typename S>
__device__ __forceinline__ void init_node_shifted(const ChanF &k, S *__restrict__ pops, const double *__restrict__ fields,
                                                  bool explicit_e, int x, int y, int buf) {
    const size_t pl = k.plane, o = (size_t)y * k.nxp + x;
    const int xm = x == 0 ? k.nx - 1 : x - 1, xp = x + 1 == k.nx ? 0 : x + 1;
    double exd, eyd;
    if (explicit_e) {
        exd = fields[F_EX * pl + o];
        eyd = fields[F_EY * pl + o];
    } else {
        efield_shifted(k, fields + F_PSI * pl, x, y, xm, xp, &exd, &eyd);
    }
    const float Ex = (float)exd, Ey = (float)eyd;
    const float ux = (float)fields[F_UX * pl + o], uy = (float)fields[F_UY * pl + o];
    const double densd[3] = {fields[F_RHO * pl + o], fields[F_CP * pl + o], fields[F_CN * pl + o]};
    const float dens[3] = {(float)densd[0], (float)densd[1], (float)densd[2]};
    const float mob[3] = {0.0f, k.mob_p, k.mob_n};
    const bool wall = y == 0 || y == k.ny - 1;
    const int w = y == 0 ? 0 : 1;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const float vx = ux + mob[s] * Ex, vy = uy + mob[s] * Ey;
        const float usq = k.hinvcs2 * (vx * vx + vy * vy);
        const bool wion = wall && s > 0;
        const float kframe = wion ? kwall_at(k, buf ^ 1, s - 1, w, x) : __ldg(k.kref + s * k.ny + y);
        const float dd = (float)(densd[s] - 36.0 * (double)kframe);
        const float base = dd - dens[s] * usq;
        const float cx = vx * k.kcu, cy = vy * k.kcu;
        const float ax = div36(dens[s] * cx), ay = div36(dens[s] * cy);
        float e[9];
        e[0] = W0F * base;
        const float cu[4] = {cx, cy, cx + cy, cy - cx};
        const float an[4] = {4.0f * ax, 4.0f * ay, ax + ay, ay - ax};
        const int ia[4] = {1, 2, 5, 6};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float w = q < 2 ? WSF : WDF;
            const float sym = w * (base + dens[s] * 0.5f * cu[q] * cu[q]);
            const float anti = an[q];
            e[ia[q]] = sym + anti;
            e[oppd(ia[q])] = sym - anti;
        }
        if (wion) {
            float r[9];
            ion_wall_dev(e, wdelta_at(k, s - 1, w, x), r);
#pragma unroll
            for (int d = 0; d < 9; ++d) e[d] = r[d];
        }
#pragma unroll
        for (int d = 0; d < 9; ++d) st_pop<S>(pops + (s * 9 + d) * pl + o, e[d]);
    }
}

// Wall frames of the ions at initialisation, one thread per (species s, wall
// w, x): F_a = the wall node's density on the species' grid (the frame of the
// state after the first step, buffer buf ^ 1), F_b = 2 c_w - F_a on the same
// grid (buffer buf, where the reflected initial values go), and half the
// defect (2 c_w - F_a - F_b)/2.  FP64 here: set-up, not the step.
__device__ __forceinline__ void wall_frames_dev(const ChanF &k, const double *__restrict__ fields, int qp, int qn, int buf,
                                                float *__restrict__ kwall, float *__restrict__ wdelta, int i) {
    const int x = i % k.nx, sw = i / k.nx, s = sw >> 1, w = sw & 1;
    const int y = w ? k.ny - 1 : 0;
    const double dens = fields[(s ? F_CN : F_CP) * k.plane + (size_t)y * k.nxp + x];
    const double cw = s ? (w ? k.cnhi[x] : k.cnlo[x]) : (w ? k.cphi[x] : k.cplo[x]);
    const double g = ldexp(1.0, s ? qn : qp);
    const double fa = ldexp(rint(dens / 36.0 * g), -(s ? qn : qp));      // /36
    const double fb = ldexp(rint((2.0 * cw / 36.0 - fa) * g), -(s ? qn : qp));
    kwall[((size_t)(((buf ^ 1) * 2 + s) * 2 + w)) * k.nx + x] = (float)fa;
    kwall[((size_t)((buf * 2 + s) * 2 + w)) * k.nx + x] = (float)fb;
    wdelta[(size_t)(s * 2 + w) * k.nx + x] = (float)(cw - 18.0 * (fa + fb));
}

// Half the frame defect after the wall concentrations change (per-x walls set
// after initialisation): the frames stay, the defect follows c_w.
__device__ __forceinline__ void wall_delta_dev(const ChanF &k, const float *__restrict__ kwall, float *__restrict__ wdelta,
                                               int i) {
    const int x = i % k.nx, sw = i / k.nx, s = sw >> 1, w = sw & 1;
    const double cw = s ? (w ? k.cnhi[x] : k.cnlo[x]) : (w ? k.cphi[x] : k.cplo[x]);
    const double f0 = kwall[((size_t)((0 * 2 + s) * 2 + w)) * k.nx + x];
    const double f1 = kwall[((size_t)((1 * 2 + s) * 2 + w)) * k.nx + x];
    wdelta[(size_t)(s * 2 + w) * k.nx + x] = (float)(cw - 18.0 * (f0 + f1));
}

// Row y's means of rho, c+, c- rounded to the reference grids K 2^-q (stored
// /36), FP64 sums; a block of 256 threads per row, kout[s*ny + y].
__device__ __forceinline__ void row_refs_dev(int nx, int nxp, int ny, size_t plane, const double *__restrict__ fields,
                                             int qf, int qp, int qn, float *__restrict__ kout, int y) {
    double acc[3] = {0.0, 0.0, 0.0};
    const size_t r = (size_t)y * nxp;
    for (int x = threadIdx.x; x < nx; x += blockDim.x) {
        acc[0] += fields[F_RHO * plane + r + x];
        acc[1] += fields[F_CP * plane + r + x];
        acc[2] += fields[F_CN * plane + r + x];
    }
    __shared__ double red[8][3];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        double v = acc[s];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][s] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += red[w][threadIdx.x];
        const int q = threadIdx.x == 0 ? qf : (threadIdx.x == 1 ? qp : qn);
        const double mean = v / (double)nx;
        const double K = rint(mean / 36.0 * ldexp(1.0, q));
        kout[threadIdx.x * ny + y] = (float)ldexp(K, -q);
    }
}

// Re-basing of one stored value of plane (species s, direction d) at row y:
// d += 36 w_d (kold - knew), exact in FP32.
template <typename S>
__device__ __forceinline__ void rebase_dev(S *p, int plane_idx, int ny, int y, const float *__restrict__ kold,
                                           const float *__restrict__ knew) {
    const int s = plane_idx / 9, d = plane_idx - 9 * s;
    if (s > 0 && (y == 0 || y == ny - 1)) return;  // wall ions keep their per-x frames
    const float wint = d == 0 ? 16.0f : (d < 5 ? 4.0f : 1.0f);
    const float corr = wint * (kold[s * ny + y] - knew[s * ny + y]);
    st_pop<S>(p, ld_pop<S>(p) + corr);
}

ChanF make_chanf(const Chan &c);

}  // namespace ek
