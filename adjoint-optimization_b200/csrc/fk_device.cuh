// fk_device.cuh -- device-side Fenton-Karma model for sm_100a.
//
// Data layout in HBM (every state, adjoint state and trajectory slot):
//   three planes u, v, w of a padded grid, plane = rows_alloc * ld doubles,
//   logical cell (i, j) at offset (i + HALO) * ld + (j + HALO);
//   a ring of HALO NaN cells surrounds the grid and holes hold NaN.
// With a NaN ring the reference's edge rule (mirror the inner neighbour,
// src/cuda/fk_forward_Et_mono_PARAMETERS.cu:319-361) and its hole rule (a NaN
// neighbour is replaced by the opposite one, :348-358) are the same rule, and
// the adjoint stencil's off-grid and hole cases coincide too, so the kernels
// have no boundary branches and tile loads never leave the allocation.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace fkadj {

constexpr int HALO = 4;

// Model constants as the kernels use them: reciprocals replace the divisions
// by constant time scales of the reference's F_ion / jacT (cu-F:29-45,
// cu-G:1160-1184); this moves results by at most an ulp per operation.
struct DevModel {
    double u_c, u_csi;
    // slopes of the smoothed steps in units of 2^(1/16): e^{-2 k d} =
    // 2^(s d / 16) with s = -2 k 16 / ln2, high and low parts
    double sp_h, sp_l;  // p step (k = ksm)
    double ss_h, ss_l;  // slow inward current (k = k_fk)
    double r_tau_d, r_tau_0, r_tau_r, r_tau_si;
    double tau_v1m, tau_v2m, r_tau_vp, r_tau_wm, r_tau_wp;
    double eq;          // exp(-2 ksm (u_c - u_v)): e^{-2ksm(u-u_v)} = eq * e^{-2ksm(u-u_c)}
    double cu, cv, cw;  // D / h^2
    double dt;
    double dt_6, dt_3;  // dt / 6, dt / 3: a division in the kernels is a subroutine
    // constant factors of the Jacobian (fk_jacT)
    double two_ksm;       // 2 ksm: dp/du = 2 ksm p (1 - p)
    double kfk2_rsi;      // 2 k_fk / tau_si
    double two_ksm_dv12;  // 2 ksm (tau_v2- - tau_v1-)
};

struct DevGrid {
    int nrows, ncols, ld, rows_alloc;
    long long plane;  // doubles per field plane
};

// Refinement of the reciprocal estimate (own_rcp):
//   0: two Newton-Raphson steps r <- r + r (1 - x r), each squaring the
//      relative error (4 DFMA);
//   1: one third-order step r <- r (1 + e + e^2), e = 1 - x r, which cubes it
//      (3 DFMA): 1/x = r / (1 - e) = r (1 + e + e^2 + e^3 + ...).
// Both are within one ulp of the quotient; 1 (the default) took the forward
// step from 16.5 to 16.3 us at 512^2.
#ifndef FKADJ_RCP_CUBIC
#define FKADJ_RCP_CUBIC 1
#endif

// r refined towards 1/x from the estimate r (see FKADJ_RCP_CUBIC)
__device__ __forceinline__ double rcp_refine(double x, double r) {
#if FKADJ_RCP_CUBIC
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
#else
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
#endif
}

// 1/x for positive x or x = +inf without the division's branches: the hardware
// reciprocal estimate (rcp.approx.ftz.f64) refined by rcp_refine.  Within one
// ulp of the correctly rounded quotient (tests/test_gpu_mathfn.py); x = +inf,
// and x beyond 2^1022 (where the estimate flushes the subnormal quotient),
// give 0.  The three reciprocals of every vector-field and Jacobian evaluation take
// its branch-free form (fk_rcp_finite); the IEEE division in their place cost
// about 3 % of the gradient's time at 512 x 512.
__device__ __forceinline__ double own_rcp(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = rcp_refine(x, r);
    return isinf(x) ? 0.0 : r;  // the refinement turns inf * 0 into NaN
}

// own_rcp for finite x in [2^-1000, 2^1001]: the same value, without the +inf test.
__device__ __forceinline__ double fk_rcp_finite(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return rcp_refine(x, r);
}

// The exponential of the smoothed steps, by Tang's table-driven method (ACM
// TOMS 15(2), 1989) in powers of two: e^{c d} = 2^(s d / 16), s = 16 c / ln2.
// With K = rint(s d) = 16 m + j and f = s d - K, |f| <= 1/2, it is
// 2^m 2^(j/16) (1 + p(f)), p(f) = 2^(f/16) - 1 = f (c1 + f (c2 + ...)): the
// degree-4 Chebyshev fit of (e^r - 1 - r) / r^2 on [-ln2/32, ln2/32] (error of
// p 2.8e-17) with the powers of ln2/16 folded into its coefficients, the 16
// values 2^(j/16) in shared memory (exp_table_init).  The rounding to an
// integer is the fma's own: adding 1.5 * 2^52 leaves rint(s d) in the low bits
// of the sum.  s comes in two parts, so s d is formed without a rounding of
// its own (the product and the subtraction of K are one fma each): 11 FP64
// instructions, one fewer than reducing a rounded c d by ln2/16 in two parts,
// and the rounding of c d, up to |c d| / 2 ulp of the result, is gone.  With
// the clamp in one instruction, the coefficients in constant memory and the
// regrouped currents below: 512^2 x 1000 gradient (sqrt store) 66.5 -> 64.6 ms,
// exact gradient 512^2 x 500 29.9 -> 28.3 ms, 2048^2 x 24 24.2 -> 22.8 ms.
// Within 1.2 ulp of e^x for x in [-707, 692]; it saturates instead of
// overflowing: the result stays in [2^-1020, 2^1000) (m is clamped), so the
// smoothed steps need no cap of their own.  K is read from the sum's low word:
// beyond |s d| = 2^31 (at the steps' slope of 100, |u| above 4.6e5: a state
// that has blown up) the value is one of that range, but not always the limit
// on the argument's side; beyond 2^51 and at infinities it is unspecified.  A
// NaN argument gives NaN.
__shared__ double fk_exp2_tab[16];
// 2^(j/16), j = 0..15
__constant__ double kExp2Tab[16] = {
    0x1.0000000000000p+0, 0x1.0b5586cf9890fp+0, 0x1.172b83c7d517bp+0, 0x1.2387a6e756238p+0,
    0x1.306fe0a31b715p+0, 0x1.3dea64c123422p+0, 0x1.4bfdad5362a27p+0, 0x1.5ab07dd485429p+0,
    0x1.6a09e667f3bcdp+0, 0x1.7a11473eb0187p+0, 0x1.8ace5422aa0dbp+0, 0x1.9c49182a3f090p+0,
    0x1.ae89f995ad3adp+0, 0x1.c199bdd85529cp+0, 0x1.d5818dcfba487p+0, 0x1.ea4afa2a490dap+0};
// c1 .. c6: ln2/16, (ln2/16)^2 / 2, then q_k (ln2/16)^k of the fit.  In
// constant memory: a literal of more than 32 significant bits takes moves.
constexpr double kLn2_16 = 0x1.62e42fefa39efp-5;
__constant__ double kExpC[6] = {kLn2_16,
                                0.5 * kLn2_16 * kLn2_16,
                                0x1.55555554dd44dp-3 * (kLn2_16 * kLn2_16 * kLn2_16),
                                0x1.55555555194d2p-5 * (kLn2_16 * kLn2_16 * kLn2_16 * kLn2_16),
                                0x1.11120af701debp-7 * (kLn2_16 * kLn2_16 * kLn2_16 * kLn2_16 * kLn2_16),
                                0x1.6c17bb51f236dp-10 * (kLn2_16 * kLn2_16 * kLn2_16 * kLn2_16 * kLn2_16 * kLn2_16)};

// Exponent of the smallest value, 2^-kExpBias.  The table in shared memory
// holds 2^(j/16 - kExpBias) and the shift adds 16 kExpBias to K, so that one
// instruction clamps m to its range (min with the top, then max with 0).
constexpr int kExpBias = 1020;

// Every kernel that evaluates the model calls this before its first CTA barrier.
__device__ __forceinline__ void exp_table_init() {
    if (threadIdx.x < 16) {
        const double t = kExp2Tab[threadIdx.x];
        fk_exp2_tab[threadIdx.x] = __hiloint2double(__double2hiint(t) - (kExpBias << 20), __double2loint(t));
    }
}

// e^{c d}, c given as s_h + s_l = 16 c / ln2
__device__ __forceinline__ double exp_scaled(double d, double s_h, double s_l) {
    constexpr double kShift = 0x1.8p52 + 16.0 * kExpBias;
    const double t = fma(d, s_h, kShift);
    const double kd = t - kShift;
    const int k = __double2loint(t);
    const double f = fma(d, s_l, fma(d, s_h, -kd));
    double q = fma(kExpC[5], f, kExpC[4]);
    q = fma(q, f, kExpC[3]);
    q = fma(q, f, kExpC[2]);
    q = fma(q, f, kExpC[1]);
    q = fma(q, f, kExpC[0]);
    const int m = __vimin_s32_relu(k >> 4, 998 + kExpBias);
    const double T = fk_exp2_tab[k & 15];
    // 2^m 2^(j/16): m added to the exponent field
    const double Ts = __hiloint2double(__double2hiint(T) + (m << 20), __double2loint(T));
    return fma(Ts, f * q, Ts);
}

// e^x: the same with c = 1
__device__ __forceinline__ double fk_exp(double x) {
    return exp_scaled(x, 0x1.71547652b82fep+4, 0x1.777d0ffda0d24p-52);
}

// Everything below is written with explicit fma, and with no sum that takes an
// unrounded product, so that the compiler has nothing left to contract: every
// kernel that evaluates a cell gives the same bits.

// The two smoothed steps and the voltage-dependent time scale at u.  A step is
// s = (1 + tanh x)/2 written as the logistic 1/(1 + e^{-2x}) (the same
// function; one exp and one reciprocal instead of a tanh), its complement
// 1 - s = e^{-2x} s without cancellation; the exponential stays below 2^1000,
// so 1 + e is finite and s positive.  p and q share the slope ksm, so q's
// exponential is p's times a constant.  tau_v-(q) = q tau_v1- + (1 - q)
// tau_v2- only enters as its reciprocal and, in the Jacobian, through dq/du:
// with eq = e^{-2 ksm (u - u_v)}, tau_v- = (tau_v1- + eq tau_v2-) / (1 + eq), so
//   1/tau_v- = (1 + eq) rT   and   q (1 - q) / tau_v-^2 = eq rT^2,
// rT = 1 / (tau_v1- + eq tau_v2-): one reciprocal where q's logistic and the
// time scale took two.  eq is held below about 1e300 (u < -3.4, far outside
// the model's range), where the two are at their limits 1/tau_v2- and 0.
struct Steps {
    double d;      // u - u_c
    double p, cp;  // p step and 1 - p
    double s, e2;  // slow inward step, e^{-2x} of it
    double rT, eq;
};
__device__ __forceinline__ Steps fk_steps(const DevModel& P, double u) {
    Steps S;
    S.d = u - P.u_c;
    const double e = exp_scaled(S.d, P.sp_h, P.sp_l);
    S.e2 = exp_scaled(u - P.u_csi, P.ss_h, P.ss_l);
    S.p = fk_rcp_finite(1.0 + e);
    S.cp = e * S.p;
    const double q = e * P.eq;
    // min with 1e300 on the high word (q > 0): an integer instruction
    S.eq = __hiloint2double(min(__double2hiint(q), 0x7e37e43c), __double2loint(q));
    S.rT = fk_rcp_finite(fma(S.eq, P.tau_v2m, P.tau_v1m));
    S.s = fk_rcp_finite(1.0 + S.e2);
    return S;
}

// Ionic currents (formula of cu-F:29-45):
//   ud = p (v (1-u)(u-u_c)/tau_d - 1/tau_r) - (1-p) u/tau_0 + w s/tau_si
//   vd = (1-p)(1-v)/tau_v- - p v/tau_v+,  wd likewise
__device__ __forceinline__ void fk_ion(const DevModel& P, double u, double v, double w,
                                       double& ud, double& vd, double& wd) {
    const Steps S = fk_steps(P, u);
    const double rtv = (1.0 + S.eq) * S.rT;
    const double g = (1.0 - u) * S.d;
    const double a = fma(v * g, P.r_tau_d, -P.r_tau_r);
    ud = fma(S.p, a, fma(-S.cp, u * P.r_tau_0, (S.s * w) * P.r_tau_si));
    vd = fma(-(S.p * v), P.r_tau_vp, (S.cp * (1.0 - v)) * rtv);
    wd = fma(-(S.p * w), P.r_tau_wp, (S.cp * (1.0 - w)) * P.r_tau_wm);
}

// The seven non-zero entries of the transposed Jacobian of fk_ion
// (formula of cu-G:1160-1184): jt[0]=du'/du, jt[1]=dv'/du, jt[2]=dw'/du,
// jt[3]=du'/dv, jt[4]=dv'/dv, jt[5]=du'/dw, jt[6]=dw'/dw.
struct JacT {
    double a0, a1, a2, a3, a4, a5, a6;
};

// Jacobian entries, factored: the reference's derivatives with the common
// factors taken out and the constant products precomputed,
//   a0 = hk (v g r_d + u r_0 - r_r) + p v r_d ((1-u) - (u-u_c)) + 2 k_fk r_si w s (1-s) - (1-p) r_0,
//   a1 = (1-p)(1-v) 2 ksm dtau q(1-q)/tau^2 - hk (v r_v+ + (1-v)/tau_v-),
//   a2 = -hk (w r_w+ + (1-w) r_w-),
// with hk = dp/du = 2 ksm p (1-p), g = (1-u)(u-u_c).
__device__ __forceinline__ JacT fk_jacT(const DevModel& P, double u, double v, double w) {
    const Steps S = fk_steps(P, u);
    const double rtv = (1.0 + S.eq) * S.rT;
    const double dqr = (S.eq * S.rT) * S.rT;
    const double hk = P.two_ksm * (S.p * S.cp);
    const double ds = (S.e2 * S.s) * S.s;
    const double g1 = 1.0 - u;
    const double g = g1 * S.d;
    const double omv = 1.0 - v;
    JacT J;
    J.a3 = (S.p * g) * P.r_tau_d;
    J.a5 = S.s * P.r_tau_si;
    J.a0 = fma(hk, fma(v * g, P.r_tau_d, fma(u, P.r_tau_0, -P.r_tau_r)),
               fma((S.p * v) * P.r_tau_d, g1 - S.d, fma(P.kfk2_rsi * w, ds, -(S.cp * P.r_tau_0))));
    J.a1 = fma((S.cp * omv) * P.two_ksm_dv12, dqr, -(hk * fma(v, P.r_tau_vp, omv * rtv)));
    J.a4 = fma(-S.p, P.r_tau_vp, -(S.cp * rtv));
    J.a2 = -(hk * fma(w, P.r_tau_wp, (1.0 - w) * P.r_tau_wm));
    J.a6 = fma(-S.p, P.r_tau_wp, -(S.cp * P.r_tau_wm));
    return J;
}

// Sum of the four neighbours minus four times the centre, in the order of the
// reference's stencil (cu-F:319-424).
__device__ __forceinline__ double lap4(double n, double s, double w, double e, double c) {
    return fma(-4.0, c, ((n + s) + w) + e);
}

// Forward vector field at a cell from its values y and Laplacian sums t:
// D/h^2 t + F_ion + E gh on u.
__device__ __forceinline__ void fk_field(const DevModel& P, const double (&y)[3], const double (&t)[3], double E,
                                         double gh, double& fu, double& fv, double& fw) {
    double ud, vd, wd;
    fk_ion(P, y[0], y[1], y[2], ud, vd, wd);
    fu = fma(E, gh, fma(P.cu, t[0], ud));
    fv = fma(P.cv, t[1], vd);
    fw = fma(P.cw, t[2], wd);
}

// Forward vector field at shared-memory cell q of a region W doubles wide with
// field planes RN apart.  The plain sum of the neighbours is NaN where any of
// them is missing: then (holes' edges, about one warp in five of a sheet with
// obstacles) each missing neighbour is replaced by the opposite one
// (cu-F:319-420), all three fields after u's test.
template <int W, int RN>
__device__ __forceinline__ void rhs_at(const DevModel& P, const double* __restrict__ Y, int q,
                                       double E, double gh, double& fu, double& fv, double& fw) {
    const double u = Y[q];
    if (isnan(u)) {  // holes and the NaN ring skip the arithmetic (their result is NaN either way)
        fu = fv = fw = u;
        return;
    }
    const double un = Y[q - W], us = Y[q + W], uw = Y[q - 1], ue = Y[q + 1];
    const bool nN = isnan(un), nS = !nN && isnan(us);
    const bool nW = isnan(uw), nE = !nW && isnan(ue);
    const int qa = nN ? q + W : q - W, qb = nS ? q - W : q + W;
    const int qc = nW ? q + 1 : q - 1, qd = nE ? q - 1 : q + 1;
    const double* Yv = Y + RN;
    const double* Yw = Y + 2 * RN;
    const double y[3] = {u, Yv[q], Yw[q]};
    const double t[3] = {lap4(nN ? us : un, nS ? un : us, nW ? ue : uw, nE ? uw : ue, u),
                         lap4(Yv[qa], Yv[qb], Yv[qc], Yv[qd], y[1]), lap4(Yw[qa], Yw[qb], Yw[qc], Yw[qd], y[2])};
    fk_field(P, y, t, E, gh, fu, fv, fw);
}

// Hermite combination c0 x0 + c1 m0 + c2 x1 + c3 m1, in this order
__device__ __forceinline__ double hermite4(const double (&c)[4], double x0, double m0, double x1, double m1) {
    return fma(c[3], m1, fma(c[2], x1, fma(c[1], m0, c[0] * x0)));
}

// Weight code of the transposed Laplacian at a cell: 2 bits per direction
// (north, south, west, east), value 0 (neighbour missing), 1, or 2 (the
// neighbour mirrored this cell); rule of cu-G:1004-1111.
__device__ __forceinline__ int wcode_n(int c) { return c & 3; }
__device__ __forceinline__ int wcode_s(int c) { return (c >> 2) & 3; }
__device__ __forceinline__ int wcode_w(int c) { return (c >> 4) & 3; }
__device__ __forceinline__ int wcode_e(int c) { return (c >> 6) & 3; }

// J_F^T z plus D/h^2 times the transposed-Laplacian sums t.
__device__ __forceinline__ void adj_field(const DevModel& P, const JacT& J, const double (&z)[3],
                                          const double (&t)[3], double& gu, double& gv, double& gw) {
    gu = fma(P.cu, t[0], fma(J.a0, z[0], fma(J.a1, z[1], J.a2 * z[2])));
    gv = fma(P.cv, t[1], fma(J.a3, z[0], J.a4 * z[1]));
    gw = fma(P.cw, t[2], fma(J.a5, z[0], J.a6 * z[2]));
}

// Weighted neighbour sum at shared-memory cell q of one field, minus four times
// the centre: the plain sum, missing neighbours (weight 0; they hold NaN) as 0,
// then those of weight 2 once more.
template <int W>
__device__ __forceinline__ double lapT_at(const double* __restrict__ Z, int q, int code) {
    const int cn = wcode_n(code), cs = wcode_s(code), cw = wcode_w(code), ce = wcode_e(code);
    const double vn = cn ? Z[q - W] : 0.0, vs = cs ? Z[q + W] : 0.0;  // integer tests: no FP64 compares
    const double vw = cw ? Z[q - 1] : 0.0, ve = ce ? Z[q + 1] : 0.0;
    double t = lap4(vn, vs, vw, ve, Z[q]);
    if (code & 0xaa) {
        if (cn == 2) t += vn;
        if (cs == 2) t += vs;
        if (cw == 2) t += vw;
        if (ce == 2) t += ve;
    }
    return t;
}

// Adjoint vector field L^T z + J_F(y)^T z at shared-memory cell q.
template <int W, int RN>
__device__ __forceinline__ void adj_at(const DevModel& P, const double* __restrict__ Z, int q,
                                       int code, const JacT& J, double& gu, double& gv,
                                       double& gw) {
    const double z[3] = {Z[q], Z[RN + q], Z[2 * RN + q]};
    const double t[3] = {lapT_at<W>(Z, q, code), lapT_at<W>(Z + RN, q, code), lapT_at<W>(Z + 2 * RN, q, code)};
    adj_field(P, J, z, t, gu, gv, gw);
}

}  // namespace fkadj
