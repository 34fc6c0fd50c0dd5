// line_weno.cuh -- the line passes' arithmetic: Steger-Warming split and the
// WENO7-SYMBO reconstruction evaluated point by point along a grid line.
//
// The same functions as ws_device.cuh (reference: split OCFD_NS_Jacobian3d.cpp:
// 55-129, WENO OCFD_Schemes.cpp:306-368 and :491-553), on a value type V:
//   double : one line per lane (the FP64 form);
//   float2 : two lines per lane in the halves of Blackwell's packed FP32x2
//            instructions (the mixed form).
//
// What the streaming form saves.  Taken face by face, WENO7 spends on each of
// P and M 7 differences, 45 operations on the five indicators, 16 on the
// candidates and 19 on weights and sums (87), although neighbouring faces
// share seven of their eight points.  Here each new point updates
//   D = t' - t, S = D' - D, T = S' - S, F = T' - T   (4 operations)
// and everything that belongs to the cell triple it completes:
//
// * All five indicators of the triple (a, b, c) of consecutive differences
//   are values at five points of one cubic: e_k = r_k^2 + s_k^2 + C T^2 + eps'
//   with r_k its first and s_k its second derivative there, so they follow
//   from one another by Taylor shifts (s +- T; r +- 6 s + 3 T).  24 operations
//   for five indicators instead of 45; each waits 0..4 steps for its face.
//   (The reference's k = 2 indicator takes its second derivative one point
//   further on, which makes it share s^2 + C T^2 + eps' with k = 1.)
// * The candidates' differences are multiples of the fourth differences F:
//   with q_2 the central candidate (all times 12),
//     q_1 - q_2 = F_1, q_0 - q_1 = -3 F_0, q_3 - q_2 = F_2, q_4 - q_3 = -3 F_3,
//   so the face value is the central candidate plus
//     [F_1 (w_0 + w_1) - 3 F_0 w_0 + F_2 (w_3 + w_4) - 3 F_3 w_4] / (12 sum w),
//   6 operations, and w_0 + w_1, w_3 + w_4 are needed for the sum anyway.
// * The central candidates of neighbouring faces difference to
//   (7 (g_-1 + g_0) - (g_-2 + g_1)) / 12 on the split flux's first differences g:
//   with the sum of the corrections' difference 5 operations per cell and sign.
// Per face and variable 51 FP64 operations for F+ and 50 for F-, 4 each for the
// quotient and 5 for the cell: 119 instead of 190.  All of it is an exact algebraic
// rewrite; in floating point it agrees with the reference's form to a few 1e-16
// of the flux.
//
// The split: with E_k+- = e_k +- sqrt(e_k^2 + eps^2) (twice the split
// eigenvalue) every component is a combination of sigma = c1 E1 + E2 + E3,
// E2 + E3 and m = t0 c (E3 - E2): mass t0 sigma, momentum (mass) u_i + m k_i,
// energy (mass) |u|^2/2 + (u.k) m + t0 c^2 (1/2 + c3)(E2 + E3).  63 FP64
// operations against 115 for the componentwise form.
#pragma once
#include "ws_device.cuh"

namespace ws {

// ---- value types ------------------------------------------------------------
template <typename V>
struct LineVal;
template <>
struct LineVal<double> {
    using CT = double;
    static constexpr int NL = 1;      // lines per lane
    static constexpr double SCALE = 1.0;
};
template <>
struct LineVal<float2> {
    using CT = float;
    static constexpr int NL = 2;
    // the split fluxes are scaled by this power of two (and eps' by its square),
    // so that products of two indicators stay in the FP32 range up to flux
    // differences of 5e9; the face-by-face form's pairs did up to 6e8 or 1e9,
    // these pairs without it, one of them with the largest indicator, 3e8
    static constexpr double SCALE = 0.0625;
};

// (the _rn forms are never contracted, so every kernel instance rounds alike)
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double vsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double vmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
// a b - c
__device__ __forceinline__ double vfms(double a, double b, double c) { return fma(a, b, -c); }
// maximum of two indicators: one comparison on the FP64 pipe and two selects
// (comparing the bit patterns as integers takes four instructions of the
// half-rate integer pipe); a NaN operand reaches the face value through the
// products in any case
__device__ __forceinline__ double vmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double vsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ double vrcp(double a) { return 1.0 / a; }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return add2(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return sub2(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return mul2(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return fma2(a, b, c); }
__device__ __forceinline__ float2 vfms(float2 a, float2 b, float2 c) {
    return fma2(f2(-1.f), c, mul2(a, b));
}
__device__ __forceinline__ float2 vmax(float2 a, float2 b) {
    return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y));
}
__device__ __forceinline__ float2 vsqrt(float2 a) {
    return make_float2(ws_sqrt(a.x), ws_sqrt(a.y));
}
__device__ __forceinline__ float2 vrcp(float2 a) { return rcp2(a); }
template <typename V>
__device__ __forceinline__ V vset(double c);
template <>
__device__ __forceinline__ double vset<double>(double c) { return c; }
template <>
__device__ __forceinline__ float2 vset<float2>(double c) { return f2((float)c); }

// Coefficients of the streaming form: FP64 in constant memory (an instruction
// operand; see wkc in ws_device.cuh), packed FP32 as literals (from constant
// memory they spilled).  The linear weights are divided by that of the central
// candidate.
namespace lk {
enum Coef { CC, EPS, R2, R3, RM3, R6, RM6, R11, R12, RM12, RM18, R26, W0, W1, W3, W4, M3, SEVEN,
            NCOEF };
constexpr double val[NCOEF] = {
    wk::C, wk::EPS, 2 * wk::R, 3 * wk::R, -3 * wk::R, 6 * wk::R, -6 * wk::R, 11 * wk::R,
    12 * wk::R, -12 * wk::R, -18 * wk::R, 26 * wk::R,
    wk::D0 / wk::D2, wk::D1 / wk::D2, wk::D3 / wk::D2, wk::D4 / wk::D2, -3.0, 7.0};
}  // namespace lk
static __constant__ double lkd[lk::NCOEF] = {
    lk::val[0], lk::val[1], lk::val[2], lk::val[3], lk::val[4], lk::val[5], lk::val[6],
    lk::val[7], lk::val[8], lk::val[9], lk::val[10], lk::val[11], lk::val[12], lk::val[13],
    lk::val[14], lk::val[15], lk::val[16], lk::val[17]};
template <typename V, int I>
__device__ __forceinline__ V lkc() {
    if constexpr (sizeof(typename LineVal<V>::CT) == 8) {
        return lkd[I];
    } else {
        constexpr float c =
            (float)(lk::val[I] * (I == lk::EPS ? LineVal<V>::SCALE * LineVal<V>::SCALE : 1.0));
        return f2(c);
    }
}
__device__ __forceinline__ void prefetch_l2(const void* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// ---- split ------------------------------------------------------------------
template <typename V>
struct LineSplitK {
    V eps2, c1;                // eps^2, 2(gamma-1)
};

// F+ in out[0..4], F- in out[5..9] of one point, direction DIR; CART: the
// unit vector of DIR as metric gradient, else (a1, a2, a3).  t0 = 0.25 d / gamma,
// t0c = t0 c, kc = t0c (1/2 + c3) c.
template <int DIR, bool CART, typename V>
__device__ __forceinline__ void line_split(V t0, V t0c, V kc, V u, V v, V w, V c, V a1, V a2,
                                           V a3, const LineSplitK<V>& k, V out[10]) {
    V e1, cs, un, k1, k2, k3;          // u.a, c |a|, u.k, k = a / |a|
    if (CART) {
        e1 = un = DIR == 0 ? u : (DIR == 1 ? v : w);
        cs = c;
    } else {
        const V ss = vsqrt(vfma(a1, a1, vfma(a2, a2, vmul(a3, a3))));
        const V rcp = vrcp(ss);
        k1 = vmul(a1, rcp);
        k2 = vmul(a2, rcp);
        k3 = vmul(a3, rcp);
        e1 = vfma(a1, u, vfma(a2, v, vmul(a3, w)));
        un = vfma(k1, u, vfma(k2, v, vmul(k3, w)));
        cs = vmul(c, ss);
    }
    const V e2 = vsub(e1, cs), e3 = vadd(e1, cs);
    const V s1 = vsqrt(vfma(e1, e1, k.eps2));
    const V s2 = vsqrt(vfma(e2, e2, k.eps2));
    const V s3 = vsqrt(vfma(e3, e3, k.eps2));
    const V two = vset<V>(2.0);
    const V sg = vadd(s2, s3), ds = vsub(s3, s2);
    const V qh = vmul(vset<V>(0.5), vfma(u, u, vfma(v, v, vmul(w, w))));
#pragma unroll
    for (int h = 0; h < 2; ++h) {      // +, -
        const V E1 = h ? vsub(e1, s1) : vadd(e1, s1);
        const V s23 = h ? vfms(two, e1, sg) : vfma(two, e1, sg);
        const V df = h ? vfms(two, cs, ds) : vfma(two, cs, ds);
        const V m0 = vmul(t0, vfma(k.c1, E1, s23));
        const V m = vmul(t0c, df);
        V* o = out + 5 * h;
        o[0] = m0;
        if (CART) {
            o[1] = DIR == 0 ? vfma(m0, u, m) : vmul(m0, u);
            o[2] = DIR == 1 ? vfma(m0, v, m) : vmul(m0, v);
            o[3] = DIR == 2 ? vfma(m0, w, m) : vmul(m0, w);
        } else {
            o[1] = vfma(m0, u, vmul(m, k1));
            o[2] = vfma(m0, v, vmul(m, k2));
            o[3] = vfma(m0, w, vmul(m, k3));
        }
        o[4] = vfma(m0, qh, vfma(un, m, vmul(kc, s23)));
    }
}

// ---- streaming WENO -----------------------------------------------------------
// What one split flux carries along its line: the last point, the last first,
// second and third differences, fourth differences F[0..2] of lags 1..3, and
// the indicators that wait 1..4 steps for their face (oldest first).
template <typename V>
struct WenoLine {
    V t, b, S, T;
    V F[3];
    V l1[1], l2[2], l3[3], l4[4];
};
template <int N, typename V>
__device__ __forceinline__ V lag(V (&q)[N], V x) {      // in with x, out with the oldest
    const V o = q[0];
#pragma unroll
    for (int i = 0; i + 1 < N; ++i) q[i] = q[i + 1];
    q[N - 1] = x;
    return o;
}

// Takes the next point of the line.  num / den: 12 times the face value less
// the central candidate, for the face four points back (between the fourth
// and fifth newest points), valid from the eighth point on.  MINUS: F-, whose
// reconstruction is the mirror image: its k-th indicator belongs to the
// (4-k)-th triple.  Returns D.
template <bool MINUS, typename V>
__device__ __forceinline__ V weno_push(WenoLine<V>& s, V tn, V& num, V& den) {
    using namespace lk;
    const V D = vsub(tn, s.t), Sn = vsub(D, s.b), Tn = vsub(Sn, s.S), Fn = vsub(Tn, s.T);
    // first derivatives (times R) at the points of the triple, from its middle
    // difference b and Sn, T: r1 between b and c, r2 between a and b, r0 after
    // c, r3 before a; r4 one further out
    const V B = vfma(vmul(lkc<V, CC>(), Tn), Tn, lkc<V, EPS>());
    const V c1 = vfma(lkc<V, R3>(), Sn, vmul(lkc<V, R6>(), s.b));
    const V U = vfma(lkc<V, R2>(), Tn, c1), W = vfma(lkc<V, R11>(), Tn, c1);
    const V r0 = vfma(lkc<V, R6>(), Sn, U), r2 = vfma(lkc<V, RM6>(), Sn, U);
    const V r1 = vfma(lkc<V, RM3>(), Tn, U), r3 = vfma(lkc<V, RM12>(), Sn, W);
    const V sp = vadd(Sn, Tn), sm = vsub(s.S, Tn);      // second derivatives past c / before a
    const V eo = vfma(r0, r0, vfma(sp, sp, B)), ei = vfma(r3, r3, vfma(sm, sm, B));
    V e0, e1, e2, e3, e4, F0, F1, F2, F3;
    if (!MINUS) {
        const V r4 = vfma(lkc<V, RM18>(), Sn, vfma(lkc<V, R26>(), Tn, c1)), s4 = vsub(sm, Tn);
        const V base = vfma(Sn, Sn, B);
        e4 = vfma(r4, r4, vfma(s4, s4, B));
        e3 = lag(s.l1, ei);
        e2 = lag(s.l2, vfma(r2, r2, base));
        e1 = lag(s.l3, vfma(r1, r1, base));
        e0 = lag(s.l4, eo);
        F0 = s.F[2]; F1 = s.F[1]; F2 = s.F[0]; F3 = Fn;
    } else {
        const V r4 = vfma(lkc<V, R12>(), Sn, W), s4 = vadd(sp, Tn);
        const V base = vfma(s.S, s.S, B);
        e0 = ei;
        e1 = lag(s.l1, vfma(r2, r2, base));
        e2 = lag(s.l2, vfma(r1, r1, base));
        e3 = lag(s.l3, eo);
        e4 = lag(s.l4, vfma(r4, r4, vfma(s4, s4, B)));
        F0 = Fn; F1 = s.F[0]; F2 = s.F[1]; F3 = s.F[2];
    }
    s.F[2] = s.F[1]; s.F[1] = s.F[0]; s.F[0] = Fn;
    s.t = tn; s.b = D; s.S = Sn; s.T = Tn;
    e4 = vmax(vmax(vmax(e0, e1), vmax(e2, e3)), e4);    // SYMBO
    // weights as products of the other indicators: x, y carry w_0 and w_0 + w_1
    // without e2 e3 e4, x3, y3 carry w_4 and w_3 + w_4 without e0 e1 e2
    const V x = vmul(lkc<V, W0>(), e1), y = vfma(lkc<V, W1>(), e0, x);
    const V x3 = vmul(lkc<V, W4>(), e3), y3 = vfma(lkc<V, W3>(), e4, x3);
    const V n01 = vfma(F1, y, vmul(vmul(lkc<V, M3>(), F0), x));
    const V n34 = vfma(F2, y3, vmul(vmul(lkc<V, M3>(), F3), x3));
    const V p01 = vmul(e0, e1), p34 = vmul(e3, e4);
    if constexpr (sizeof(typename LineVal<V>::CT) == 8) {
        num = vmul(e2, vfma(p34, n01, vmul(p01, n34)));
        den = vfma(e2, vfma(p34, y, vmul(p01, y3)), vmul(p01, p34));
    } else {
        // divided by all five: no FP32 overflow or underflow of a product of
        // four indicators
        const V i01 = vrcp(p01), i34 = vrcp(p34), i2 = vrcp(e2);
        num = vfma(i01, n01, vmul(i34, n34));
        den = vfma(i01, y, vfma(i34, y3, i2));
    }
    return D;
}

// num / den.  FP64: a third-order Newton (Householder) step on the hardware's
// reciprocal approximation (relative error below 2^-20, so below 2^-60 after
// the step), 4 operations, within 2 ulp of the quotient (one rounding each of the
// step and the product), which is a correction to the central value.  No range
// test: den is a sum of products of four indicators, each at least eps' = 9e-11,
// so it is never small; num, such a product times a flux difference, overflows
// before den reaches 2^1022, where the approximation would underflow, and does so
// from flux differences of 1e33 on (alternating signs: 2e33; a single jump: 1e34).
// The face-by-face form, which shared P's and M's division, overflowed from 1e17
// on.  A branch here would keep the compiler from overlapping neighbouring points.
__device__ __forceinline__ double weno_quot(double n, double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return vmul(n, fma(y, fma(e, e, e), y));
}

}  // namespace ws
