// Nonlinear WENO reconstruction of one interface value from point values.
//
// weno5: Jiang-Shu weights a_r = d_r/(eps+beta_r)^2 (src/WENO.cu:3033-3088).
// weno7: Z-type weights a_r = d_r (1 + tau7/(eps+beta_r)^2), tau7 = (b0+3b1-3b2-b3)^2
//        (src/WENO.cu:3090-3196).
// Both fall back to the linear (optimal) weights when `shock` is false.
// The normalised weights are evaluated with one reciprocal per side: every a_r is multiplied
// by the product of all (eps+beta)^2 terms, which leaves sum(a_r q_r)/sum(a_r) unchanged
// (the reference divides once per sub-stencil, src/WENO.cu:3051-3053, 3127-3130).
//
// The "plus" side reconstructs the left-biased value at i+1/2 from v[i-r+1 .. i+r-1]
// (r = 3 or 4, v[r-1] is node i); the "minus" side reconstructs the right-biased value
// from v[i-r+2 .. i+r] (v[r-2] is node i).  The interface value is plus + minus.
#pragma once
#include "common.cuh"
#include "rcp.cuh"

namespace cb2 {

template <typename T>
__device__ __forceinline__ T sq(T x) { return x * x; }

// Exact power of two s with x*s in [1, 2) for a positive normal x (the reciprocal of x's
// binade).  The nonlinear weights below are products of three or four (eps + beta)^2 terms;
// scaling every term by the same s keeps the normalised weights unchanged, changes no
// rounding, and keeps the products far from FP underflow and overflow.
__device__ __forceinline__ double binade_inv(double x) {
  return __hiloint2double(0x7FE00000 - (__double2hiint(x) & 0x7FF00000), 0);
}
__device__ __forceinline__ float binade_inv(float x) {
  return __int_as_float(0x7F000000 - (__float_as_int(x) & 0x7F800000));
}

// ---- one side of an interface ------------------------------------------------------------
// FP64, from the undivided differences of the stencil (see the node-centred pair below): the
// smoothness indicators and the candidate values, relative to the middle node, share them.
__device__ __forceinline__ double pow2_inv_max(double a, double b, double c, double d) {
  // the reciprocal binade of the largest: positive doubles order as their high words do
  const int h = max(max(__double2hiint(a), __double2hiint(b)), max(__double2hiint(c), __double2hiint(d)));
  return __hiloint2double(0x7FE00000 - (h & 0x7FF00000), 0);
}

__device__ __forceinline__ double weno5_side(double u0, double u1, double u2, double u3, double u4, double eps,
                                             bool shock) {
  const double d0 = u1 - u0, d1 = u2 - u1, d2 = u3 - u2, d3 = u4 - u3;
  const double s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2;
  const double k3 = 1.0 / 3, k6 = 1.0 / 6, h1 = 0.5 * d1;
  // candidates relative to u2; linear weights times ten: 1, 6, 3
  const double c0 = fma(k3, s0, h1), c1 = fma(k3, s1, h1), c2 = fma(-k6, s2, 0.5 * d2);
  if (!shock) return fma(0.3, c2, fma(0.6, c1, fma(0.1, c0, u2)));
  const double f0 = fma(0.5, s0, d1), f1 = fma(0.5, s1, d1), f2 = fma(-0.5, s2, d2);
  const double k13 = 13.0 / 12;
  double A0 = fma(f0, f0, fma(k13 * s0, s0, eps)), A1 = fma(f1, f1, fma(k13 * s1, s1, eps)),
         A2 = fma(f2, f2, fma(k13 * s2, s2, eps));
  const double sc = pow2_inv_max(A0, A1, A2, A2);
  A0 *= sc; A1 *= sc; A2 *= sc;
  const double D0 = A0 * A0, D1 = A1 * A1, D2 = A2 * A2;
  const double w0 = D1 * D2, w1 = 6.0 * (D0 * D2), E2 = D0 * D1, w2 = 3.0 * E2;
  return fma(fma(w2, c2, fma(w1, c1, w0 * c0)), recip(fma(3.0, E2, w0 + w1)), u2);
}

__device__ __forceinline__ double weno7_side(double u0, double u1, double u2, double u3, double u4, double u5,
                                             double u6, double eps, bool shock) {
  const double d0 = u1 - u0, d1 = u2 - u1, d2 = u3 - u2, d3 = u4 - u3, d4 = u5 - u4, d5 = u6 - u5;
  const double s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2, s3 = d4 - d3, s4 = d5 - d4;
  const double t0 = s1 - s0, t1 = s2 - s1, t2 = s3 - s2, t3 = s4 - s3;
  const double k3 = 1.0 / 3, k6 = 1.0 / 6, k12 = 1.0 / 12;
  const double h2 = 0.5 * d2, e = fma(k3, s2, h2);
  const double c0 = fma(0.25, t0, fma(k3, s1, h2)), c1 = fma(-k12, t1, e), c2 = fma(-k12, t2, e),
               c3 = fma(k12, t3, fma(-k6, s3, 0.5 * d3));
  if (!shock)
    return fma(4.0 / 35, c3, fma(18.0 / 35, c2, fma(12.0 / 35, c1, fma(1.0 / 35, c0, u3))));
  const double c = fma(0.5, s2, d2);
  const double f0 = fma(k3, t0, fma(0.5, s1, d2)), f1 = fma(-k6, t1, c), f2 = fma(-k6, t2, c),
               f3 = fma(k3, t3, fma(-0.5, s3, d3));
  const double g0 = s1 + t0, g3 = s3 - t3;
  const double kg = 13.0 / 12, kt = 1043.0 / 960;
  const double gm = (kg * s2) * s2;
  const double b0 = fma(f0, fma(k12, t0, f0), fma(kt * t0, t0, (kg * g0) * g0));
  const double b1 = fma(f1, fma(k12, t1, f1), fma(kt * t1, t1, gm));
  const double b2 = fma(f2, fma(k12, t2, f2), fma(kt * t2, t2, gm));
  const double b3 = fma(f3, fma(k12, t3, f3), fma(kt * t3, t3, (kg * g3) * g3));
  double tz = fma(3.0, b1 - b2, b0 - b3);
  double A0 = eps + b0, A1 = eps + b1, A2 = eps + b2, A3 = eps + b3;
  const double sc = pow2_inv_max(A0, A1, A2, A3);
  A0 *= sc; A1 *= sc; A2 *= sc; A3 *= sc; tz *= sc;
  const double D0 = A0 * A0, D1 = A1 * A1, D2 = A2 * A2, D3 = A3 * A3;
  const double D01 = D0 * D1, D23 = D2 * D3;
  const double w0 = fma(tz, tz, D0) * (D1 * D23), w1 = 12.0 * (fma(tz, tz, D1) * (D0 * D23));
  const double w2 = 18.0 * (fma(tz, tz, D2) * (D01 * D3)), E3 = fma(tz, tz, D3) * (D01 * D2), w3 = 4.0 * E3;
  return fma(fma(w3, c3, fma(w2, c2, fma(w1, c1, w0 * c0))), recip(fma(4.0, E3, (w0 + w1) + w2)), u3);
}

// FP32 weights.  The single-division product form needs the product of three or four
// (eps + beta)^2 terms, which FP32 cannot hold across the dynamic range of a discontinuity.  The
// FP32 path normalises by the smallest term instead, and takes every ratio before squaring so
// that nothing underflows: with A_s = eps + beta_s (D_s = A_s^2), q_s = (A_min / A_s)^2 in (0, 1],
// T = |b0 + 3 b1 - 3 b2 - b3| (tau = T^2) and t = 1 / (1 + (A_min / T)^2) = tau / (D_min + tau),
//   WENO-JS  alpha_s ~ c_s q_s,   WENO-Z  alpha_s ~ c_s ((1 - t) + t q_s),
// the same weights up to a common factor, every term bounded by c_s.  (The square of a small A_s,
// e.g. eps + 0 for a uniform density of 0.3, is below the smallest normal FP32 number, and the
// paired FP32 instructions flush such results to zero.)
// The reciprocal is the hardware approximation (rcp.approx, within 1 ulp): 1/0 = inf and
// 1/inf = 0 as the formulas above require.
__device__ __forceinline__ float rcp32(float x) { return __fdividef(1.0f, x); }

// ---- node-centred pair ---------------------------------------------------------------
// Both one-sided values that the stencil centred on node n produces: the left-biased value at
// n+1/2 (`lp`, the plus side) and the right-biased value at n-1/2 (`rm`, the minus side).
// The two sides integrate over the same cell n with the same sub-stencils, so they share the
// smoothness indicators: beta of minus sub-stencil r equals beta of plus sub-stencil
// (last - r).  The pair costs one set of indicators instead of two.
//   WENO5: v[0..4], v[2] = node n.   WENO7: v[0..6], v[3] = node n.
//
// Both are written with the undivided differences of the stencil, d (first), s (second), t (third),
// shared by the smoothness indicators, which are quadratic forms of them, and by the candidate
// values, taken relative to node n.  That form needs 121 FP64 operations per WENO7 pair where the
// sums over point values took about 190, and it is the more exact one (no cancellation of the node
// values).  Sums of products are written as fused operations, so that every kernel that inlines
// these functions rounds alike.  FP64 only; the FP32 pair is packed (below).
__device__ __forceinline__ void weno5_node(const double *v, double eps, double &lp, double &rm) {
  const double d0 = v[1] - v[0], d1 = v[2] - v[1], d2 = v[3] - v[2], d3 = v[4] - v[3];
  const double s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2;
  const double f0 = fma(0.5, s0, d1), f1 = fma(0.5, s1, d1), f2 = fma(-0.5, s2, d2);
  const double k13 = 13.0 / 12;
  double A0 = fma(f0, f0, fma(k13 * s0, s0, eps)), A1 = fma(f1, f1, fma(k13 * s1, s1, eps)),
         A2 = fma(f2, f2, fma(k13 * s2, s2, eps));
  const double sc = pow2_inv_max(A0, A1, A2, A2);
  A0 *= sc; A1 *= sc; A2 *= sc;
  const double D0 = A0 * A0, D1 = A1 * A1, D2 = A2 * A2;
  // products of the D of the other sub-stencils, times ten times the linear weights
  const double E0 = D1 * D2, E1 = 6.0 * (D0 * D2), E2 = D0 * D1;
  const double k3 = 1.0 / 3, k6 = 1.0 / 6, h1 = 0.5 * d1, h2 = 0.5 * d2;
  const double W2 = 3.0 * E2, V0 = 3.0 * E0;
  const double np = fma(W2, fma(-k6, s2, h2), fma(E1, fma(k3, s1, h1), E0 * fma(k3, s0, h1)));
  const double nm = fma(V0, fma(-k6, s0, -h1), fma(E1, fma(k3, s1, -h2), E2 * fma(k3, s2, -h2)));
  lp = fma(np, recip(fma(3.0, E2, E0 + E1)), v[2]);
  rm = fma(nm, recip(fma(3.0, E0, E2 + E1)), v[2]);
}

__device__ __forceinline__ void weno7_node(const double *u, double eps, double &lp, double &rm) {
  const double d0 = u[1] - u[0], d1 = u[2] - u[1], d2 = u[3] - u[2], d3 = u[4] - u[3], d4 = u[5] - u[4],
               d5 = u[6] - u[5];
  const double s0 = d1 - d0, s1 = d2 - d1, s2 = d3 - d2, s3 = d4 - d3, s4 = d5 - d4;
  const double t0 = s1 - s0, t1 = s2 - s1, t2 = s3 - s2, t3 = s4 - s3;
  // first and second derivatives of the sub-stencils' cubics at node n (the third are t0 .. t3)
  const double k3 = 1.0 / 3, k6 = 1.0 / 6, k12 = 1.0 / 12;
  const double c = fma(0.5, s2, d2);
  const double f0 = fma(k3, t0, fma(0.5, s1, d2)), f1 = fma(-k6, t1, c), f2 = fma(-k6, t2, c),
               f3 = fma(k3, t3, fma(-0.5, s3, d3));
  const double g0 = s1 + t0, g3 = s3 - t3;
  // A = eps + beta, beta = f^2 + f t / 12 + 13/12 g^2 + 1043/960 t^2
  const double kg = 13.0 / 12, kt = 1043.0 / 960;
  const double gm = (kg * s2) * s2;
  const double b0 = fma(f0, fma(k12, t0, f0), fma(kt * t0, t0, (kg * g0) * g0));
  const double b1 = fma(f1, fma(k12, t1, f1), fma(kt * t1, t1, gm));
  const double b2 = fma(f2, fma(k12, t2, f2), fma(kt * t2, t2, gm));
  const double b3 = fma(f3, fma(k12, t3, f3), fma(kt * t3, t3, (kg * g3) * g3));
  double tz = fma(3.0, b1 - b2, b0 - b3);
  double A0 = eps + b0, A1 = eps + b1, A2 = eps + b2, A3 = eps + b3;
  const double sc = pow2_inv_max(A0, A1, A2, A3);
  A0 *= sc; A1 *= sc; A2 *= sc; A3 *= sc; tz *= sc;
  const double D0 = A0 * A0, D1 = A1 * A1, D2 = A2 * A2, D3 = A3 * A3;
  // Z weights (1 + tau / D_s) times the product of every D
  const double D01 = D0 * D1, D23 = D2 * D3;
  const double E0 = fma(tz, tz, D0) * (D1 * D23), E1 = fma(tz, tz, D1) * (D0 * D23);
  const double E2 = fma(tz, tz, D2) * (D01 * D3), E3 = fma(tz, tz, D3) * (D01 * D2);
  // candidates relative to u[3]; linear weights times 35: 1, 12, 18, 4
  const double h2 = 0.5 * d2, h3 = 0.5 * d3, e = fma(k3, s2, h2), em = fma(k3, s2, -h3);
  const double w1 = 12.0 * E1, w2 = 18.0 * E2, v1 = 12.0 * E2, v2 = 18.0 * E1;
  const double w3 = 4.0 * E3, v3 = 4.0 * E0;
  const double np = fma(w3, fma(k12, t3, fma(-k6, s3, h3)),
                        fma(w2, fma(-k12, t2, e), fma(w1, fma(-k12, t1, e), E0 * fma(0.25, t0, fma(k3, s1, h2)))));
  const double nm = fma(v3, fma(-k12, t0, fma(-k6, s1, -h2)),
                        fma(v2, fma(k12, t1, em), fma(v1, fma(k12, t2, em), E3 * fma(-0.25, t3, fma(k3, s3, -h3)))));
  lp = fma(np, recip(fma(4.0, E3, fma(18.0, E2, fma(12.0, E1, E0)))), u[3]);
  rm = fma(nm, recip(fma(4.0, E0, fma(18.0, E1, fma(12.0, E2, E3)))), u[3]);
}

// ---- packed FP32 node-centred pair ------------------------------------------------------
// The minus side is the plus formula applied to the mirrored stencil, so both sides run as one
// stream of float2 values through the sm_100 paired FP32 instructions (FFMA2, FADD2, FMUL2):
// lane x is the plus side on u[k], lane y the minus side on u[last - k].  Mirroring maps the
// plus sub-stencil r onto sub-stencil last - r, so the packed indicators of the first half of
// the sub-stencils carry the others in lane y.  Per lane the arithmetic is the FP32 node form
// above (D_min normalisation), with the final division done as a reciprocal and a product.
__device__ __forceinline__ float2 p2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 swap2(float2 a) { return make_float2(a.y, a.x); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(rcp32(a.x), rcp32(a.y)); }
// c0 a + c1 b + c2 c (+ c3 d) with scalar coefficients
__device__ __forceinline__ float2 lin3(float c0, float2 a, float c1, float2 b, float c2, float2 c) {
  return fma2(p2(c2), c, fma2(p2(c1), b, mul2(p2(c0), a)));
}
__device__ __forceinline__ float2 lin4(float c0, float2 a, float c1, float2 b, float c2, float2 c, float c3,
                                       float2 d) {
  return fma2(p2(c3), d, lin3(c0, a, c1, b, c2, c));
}
__device__ __forceinline__ float2 beta7_x2(float2 d1, float2 d2, float2 d3) {
  // d1^2 + 13/12 d2^2 + 1043/960 d3^2 + d1 d3/12; invariant under (d1, d3) -> (-d1, -d3), the
  // sign change that mirroring gives the first and third differences
  const float2 t = fma2(p2(1.0f / 12), d3, d1);
  return fma2(p2(1043.0f / 960), mul2(d3, d3), fma2(p2(13.0f / 12), mul2(d2, d2), mul2(d1, t)));
}

__device__ __forceinline__ void weno5_node_x2(const float *v, float eps, float &lp, float &rm) {
  const float2 U0 = make_float2(v[0], v[4]), U1 = make_float2(v[1], v[3]), U2 = p2(v[2]);
  const float2 U3 = make_float2(v[3], v[1]), U4 = make_float2(v[4], v[0]);
  const float k6 = 1.0f / 6;
  const float2 Q0 = lin3(2 * k6, U0, -7 * k6, U1, 11 * k6, U2);  // (q0, m0)
  const float2 Q1 = lin3(-k6, U1, 5 * k6, U2, 2 * k6, U3);       // (q1, m1)
  const float2 Q2 = lin3(2 * k6, U2, 5 * k6, U3, -k6, U4);       // (q2, m2)
  const float2 e0 = lin3(1, U0, -2, U1, 1, U2), f0 = lin3(1, U0, -4, U1, 3, U2);
  const float2 B0 = fma2(p2(13.0f / 12), mul2(e0, e0), mul2(p2(0.25f), mul2(f0, f0)));  // (b0, b2)
  const float e1 = v[1] + v[3] - 2 * v[2], f1 = v[1] - v[3];
  const float b1 = 13.0f / 12 * (e1 * e1) + 0.25f * (f1 * f1);
  const float2 AA = add2(p2(eps), B0);  // (A0, A2)
  const float A1 = eps + b1;
  const float Am = fminf(fminf(AA.x, AA.y), A1);
  const float2 RA = mul2(p2(Am), rcp2(AA));
  const float2 EA = mul2(RA, RA);  // (E0, E2)
  const float R1 = Am * rcp32(A1), E1 = R1 * R1;
  const float2 W0 = mul2(p2(0.1f), EA), W1 = p2(0.6f * E1), W2 = mul2(p2(0.3f), swap2(EA));
  const float2 num = fma2(W2, Q2, fma2(W1, Q1, mul2(W0, Q0)));
  const float2 den = add2(add2(W0, W1), W2);
  const float2 r = mul2(num, rcp2(den));
  lp = r.x;
  rm = r.y;
}

__device__ __forceinline__ void weno7_node_x2(const float *u, float eps, float &lp, float &rm) {
  float2 U[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) U[k] = make_float2(u[k], u[6 - k]);
  const float2 Q0 = lin4(-3, U[0], 13, U[1], -23, U[2], 25, U[3]);  // (q0, m0)
  const float2 Q1 = lin4(1, U[1], -5, U[2], 13, U[3], 3, U[4]);
  const float2 Q2 = lin4(-1, U[2], 7, U[3], 7, U[4], -1, U[5]);
  const float2 Q3 = lin4(3, U[3], 13, U[4], -5, U[5], 1, U[6]);
  const float k6 = 1.0f / 6;
  const float2 B0 = beta7_x2(lin4(-2 * k6, U[0], 9 * k6, U[1], -18 * k6, U[2], 11 * k6, U[3]),
                             lin4(-1, U[0], 4, U[1], -5, U[2], 2, U[3]), lin4(-1, U[0], 3, U[1], -3, U[2], 1, U[3]));
  const float2 B1 = beta7_x2(lin4(k6, U[1], -6 * k6, U[2], 3 * k6, U[3], 2 * k6, U[4]), lin3(1, U[2], -2, U[3], 1, U[4]),
                             lin4(-1, U[1], 3, U[2], -3, U[3], 1, U[4]));
  // plus side: b0 = B0.x, b1 = B1.x, b2 = B1.y, b3 = B0.y
  const float2 A0 = add2(p2(eps), B0), A1 = add2(p2(eps), B1);  // (A0, A3), (A1, A2)
  const float Am = fminf(fminf(A0.x, A0.y), fminf(A1.x, A1.y));
  const float2 R0 = mul2(p2(Am), rcp2(A0)), R1 = mul2(p2(Am), rcp2(A1));
  // t = tau / (D_min + tau), tau unchanged by the mirroring; T = 0 gives rz = inf and t = 0
  const float rz = Am * rcp32(fabsf((B0.x - B0.y) + 3 * (B1.x - B1.y)));
  const float t = rcp32(1.0f + rz * rz);
  const float2 EA = fma2(p2(t), mul2(R0, R0), p2(1.0f - t));  // (E0, E3)
  const float2 EB = fma2(p2(t), mul2(R1, R1), p2(1.0f - t));  // (E1, E2)
  const float2 W0 = mul2(p2(1.0f / 35), EA), W1 = mul2(p2(12.0f / 35), EB);
  const float2 W2 = mul2(p2(18.0f / 35), swap2(EB)), W3 = mul2(p2(4.0f / 35), swap2(EA));
  const float2 num = fma2(W3, Q3, fma2(W2, Q2, fma2(W1, Q1, mul2(W0, Q0))));
  const float2 den = add2(add2(W0, W1), add2(W2, W3));
  const float2 r = mul2(mul2(num, p2(1.0f / 12)), rcp2(den));
  lp = r.x;
  rm = r.y;
}

// plus + minus value of an interface; vp / vm: the NW values of each side's stencil
template <int ORDER>
__device__ __forceinline__ double weno_pm(const double *vp, const double *vm, double eps, bool shock) {
  if constexpr (ORDER == 5)
    return weno5_side(vp[0], vp[1], vp[2], vp[3], vp[4], eps, shock) +
           weno5_side(vm[4], vm[3], vm[2], vm[1], vm[0], eps, shock);
  else
    return weno7_side(vp[0], vp[1], vp[2], vp[3], vp[4], vp[5], vp[6], eps, shock) +
           weno7_side(vm[6], vm[5], vm[4], vm[3], vm[2], vm[1], vm[0], eps, shock);
}

}  // namespace cb2
