// Mixture-averaged transport (transport.cuh's formulas, FP64) on a repacked mechanism that a kernel
// takes by value, so that its constants are constant-bank operands.
#pragma once
#include "common.cuh"
#include "rcp.cuh"

namespace cb2 {

template <int NS>
struct TransTab {
  static constexpr int kPairs = NS * (NS + 1) / 2;  // pairs a <= b
  double imw[NS], mw[NS], gas[NS];
  double vis_coeff[NS], lj_inv[NS], vis_a[NS];  // vis_a = 1.147 lj_inv^-0.145
  double w14[NS][NS], sq[NS][NS];               // sq = sqrt(sqrt_WiDivWjPl1Mul8), w14 = (W_j/W_i)^(1/4) sq
  int geometry[NS];                             // 0 atom, 1 linear, 2 nonlinear
  double zrot_pi[NS], kbe_inv[NS], bdc_r[NS];   // pi ZRot298; 1/kbe, binary coefficient / R of the pair (s, s)
  double ibdc[NS][NS];                          // 1 / binary coefficient, a < b
  // Omega_D depends on a pair through kb/eps alone, and few of the pairs differ in it (22 of 45 for
  // the H2/air mechanism): the distinct values, and each pair's number among them
  int n_red;
  double kbe[kPairs], om_a[kPairs];  // om_a = 1.0548 kbe^-0.15504
  int pair[NS][NS];
};

struct TransTabs {
  int ns = 0;  // 0: the mechanism does not fit
  TransTab<5> t5;
  TransTab<9> t9;
};

// om: NS (NS + 1) / 2 values of this thread, `stride` apart (shared memory: pair numbers index it).
//
// Bound by the FP64 pipe.  The powers T^-0.15504 and T^-0.145 are taken once per node and scaled by
// tabulated powers of the pair's constant, (T k)^a = T^a k^a; the shifted power
// (T k + 0.55909)^-2.1705 once per distinct k.
template <int NS>
__device__ __forceinline__ void transport_properties_tab(double t, double mw_total, const double *y, const double *cp,
                                                         const TransTab<NS> &m, double *om, int stride, double &mu,
                                                         double &kappa, double *rhoD) {
  constexpr double pi = 3.141592653589793;
  const double lnt = log(t), st = sqrt(t), it = recip(t);
  {
    const double ta = exp(-0.15504 * lnt);
#pragma unroll 1
    for (int u = 0; u < m.n_red; ++u)
      om[u * stride] = fma(m.om_a[u], ta, exp(-2.1705 * log(fma(t, m.kbe[u], 0.55909))));
  }
  double X[NS], vs[NS], rs[NS];
  const double tv = exp(-0.145 * lnt);
#pragma unroll
  for (int l = 0; l < NS; ++l) {
    X[l] = y[l] * mw_total * m.imw[l];
    const double q = fma(t, m.lj_inv[l], 0.5), q2 = q * q;
    vs[l] = m.vis_coeff[l] * st * q2 * recip(fma(m.vis_a[l] * tv, q2, 1.0));
    rs[l] = rsqrt(vs[l]);
  }
  double visc = 0, cond = 0;
  const double t12 = st;  // T^(3/2) / T
#pragma unroll
  for (int a = 0; a < NS; ++a) {
    const double Ra = m.gas[a];
    double lambda = 15 * 0.25 * vs[a] * Ra;
    if (m.geometry[a] != 0) {
      const double tri = it * m.kbe_inv[a];
      const double tmp = sqrt(tri * pi) * pi;
      const double FT = 1 + 0.5 * tmp + (2 + 0.25 * pi * pi) * tri + tmp * tri;
      const double rd = m.bdc_r[a] * t12 * recip(om[m.pair[a][a] * stride]);
      const bool lin = m.geometry[a] == 1;
      const double f1 = lin ? 10.0 / 3 : 5.0, f2 = lin ? 5.0 : 7.5, f3 = lin ? 2.0 : 3.0;
      const double adpb =
          (2.5 * vs[a] - rd) * FT * recip(fma(m.zrot_pi[a], vs[a], FT * fma(f1, vs[a], 2.0 * rd)));
      lambda += -f2 * adpb * vs[a] * Ra + rd * cp[a] + rd * (f3 * adpb - 2.5) * Ra;
    }
    double den = 0;
    const double sva = vs[a] * rs[a];
#pragma unroll
    for (int b = 0; b < NS; ++b) {
      if (a == b) {
        den += X[b];
      } else {
        const double f = fma(rs[b] * sva, m.w14[a][b], m.sq[a][b]);
        den = fma(f * f, X[b], den);
      }
    }
    visc = fma(vs[a] * X[a], recip(den), visc);
    cond = fma(lambda * X[a], recip(fma(1.065, den, -0.065 * X[a])), cond);
  }
  mu = visc;
  kappa = cond;
  // mixture-averaged diffusivity
  constexpr double eps = 1e-12;
  double sum = 0, dsum[NS];
#pragma unroll
  for (int l = 0; l < NS; ++l) {
    X[l] += eps;
    sum = fma(X[l], m.mw[l], sum);
    dsum[l] = 0;
  }
#pragma unroll
  for (int l = 0; l < NS; ++l)
#pragma unroll
    for (int n = l + 1; n < NS; ++n) {
      const double inv = om[m.pair[l][n] * stride] * m.ibdc[l][n];
      dsum[l] = fma(X[n], inv, dsum[l]);
      dsum[n] = fma(X[l], inv, dsum[n]);
    }
  const double f = st * (1.0 / kRu);  // T^(3/2) / (T R_u)
#pragma unroll
  for (int l = 0; l < NS; ++l) rhoD[l] = (sum - X[l] * m.mw[l]) * f * recip(dsum[l]);
}

}  // namespace cb2
