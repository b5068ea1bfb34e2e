// The adaptive ROK4E reactor with the full Jacobian on a repacked mechanism (chem_tab.cuh), one warp
// per reactor: k_reactor_advance's integrator (reactor.cu) for one-temperature NASA7 mechanisms of at
// most kChemTabReac reactions.
//
// A reactor is a serial chain, so what counts is the latency of an attempt.  The generic kernel takes
// 46 us for one, in dense loops over integer coefficients, in a temperature iteration that re-reads
// and re-sums the species' polynomials, and in triangular solves on one lane.  Here
//   - a lane keeps the constants of its reaction in registers and reads concentrations and g/(RT) by
//     species lists from shared memory;
//   - the sums over reactions are spread over 32 / NS lanes per species;
//   - the mixture's polynomial coefficients are formed once per composition, so that an iteration of
//     the temperature is two Horner evaluations;
//   - a lane holds a row of the matrix; elimination and substitutions broadcast by shuffles.
// 1024 H2/air reactors, 24 attempts: 46 -> 19 us per attempt.
#pragma once
#include "chem_tab.cuh"
#include "rcp.cuh"
#include "thermo.cuh"

namespace cb2 {

constexpr unsigned kFullWarp = 0xffffffffu;

template <int NS>
struct RokTables {  // per CTA
  ChemReac<NS> r[kChemTabReac];
  double gib[2][NS][7];   // g/(RT) coefficients of both ranges
  double th[2][11][NS];   // h: a0, c0, a1 .. a4; cp: c1 .. c4 (with c0); 1/W
};

template <int NS>
struct RokWarp {
  double c[NS + 1], g[NS + 1], yk[NS], co[12];
  double q1[kChemTabReac], q2[kChemTabReac];
  double D[kChemTabReac][NS];
};

// The constants of one lane's reaction.
struct RokLane {
  double A, b, Ea, A2, b2, Ea2, order, order_ln;
  unsigned fl, bl;
  int type, back;
};

// Net rates omega [kg/(m^3 s)] of the state y (lane s: partial density of species s) at t; q1, q2 of
// every reaction stay in W.  nu: this lane's share of the coefficients of species lane % NS.
template <int NS>
__device__ __noinline__ double rok_source(double t, double y, const RokLane &L, const ChemHead<NS> &m,
                                          const RokTables<NS> &tab, RokWarp<NS> &W, int lane) {
  constexpr int P = 32 / NS;                       // lanes per species
  constexpr int K = (kChemTabReac + P - 1) / P;    // reactions per lane
  const double lnt = log(t), it = 1.0 / t;
  if (lane < NS) {
    W.c[lane] = y * tab.th[0][10][lane] * 1e-3;
    double tt = t, lt = lnt, itt = it;
    bool low = t < m.tm[lane];
    if (t < m.tl[lane] || t > m.th[lane]) {
      low = t < m.tl[lane];
      tt = low ? m.tl[lane] : m.th[lane];
      lt = log(tt);
      itt = 1.0 / tt;
    }
    const double *a = tab.gib[low ? 0 : 1][lane];
    W.g[lane] = fma(-tt, fma(tt, fma(tt, fma(tt, a[4], a[3]), a[2]), a[1]), fma(a[0], 1.0 - lt, fma(a[5], itt, -a[6])));
  }
  __syncwarp();
  if (lane < m.n_reac) {
    const ChemReac<NS> &x = tab.r[lane];
    const int ty = L.type;
    double kf = L.A * exp(fma(L.b, lnt, -L.Ea * it));
    const double kl = L.A2 * exp(fma(L.b2, lnt, -L.Ea2 * it));
    double cc = 0;
    if (ty > 3) {
#pragma unroll
      for (int s = 0; s < NS; ++s) cc = fma(W.c[s], x.tb[s], cc);
      if (ty == 4) {
        kf *= cc;
      } else if (kf < 1e-25 && kl < 1e-25) {
        kf = 0;
      } else {
        const double pr = kl * cc / kf;
        double F = 1.0;
        if (ty > 5) {
          double fc = (1 - x.alpha) * exp(-t * x.it3) + x.alpha * exp(-t * x.it1);
          if (ty == 7) fc += exp(-x.t2 * it);
          constexpr double log10e = 0.43429448190325182765;
          const double lnf = log(fc), lfc = lnf * log10e;
          const double cq = -0.4 - 0.67 * lfc, nq = 0.75 - 1.27 * lfc;
          const double lp = fma(log(pr), log10e, cq);
          const double tmp = lp / (nq - 0.14 * lp);
          F = exp(lnf / (1.0 + tmp * tmp));
        }
        kf = kf * pr / (1.0 + pr) * F;
      }
    } else if (ty == 3) {
      kf += kl;
    }
    double dg = fma(L.order, lnt, -L.order_ln), pf = 1.0, pb = 1.0;
    unsigned fl = L.fl, bl = L.bl;
    for (int a = 0; a < m.list_len; ++a, fl >>= 4, bl >>= 4) {
      const int f = fl & 15u, b = bl & 15u;
      dg += W.g[b] - W.g[f];
      pf *= W.c[f];
      pb *= W.c[b];
    }
    double kb = 0;
    if (L.back == kBackEquilibrium) kb = kf * exp(dg);
    else if (L.back == kBackArrhenius) kb = ty == 4 ? kl * cc : kl;
    W.q1[lane] = kf * pf;
    W.q2[lane] = kb * pb;
  }
  __syncwarp();
  const int s = lane % NS, part = lane / NS;
  double v = 0;
  if (part < P) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int r = part + P * i;
      if (r < m.n_reac) v = fma(W.q1[r] - W.q2[r], tab.r[r].nu[s], v);
    }
  }
  double sum = v;
#pragma unroll
  for (int q = 1; q < P; ++q) sum += __shfl_sync(kFullWarp, v, s + q * NS);
  return sum * m.w[s];
}

// h and cp sums of the composition W.yk at t, each species' own fit (outside the common range).
template <int NS>
__device__ __noinline__ void rok_h_cp_any(double t, const Mech &mech, const RokWarp<NS> &W, int lane, double &ht,
                                          double &cpt) {
  double h = 0, cp = 0;
  if (lane < NS) {
    Mech o = mech;
    o.tab.use = 0;
    o.t_low += lane; o.t_mid += lane; o.t_high += lane;
    o.lo += 7 * lane; o.hi += 7 * lane;
    o.gas_const += lane;
    species_h_cp<1>(t, o, &h, &cp);
    h *= W.yk[lane];
    cp *= W.yk[lane];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    h += __shfl_xor_sync(kFullWarp, h, o);
    cp += __shfl_xor_sync(kFullWarp, cp, o);
  }
  ht = h;
  cpt = cp;
}

// Newton T from the internal energy E of the partial densities y (lane s) at density rho, from t0:
// |1 - T1/T| <= 1e-8, at most 100 iterations.  imw receives sum Y/W.
template <int NS>
__device__ __noinline__ double rok_temperature(double t0, double y, double irho, double E, const Mech &mech,
                                               const RokTables<NS> &tab, RokWarp<NS> &W, int lane, double &imw) {
  __syncwarp();
  if (lane < NS) W.yk[lane] = y * irho;
  __syncwarp();
  double t = t0, err = 1e+6, R = 0;
  double h0, c0, a1, a2, a3, a4, c1, c2, c3, c4;
  int range = -1;
  for (int iter = 0; err > 1e-8 && iter < 100; ++iter) {
    const int want = t < mech.tab.cut[0] ? 0 : 1;
    if (want != range) {
      range = want;
      __syncwarp();
      if (lane < 11) {
        double v = 0;
#pragma unroll
        for (int s = 0; s < NS; ++s) v = fma(W.yk[s], tab.th[range][lane][s], v);
        W.co[lane] = v;
      }
      __syncwarp();
      h0 = W.co[0]; c0 = W.co[1]; a1 = W.co[2]; a2 = W.co[3]; a3 = W.co[4]; a4 = W.co[5];
      c1 = W.co[6]; c2 = W.co[7]; c3 = W.co[8]; c4 = W.co[9];
      imw = W.co[10];
      R = kRu * imw;
    }
    double ht, cpt;
    if (t >= mech.tab.t_low && t <= mech.tab.t_high) {
      ht = fma(t, fma(t, fma(t, fma(t, fma(t, a4, a3), a2), a1), c0), h0);
      cpt = fma(t, fma(t, fma(t, fma(t, c4, c3), c2), c1), c0);
    } else {
      rok_h_cp_any<NS>(t, mech, W, lane, ht, cpt);
    }
    const double t1 = t - (fma(-R, t, ht) - E) / (cpt - R);
    err = fabs(1 - t1 / t);
    t = t1;
  }
  return t;
}

// Rows of a matrix on lanes 0 .. N-1, factored by elimination with row pivoting.  Rows stay on their
// lanes; piv[n] is the lane whose row was taken at step n, rinv[n] the reciprocal of its pivot (on
// every lane), l[n] this lane's multiplier of step n.
template <int N>
struct RokLU {
  double a[N], l[N], rinv[N];
  int piv[N];
  int step;  // the step at which this lane's row was taken

  __device__ __forceinline__ void factor(int lane) {
    bool used = lane >= N;
    step = N;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      // the largest |a| by its leading bits (15 of the mantissa); ties go to the lowest lane
      const unsigned key = used ? 0u : (((unsigned)__double2hiint(fabs(a[n])) & ~31u) | (31u - lane)) | 1u << 31;
      const unsigned best = __reduce_max_sync(kFullWarp, key);
      const int p = 31 - (int)(best & 31u);
      piv[n] = p;
      if (lane == p) {
        used = true;
        step = n;
      }
      rinv[n] = recip(__shfl_sync(kFullWarp, a[n], p));
      l[n] = used ? 0.0 : a[n] * rinv[n];
#pragma unroll
      for (int j = n + 1; j < N; ++j) {
        const double pj = __shfl_sync(kFullWarp, a[j], p);
        a[j] = fma(-l[n], pj, a[j]);
      }
    }
  }

  // lane s < N: component s of the solution for the right-hand side b (lane r: row r)
  __device__ __forceinline__ double solve(double b, int lane) const {
#pragma unroll
    for (int n = 0; n < N; ++n) b = fma(-l[n], __shfl_sync(kFullWarp, b, piv[n]), b);
    double x = 0;
#pragma unroll
    for (int n = N - 1; n >= 0; --n) {
      const double xn = __shfl_sync(kFullWarp, b * rinv[n], piv[n]);
      if (lane == n) x = xn;
      if (step < n) b = fma(-a[n], xn, b);
    }
    return x;
  }
};

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullWarp, v, o);
  return v;
}

template <int NS>
__global__ void __launch_bounds__(32 * kReactorWarps, 3)
k_reactor_rok4e(cb2_reactor *R, int n, const __grid_constant__ Mech mech, const __grid_constant__ ChemHead<NS> m,
                const ChemReac<NS> *rows, int max_attempts, double rtol, double atol) {
  using namespace rok4e;
  constexpr int P = 32 / NS, CPL = (NS + P - 1) / P;  // lanes per species; columns per lane in the Jacobian
  __shared__ RokTables<NS> tab;
  __shared__ RokWarp<NS> warps[kReactorWarps];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  {
    const double2 *src = reinterpret_cast<const double2 *>(rows);
    double2 *dst = reinterpret_cast<double2 *>(tab.r);
    for (int e = tid; e < m.n_reac * (int)(sizeof(ChemReac<NS>) / sizeof(double2)); e += 32 * kReactorWarps)
      dst[e] = __ldg(src + e);
    for (int e = tid; e < 2 * NS * 7; e += 32 * kReactorWarps) (&tab.gib[0][0][0])[e] = (&m.g[0][0][0])[e];
    for (int e = tid; e < 2 * NS; e += 32 * kReactorWarps) {
      const int h = e / NS, s = e % NS;
      const double *a = mech.tab.h[h][s], *c = mech.tab.cp[h][s];
      const double v[11] = {a[0], c[0], a[1], a[2], a[3], a[4], c[1], c[2], c[3], c[4], __ldg(mech.imw + s)};
#pragma unroll
      for (int q = 0; q < 11; ++q) tab.th[h][q][s] = v[q];
    }
  }
  __syncthreads();
  const int id = blockIdx.x * kReactorWarps + wid;
  if (id >= n) return;  // warp-uniform; no CTA barrier follows
  RokWarp<NS> &W = warps[wid];
  double time = R[id].time, hh = R[id].h, err_last = R[id].err_last, T = R[id].T, pr = R[id].p;
  const double t_end = R[id].t_end;
  int step = R[id].step, n_reject = R[id].n_reject, status = R[id].status;
  if (status || time >= t_end) return;
  const double rho = R[id].rho, E = R[id].E, irho = 1.0 / rho;
  double y = lane < NS ? R[id].rhoY[lane] : 0.0;
  RokLane L{};
  if (lane < m.n_reac) {
    const ChemReac<NS> &x = tab.r[lane];
    L = RokLane{x.A, x.b, x.Ea, x.A2, x.b2, x.Ea2, x.order, x.order_ln, x.flist, x.blist, x.type, x.back};
  }
  if (lane == 0) {
    W.c[NS] = 1.0;
    W.g[NS] = 0.0;
  }
  __syncwarp();
  const int row = lane % NS, part = lane / NS;
  for (int a = 0; a < max_attempts && time < t_end; ++a) {
    const double om = rok_source<NS>(T, y, L, m, tab, W, lane);
    const double h = fmin(hh, t_end - time);
    if (!(h > 0) || !isfinite(h)) {
      status |= CB2_REACTOR_NONPHYSICAL;
      break;
    }
    RokLU<NS> lu;
    {
      // J_rc = 1e3 W_r / (rho Y)_c sum_q nu_qr (f_qc q1 - b_qc q2); columns of absent species are zero
      for (int e = lane; e < m.n_reac * NS; e += 32) {
        const int q = e / NS, c = e - q * NS;
        W.D[q][c] = tab.r[q].f[c] * W.q1[q] - tab.r[q].bk[c] * W.q2[q];
      }
      if (lane < NS) W.yk[lane] = y > 1e-30 ? 1.0 / y : 0.0;
      __syncwarp();
      double J[CPL];
#pragma unroll
      for (int q = 0; q < CPL; ++q) J[q] = 0;
      if (part < P) {
        for (int q = 0; q < m.n_reac; ++q) {
          const double nu = tab.r[q].nu[row];
#pragma unroll
          for (int cq = 0; cq < CPL; ++cq) {
            const int c = part * CPL + cq;
            if (c < NS) J[cq] = fma(nu, W.D[q][c], J[cq]);
          }
        }
#pragma unroll
        for (int cq = 0; cq < CPL; ++cq) {
          const int c = part * CPL + cq;
          if (c < NS) J[cq] = -h * gamma * (J[cq] * W.yk[c] * m.w[row]);
        }
      }
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        const double v = __shfl_sync(kFullWarp, J[c % CPL], row + NS * (c / CPL));
        lu.a[c] = lane < NS ? v + (lane == c ? 1.0 : 0.0) : 0.0;
      }
      lu.factor(lane);
    }
    const double k1 = lu.solve(om, lane);
    double imw;
    double ys = fma(h * a21, k1, y);
    double ts = rok_temperature<NS>(T, ys, irho, E, mech, tab, W, lane, imw);
    double f = rok_source<NS>(ts, ys, L, m, tab, W, lane);
    const double c2 = g21 * k1;
    const double k2 = lu.solve(f + c2, lane) - c2;
    ys = fma(h, a31 * k1 + a32 * k2, y);
    ts = rok_temperature<NS>(ts, ys, irho, E, mech, tab, W, lane, imw);
    f = rok_source<NS>(ts, ys, L, m, tab, W, lane);
    const double c3 = g31 * k1 + g32 * k2;
    const double k3 = lu.solve(f + c3, lane) - c3;
    const double c4 = g41 * k1 + g42 * k2 + g43 * k3;  // stage 4 takes the source of stage 3 again
    const double k4 = lu.solve(f + c4, lane) - c4;
    // embedded error estimate and step control
    ys = fma(h, b1 * k1 + b2 * k2 + b4 * k4, y);
    double dy = h * (e1 * k1 + e2 * k2 + e3 * k3 + e4 * k4) / (rtol * ys + atol);
    if (lane >= NS) dy = 0;
    const double err = sqrt(warp_sum_all(dy * dy) / NS);
    double h_next = h;
    // 0.8 err_last^0.1 err^-0.175
    if (step > 0) h_next *= fmin(5.0, fmax(0.2, 0.8 * exp(0.1 * log(err_last) - 0.175 * log(err + 1e-20))));
    else if (err > 1) h_next *= 0.2;
    hh = h_next;
    if (err <= 1) {
      if (lane < NS) y = ys;
      time += h;
      err_last = err;
      T = rok_temperature<NS>(T, y, irho, E, mech, tab, W, lane, imw);
      pr = rho * kRu * imw * T;
      ++step;
      if (!(T > 0) || !isfinite(T)) {
        status |= CB2_REACTOR_NONPHYSICAL;
        break;
      }
    } else {
      ++n_reject;
    }
  }
  if (lane < NS) R[id].rhoY[lane] = y;
  if (lane == 0) {
    if (time >= t_end) status |= CB2_REACTOR_DONE;
    R[id].time = time;
    R[id].h = hh;
    R[id].err_last = err_last;
    R[id].T = T;
    R[id].p = pr;
    R[id].step = step;
    R[id].n_reject = n_reject;
    R[id].status = status;
  }
}

}  // namespace cb2
