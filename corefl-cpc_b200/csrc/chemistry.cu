// Explicit finite-rate chemistry source over a block (the launch of finite_rate_chemistry,
// src/FiniteRateChem.cu:1406-1488).  One-temperature NASA7 mechanisms of up to kChemTabReac
// reactions run k_chemistry_tab on a repacked mechanism; the others (NASA9, control temperatures,
// two temperatures, longer mechanisms) run the generic arithmetic of chem.cuh.
#include <algorithm>
#include <cmath>
#include "chem.cuh"
#include "chem_tab.cuh"
#include "launch.h"

namespace cb2 {

constexpr int kChemThreads = 128;

// Bounded to 128 registers (4 CTAs of 128 threads per SM): the 9-species kernel otherwise takes
// 168 and runs 3 CTAs; its latency-bound exponentials gain more from the extra warps than the
// few spills cost (192^3 H2/air box: 27.0 -> 22.7 ms per step).
template <int NS>
__global__ void __launch_bounds__(kChemThreads, 4) k_chemistry(Zone z, Param p) {
  const int i = blockIdx.x * kChemThreads + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= z.mx) return;
  chemistry_point<NS>(z, p, i, j, k);
}

// The arrays the table kernel touches: a small argument beside the table.
struct ChemZone {
  int mx, plane;  // nodes per line and per k plane
  Layout L;
  idx_t sz0;
  const double *bv, *sv, *jac;
  double *dq, *rts;
};

// g/(RT) of every species, each fit evaluated at the edge of its range outside it.
template <int NS>
__device__ __forceinline__ void tab_gibbs(const ChemTab<NS> &m, double t, double lnt, double it, double *g) {
  if (m.same_mid && t >= m.t_in_low && t <= m.t_in_high) {
    const double l1 = 1.0 - lnt;
    if (t < m.t_mid) {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double *c = m.g[0][s];
        g[s] = fma(-t, fma(t, fma(t, fma(t, c[4], c[3]), c[2]), c[1]), fma(c[0], l1, fma(c[5], it, -c[6])));
      }
    } else {
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double *c = m.g[1][s];
        g[s] = fma(-t, fma(t, fma(t, fma(t, c[4], c[3]), c[2]), c[1]), fma(c[0], l1, fma(c[5], it, -c[6])));
      }
    }
  } else {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double tt = t < m.tl[s] ? m.tl[s] : (t > m.th[s] ? m.th[s] : t);
      const double lt = tt == t ? lnt : log(tt);
      // inside the fit the middle decides the range; outside it the edge's own range is taken
      const double *c = m.g[(tt == t ? t < m.tm[s] : t < m.tl[s]) ? 0 : 1][s];
      g[s] = c[0] * (1.0 - lt) - tt * (c[1] + tt * (c[2] + tt * (c[3] + tt * c[4]))) + c[5] / tt - c[6];
    }
  }
}

// The source of one node per thread, J omega_k added to dq and the reaction time scale.
//
// Bound by the FP64 pipe and by issue: 40 exponentials and some 36 products with coefficient rows per
// reaction and node.  Everything about the mechanism is a constant-bank read (the generic kernel spent
// four fifths of its time on loads and integer-to-double conversions), kf / Kc is one exponential
// without a division, Troe's powers of ten are exponentials of natural logarithms.  Sums over species
// run over whole rows: skipping zero coefficients costs more in tests than the operations it saves.
// Only the products of concentrations pick species by number, from shared memory (one column per
// thread, no bank conflicts).  The tile runs along the k plane's nodes, not along one line, so a
// ragged mx leaves no idle threads.  Five CTAs per SM, 96 registers (192^3 H2/air, per step: generic
// kernel 23.0 ms; five CTAs 5.9, four 6.7, three without spills 8.3).
template <int NS>
__global__ void __launch_bounds__(kChemThreads, 5)
k_chemistry_tab(const __grid_constant__ ChemZone z, const __grid_constant__ ChemTab<NS> m) {
  __shared__ double sc[NS + 1][kChemThreads];
  chain_begin();
  const int tid = threadIdx.x;
  const int q = blockIdx.x * kChemThreads + tid;
  if (q >= z.plane) return;
  const int j = q / z.mx, i = q - j * z.mx, k = blockIdx.y;
  const idx_t gn = z.L.at(i, j, k), sz = z.L.sz;
  const double rho = z.bv[gn], t = z.bv[gn + 5 * sz];
  double c[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) sc[s][tid] = c[s] = rho * z.sv[gn + s * sz] * m.c_per_rho_y[s];
  sc[NS][tid] = 1.0;
  const double lnt = log(t), it = 1.0 / t;
  double g[NS], net[NS], des[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) g[s] = net[s] = des[s] = 0;
  if (m.need_gibbs) tab_gibbs<NS>(m, t, lnt, it, g);
#pragma unroll 1
  for (int r = 0; r < m.n_reac; ++r) {
    const ChemReac<NS> &x = m.r[r];
    const int ty = x.type;
    double kf = x.A * exp(fma(x.b, lnt, -x.Ea * it));
    double cc = 0;
    if (ty > 3) {
#pragma unroll
      for (int s = 0; s < NS; ++s) cc = fma(c[s], x.tb[s], cc);
    }
    if (ty == 3) {
      kf += x.A2 * exp(fma(x.b2, lnt, -x.Ea2 * it));
    } else if (ty == 4) {
      kf *= cc;
    } else if (ty > 4) {
      const double kl = x.A2 * exp(fma(x.b2, lnt, -x.Ea2 * it));
      if (kf < 1e-25 && kl < 1e-25) {
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
    }
    unsigned list = x.flist;
    double q1 = kf * (sc[list & 15u][tid] * sc[list >> 4 & 15u][tid]), q2 = 0;
    if (x.nf > 2) {
#pragma unroll 1
      for (int a = 2; a < x.nf; ++a) q1 *= sc[list >> (4 * a) & 15u][tid];
    }
    if (x.back != kBackNone) {
      if (x.back == kBackEquilibrium) {
        // kb = kf / Kc, Kc = (p_atm / (R_u T) 1e-3)^order exp(-sum nu g/(RT))
        double dg = fma(x.order, lnt, -x.order_ln);
#pragma unroll
        for (int s = 0; s < NS; ++s) dg = fma(g[s], x.nu[s], dg);
        q2 = kf * exp(dg);
      } else {
        q2 = x.A2 * exp(fma(x.b2, lnt, -x.Ea2 * it));
        if (ty == 4) q2 *= cc;
      }
      list = x.blist;
      q2 *= sc[list & 15u][tid] * sc[list >> 4 & 15u][tid];
      if (x.nb > 2) {
#pragma unroll 1
        for (int a = 2; a < x.nb; ++a) q2 *= sc[list >> (4 * a) & 15u][tid];
      }
    }
    const double dq12 = q1 - q2;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      net[s] = fma(dq12, x.nu[s], net[s]);
      des[s] = fma(q1, x.f[s], fma(q2, x.bk[s], des[s]));
    }
  }
  const double jac = z.jac[gn];
  const idx_t g0 = q + (idx_t)k * z.plane;
  double ts = 1e+6;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double od = des[s] * m.w[s], om = net[s] * m.w[s];
    z.dq[g0 + (5 + s) * z.sz0] += jac * om;
    const double y = z.sv[gn + s * sz];
    if (y > 1e-25 && fabs(od) > 1e-25) ts = fmin(ts, fabs(rho * y / od));
  }
  if (z.rts) z.rts[gn] = ts;
}

template <int NS>
static int launch_chemistry_tab(const Zone &z, const ChemTab<NS> &m, cudaStream_t s) {
  ChemZone c{};
  c.mx = z.mx;
  c.plane = z.mx * z.my;
  c.L = z.L;
  c.sz0 = z.L0.sz;
  c.bv = z.bv; c.sv = z.sv; c.jac = z.jac; c.dq = z.dq; c.rts = z.rts;
  const dim3 grid((unsigned)((c.plane + kChemThreads - 1) / kChemThreads), (unsigned)z.mz);
  return launch_chain(k_chemistry_tab<NS>, grid, kChemThreads, 0, s, c, m);
}

int launch_chemistry(const Zone &z, const Param &p, cudaStream_t s, int &n_launch) {
  ProfScope prof("chemistry", s);
  ++n_launch;
  const ChemTabs *tab = p.i_eve < 0 ? p.mech.chem_tabs : nullptr;
  if (tab && tab->ns == 9) return launch_chemistry_tab<9>(z, tab->t9, s);
  if (tab && tab->ns == 5) return launch_chemistry_tab<5>(z, tab->t5, s);
  dim3 grid((z.mx + kChemThreads - 1) / kChemThreads, z.my, z.mz);
  switch (p.n_spec) {
    case 5: k_chemistry<5><<<grid, kChemThreads, 0, s>>>(z, p); break;
    case 9: k_chemistry<9><<<grid, kChemThreads, 0, s>>>(z, p); break;
    default: return CB2_ERR_UNSUPPORTED;
  }
  return check_launch();
}

// ---- repacking (host) --------------------------------------------------------------------------
namespace {

// The species of one side of a reaction, repeated by their coefficients and padded to two; false if
// they do not fit.
bool pack_side(const int *stoi, int ns, unsigned &list, int &n) {
  list = 0;
  n = 0;
  for (int s = 0; s < ns; ++s) {
    if (stoi[s] < 0) return false;
    for (int a = 0; a < stoi[s]; ++a) {
      if (n == kChemTabList) return false;
      list |= (unsigned)s << (4 * n++);
    }
  }
  for (int a = n; a < kChemTabList; ++a) list |= (unsigned)ns << (4 * a);
  n = std::max(n, 2);
  return true;
}

template <int NS>
bool fill_tab(const cb2_mechanism &m, ChemTab<NS> &t) {
  const int nr = m.n_reac;
  t.n_reac = nr;
  t.same_mid = 1;
  t.t_mid = m.t_mid[0];
  t.t_in_low = m.t_low[0];
  t.t_in_high = m.t_high[0];
  for (int s = 0; s < NS; ++s) {
    const double imw = 1.0 / m.mw[s];
    t.c_per_rho_y[s] = imw * 1e-3;
    t.w[s] = 1e+3 / imw;
    t.tl[s] = m.t_low[s]; t.tm[s] = m.t_mid[s]; t.th[s] = m.t_high[s];
    t.t_in_low = std::max(t.t_in_low, t.tl[s]);
    t.t_in_high = std::min(t.t_in_high, t.th[s]);
    if (t.tm[s] != t.t_mid) t.same_mid = 0;
    for (int h = 0; h < 2; ++h) {
      const double *a = (h ? m.high_temp_coeff : m.low_temp_coeff) + 7 * s;
      const double c[7] = {a[0], 0.5 * a[1], a[2] / 6.0, a[3] / 12.0, a[4] / 20.0, a[5], a[6]};
      for (int n = 0; n < 7; ++n) t.g[h][s][n] = c[n];
    }
  }
  for (int r = 0; r < nr; ++r) {
    ChemReac<NS> &x = t.r[r];
    x = ChemReac<NS>{};
    const int ty = m.reac_type[r], rev = m.rev_type[r];
    if (!pack_side(m.stoi_f + r * NS, NS, x.flist, x.nf) || !pack_side(m.stoi_b + r * NS, NS, x.blist, x.nb))
      return false;
    t.list_len = std::max(t.list_len, std::max(x.nf, x.nb));
    for (int s = 0; s < NS; ++s) {
      x.f[s] = m.stoi_f[r * NS + s];
      x.bk[s] = m.stoi_b[r * NS + s];
      x.nu[s] = x.bk[s] - x.f[s];
    }
    x.type = ty;
    x.back = ty == 0 ? kBackNone : rev == 1 ? kBackArrhenius : ty != 2 ? kBackEquilibrium : kBackNone;
    if (x.back == kBackEquilibrium) t.need_gibbs = 1;
    x.A = m.A[r]; x.b = m.b[r]; x.Ea = m.Ea[r];
    auto opt = [&](const double *a) { return a ? a[r] : 0.0; };
    x.A2 = opt(m.A2); x.b2 = opt(m.b2); x.Ea2 = opt(m.Ea2);
    x.order = m.reac_order ? m.reac_order[r] : 0;
    x.order_ln = x.order * std::log(kPatm / kRu * 1e-3);
    if (ty > 5) {
      if (!m.troe_alpha || !m.troe_t3 || !m.troe_t1 || m.troe_t3[r] == 0 || m.troe_t1[r] == 0) return false;
      x.alpha = m.troe_alpha[r];
      x.it3 = 1.0 / m.troe_t3[r];
      x.it1 = 1.0 / m.troe_t1[r];
      x.t2 = opt(m.troe_t2);
    }
    for (int s = 0; s < NS; ++s) x.tb[s] = m.third_body_coeff ? m.third_body_coeff[r * NS + s] : 0.0;
  }
  return true;
}

}  // namespace

template <int NS>
static bool upload_rows(const ChemTab<NS> &t, void *&rows) {
  const size_t bytes = sizeof(ChemReac<NS>) * t.n_reac;
  return cudaMalloc(&rows, bytes) == cudaSuccess &&
         cudaMemcpy(rows, t.r, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
}

ChemTabs *make_chem_tabs(const cb2_mechanism &m) {
  if (m.therm_nasa_7_9 == 9 || m.two_temperature_reaction_temperature || m.n_reac < 1 || m.n_reac > kChemTabReac ||
      !m.reac_type || !m.rev_type || !m.stoi_f || !m.stoi_b || !m.A || !m.b || !m.Ea)
    return nullptr;
  ChemTabs *t = new ChemTabs{};
  const bool ok = m.n_spec == 5 ? fill_tab<5>(m, t->t5) && upload_rows(t->t5, t->rows)
                                : m.n_spec == 9 && fill_tab<9>(m, t->t9) && upload_rows(t->t9, t->rows);
  if (ok) {
    t->ns = m.n_spec;
    return t;
  }
  cudaGetLastError();  // without a table the generic kernels run
  free_chem_tabs(t);
  return nullptr;
}

void free_chem_tabs(ChemTabs *t) {
  if (!t) return;
  cudaFree(t->rows);
  delete t;
}

}  // namespace cb2
