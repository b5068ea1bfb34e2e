// Physical properties over interior and ghost nodes (update_physical_properties<mix>,
// src/FieldOperation.cuh:183-247), the local CFL time step (local_time_step<mix>,
// src/TimeAdvanceFunc.cuh:28-127) and its global minimum (min_of_arr + global_time_step,
// src/TimeAdvanceFunc.cu:114-164).
#include <algorithm>
#include <cmath>
#include "point.cuh"
#include "launch.h"

namespace cb2 {

constexpr int kPropThreads = 128;
constexpr int kPropTabCtas = 4;  // CTAs per SM of the FP64 transport kernels: 128 registers

// Mixtures whose mechanism is not repacked, and the mixed form.  Bounded to 80 registers (6 CTAs of
// 128 threads per SM; the FP64 9-species transport otherwise takes 163): the exponential and
// logarithm chains are latency-bound (192^3 H2/air box: 29.9 -> 20.7 ms per step).
template <int NS, bool F32T = false>
__global__ void __launch_bounds__(kPropThreads, 6) k_properties(const __grid_constant__ Zone z, const __grid_constant__ Param p) {
  chain_begin();
  const int g_ = z.ngg, px = z.mx + 2 * g_;
  const int q = blockIdx.x * kPropThreads + threadIdx.x;
  if (q >= px * (z.my + 2 * g_)) return;
  const int j = q / px, i = q - j * px;
  properties_point<NS, F32T>(z, p, i - g_, j - g_, (int)blockIdx.y - g_);
}

// FP64 transport on the repacked mechanism (transport_tab.cuh).  A tile runs along the padded k
// plane's nodes, so a ragged line leaves no idle threads; shared memory holds the distinct
// collision integrals of each thread.
template <int NS>
__global__ void __launch_bounds__(kPropThreads, kPropTabCtas)
k_properties_tab(const __grid_constant__ Zone z, const __grid_constant__ Param p, const __grid_constant__ TransTab<NS> m) {
  extern __shared__ double s_om[];
  chain_begin();
  const int g_ = z.ngg, px = z.mx + 2 * g_;
  const int q = blockIdx.x * kPropThreads + threadIdx.x;
  if (q >= px * (z.my + 2 * g_)) return;
  const int j = q / px, i = q - j * px;
  properties_point<NS>(z, p, i - g_, j - g_, (int)blockIdx.y - g_, true, &m, s_om + threadIdx.x, kPropThreads);
}

// A 2-D block (mz = 1) carries ngg ghost planes on each side of its one k plane.  The reference
// evaluates the properties on every one of them (src/RK.cuh:230-235); after eliminate_k_gradient
// their basic and scalar variables are copies of plane 0, so their properties are copies of
// plane 0's, which is how they are filled here: the transport evaluation runs once per (i, j)
// instead of 2 ngg + 1 times.  Only kappa_ve, which also depends on the plane's own T_ve (not
// copied by eliminate_k_gradient), is re-evaluated where that differs.
// Copies of plane 0's properties of column (i, j) on the ghost planes.
template <int NS>
__device__ __forceinline__ void spread_properties(const Zone &z, const Param &p, int i, int j) {
  const int g_ = z.ngg;
  const idx_t sz = z.L.sz, g0 = z.L.at(i, j, 0);
  for (int kk = -g_; kk <= g_; ++kk) {
    if (kk == 0) continue;
    const idx_t gk = z.L.at(i, j, kk);
    z.mul[gk] = z.mul[g0];
    if (z.mach) z.mach[gk] = z.mach[g0];
    if constexpr (NS > 0) {
      z.gamma[gk] = z.gamma[g0];
      z.acoustic[gk] = z.acoustic[g0];
      z.kappa[gk] = z.kappa[g0];
#pragma unroll
      for (int s = 0; s < NS; ++s) z.rhoD[gk + s * sz] = z.rhoD[g0 + s * sz];
      if (p.i_eve >= 0) {
        if (z.tve[gk] <= 0) z.tve[gk] = z.bv[gk + 5 * sz];
        if (z.kappa_ve) {
          const double tk = z.tve[gk];
          if (tk == z.tve[g0]) {
            z.kappa_ve[gk] = z.kappa_ve[g0];
          } else {
            double y[NS], cp[NS], cv_ve, cpt = 0;
#pragma unroll
            for (int s = 0; s < NS; ++s) y[s] = z.sv[gk + s * sz];
            species_cp<NS>(z.bv[gk + 5 * sz], p.mech, cp);
#pragma unroll
            for (int s = 0; s < NS; ++s) cpt = fma(y[s], cp[s], cpt);
            mixture_ve_energy<NS>(tk, y, p.mech, &cv_ve);
            z.kappa_ve[gk] = z.kappa[g0] * cv_ve / fmax(cpt, 1e-8);
          }
        }
      }
    }
  }
}

template <int NS, bool F32T = false>
__global__ void __launch_bounds__(kPropThreads) k_properties_planar(const __grid_constant__ Zone z, const __grid_constant__ Param p) {
  chain_begin();
  const int g_ = z.ngg;
  const int i = blockIdx.x * kPropThreads + threadIdx.x - g_;
  const int j = blockIdx.y - g_;
  if (i >= z.mx + g_) return;
  properties_point<NS, F32T>(z, p, i, j, 0);
  spread_properties<NS>(z, p, i, j);
}

template <int NS>
__global__ void __launch_bounds__(kPropThreads, kPropTabCtas)
k_properties_planar_tab(const __grid_constant__ Zone z, const __grid_constant__ Param p,
                        const __grid_constant__ TransTab<NS> m) {
  extern __shared__ double s_om[];
  chain_begin();
  const int g_ = z.ngg, px = z.mx + 2 * g_;
  const int q = blockIdx.x * kPropThreads + threadIdx.x;
  if (q >= px * (z.my + 2 * g_)) return;
  const int j = q / px, i = q - j * px;
  properties_point<NS>(z, p, i - g_, j - g_, 0, true, &m, s_om + threadIdx.x, kPropThreads);
  spread_properties<NS>(z, p, i - g_, j - g_);
}

template <int NS>
static int launch_properties_tab(const Zone &z, const Param &p, const TransTab<NS> &m, bool planar, cudaStream_t s) {
  const int g = z.ngg;
  const int plane = (z.mx + 2 * g) * (z.my + 2 * g);
  const dim3 grid((unsigned)((plane + kPropThreads - 1) / kPropThreads), (unsigned)(planar ? 1 : z.mz + 2 * g));
  const size_t smem = sizeof(double) * m.n_red * kPropThreads;
  return launch_chain(planar ? k_properties_planar_tab<NS> : k_properties_tab<NS>, grid, kPropThreads, smem, s, z, p, m);
}

int launch_properties(const Zone &z, const Param &p, cudaStream_t s, int &n_launch) {
  const int g = z.ngg;
  const bool planar = z.mz == 1 && p.dim == 2;
  const bool mixed = p.precision == CB2_PREC_MIXED;  // transport in FP32
  const dim3 grid((z.mx + 2 * g + kPropThreads - 1) / kPropThreads, z.my + 2 * g);  // 2-D blocks
  ++n_launch;
  ProfScope prof("properties", s);
  const TransTabs *tab = mixed ? nullptr : p.mech.trans_tabs;
  if (tab && p.n_spec == 9) return launch_properties_tab<9>(z, p, tab->t9, planar, s);
  if (tab && p.n_spec == 5) return launch_properties_tab<5>(z, p, tab->t5, planar, s);
  // nothing changes for air of constant viscosity without a Mach array
  if (p.n_spec == 0 && p.mu_constant > 0 && !z.mach) { --n_launch; return CB2_OK; }
  const int plane = (z.mx + 2 * g) * (z.my + 2 * g);
  const dim3 pgrid((unsigned)((plane + kPropThreads - 1) / kPropThreads), (unsigned)(z.mz + 2 * g));
  auto go = [&](auto flat, auto all) {
    return planar ? launch_chain(flat, grid, kPropThreads, 0, s, z, p) : launch_chain(all, pgrid, kPropThreads, 0, s, z, p);
  };
  switch (p.n_spec) {
    case 0: return go(k_properties_planar<0>, k_properties<0>);
    case 5:
      if (mixed) return go(k_properties_planar<5, true>, k_properties<5, true>);
      return go(k_properties_planar<5>, k_properties<5>);
    case 9:
      if (mixed) return go(k_properties_planar<9, true>, k_properties<9, true>);
      return go(k_properties_planar<9>, k_properties<9>);
    default: return CB2_ERR_UNSUPPORTED;
  }
}

// ---- repacking (host) ----------------------------------------------------------------------
template <int NS>
static bool fill_trans(const cb2_mechanism &m, TransTab<NS> &t) {
  for (int a = 0; a < NS; ++a) {
    t.imw[a] = 1.0 / m.mw[a];
    t.mw[a] = 1.0 / t.imw[a];
    t.gas[a] = kRu / m.mw[a];
    t.vis_coeff[a] = m.vis_coeff[a];
    t.lj_inv[a] = m.LJ_potent_inv[a];
    if (!(t.lj_inv[a] > 0)) return false;
    t.vis_a[a] = 1.147 * std::pow(t.lj_inv[a], -0.145);
    t.geometry[a] = m.geometry[a] == 1 ? 1 : (m.geometry[a] == 2 ? 2 : 0);
    t.zrot_pi[a] = 3.141592653589793 * m.ZRotF298[a];
    t.bdc_r[a] = m.binary_diffusivity_coeff[a * NS + a] / t.gas[a];
    for (int b = 0; b < NS; ++b) {
      const double sq8 = m.sqrt_WiDivWjPl1Mul8[a * NS + b], bdc = m.binary_diffusivity_coeff[a * NS + b];
      if (!(sq8 >= 0) || (a < b && !(bdc > 0))) return false;
      t.sq[a][b] = std::sqrt(sq8);
      t.w14[a][b] = m.WjDivWi_to_One4th[a * NS + b] * t.sq[a][b];
      t.ibdc[a][b] = bdc > 0 ? 1.0 / bdc : 0.0;
    }
  }
  t.n_red = 0;
  for (int a = 0; a < NS; ++a)
    for (int b = a; b < NS; ++b) {
      const double k = m.kb_over_eps_jk[a * NS + b];
      if (!(k > 0)) return false;
      int u = 0;
      while (u < t.n_red && t.kbe[u] != k) ++u;
      if (u == t.n_red) {
        t.kbe[u] = k;
        t.om_a[u] = 1.0548 * std::pow(k, -0.15504);
        ++t.n_red;
      }
      t.pair[a][b] = t.pair[b][a] = u;
      if (a == b) t.kbe_inv[a] = 1.0 / k;
    }
  return true;
}

TransTabs *make_trans_tabs(const cb2_mechanism &m) {
  if (!m.vis_coeff || !m.LJ_potent_inv || !m.geometry || !m.ZRotF298 || !m.binary_diffusivity_coeff ||
      !m.kb_over_eps_jk || !m.sqrt_WiDivWjPl1Mul8 || !m.WjDivWi_to_One4th)
    return nullptr;
  TransTabs *t = new TransTabs{};
  if (m.n_spec == 5 ? fill_trans<5>(m, t->t5) : m.n_spec == 9 && fill_trans<9>(m, t->t9)) {
    t->ns = m.n_spec;
    return t;
  }
  delete t;
  return nullptr;
}

void free_trans_tabs(TransTabs *t) { delete t; }

// ---- local time step and its minimum ------------------------------------------------------
// The smaller of *out and v, exactly and for any sign: bits of non-negative doubles order as signed
// integers, bits of negative ones in reverse as unsigned.
__device__ __forceinline__ void atomic_min_double(double *out, double v) {
  if (v >= 0) atomicMin(reinterpret_cast<long long *>(out), __double_as_longlong(v));
  else atomicMax(reinterpret_cast<unsigned long long *>(out), (unsigned long long)__double_as_longlong(v));
}

// dt of every interior node; the minimum goes to *dt_min (seeded by the caller), one atomic per warp.
// The reference seeds its minimum with 1e+6 (src/TimeAdvanceFunc.cu:152), so a block whose every dt
// exceeds 1e6 reports 1e6; NaN does not count.
template <int NS>
__global__ void __launch_bounds__(kPropThreads) k_local_dt(const __grid_constant__ Zone z, const __grid_constant__ Param p,
                                                           double *dt_min) {
  chain_begin();
  const int i = blockIdx.x * kPropThreads + threadIdx.x;
  const int j = blockIdx.y, k = blockIdx.z;
  double v = 1e+6;
  if (i < z.mx) {
    const double dt = local_dt_point<NS>(z, p, i, j, k);
    z.dtl[z.L0.at(i, j, k)] = dt;
    v = fmin(v, dt);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0 && v < 1e+6) atomic_min_double(dt_min, v);
}

int launch_local_dt(const Zone &z, const Param &p, double *dt_min, cudaStream_t s, int &n_launch) {
  dim3 grid((z.mx + kPropThreads - 1) / kPropThreads, z.my, z.mz);
  ++n_launch;
  ProfScope prof("local_dt", s);
  switch (p.n_spec) {
    case 0: return launch_chain(k_local_dt<0>, grid, kPropThreads, 0, s, z, p, dt_min);
    case 5: return launch_chain(k_local_dt<5>, grid, kPropThreads, 0, s, z, p, dt_min);
    case 9: return launch_chain(k_local_dt<9>, grid, kPropThreads, 0, s, z, p, dt_min);
    default: return CB2_ERR_UNSUPPORTED;
  }
}

__global__ void k_set_value(double *dst, double v) {
  chain_begin();
  *dst = v;
}

int launch_set_value(double *dst, double v, cudaStream_t s, int &n_launch) {
  ++n_launch;
  return launch_chain(k_set_value, 1, 1, 0, s, dst, v);
}

// Grid-stride FP64 -> FP32 conversion (coalesced 8-byte loads and 4-byte stores).
__global__ void k_to_f32(const double *__restrict__ src, float *__restrict__ dst, size_t n) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = (float)src[i];
}

int launch_to_f32(const double *src, float *dst, size_t n, cudaStream_t s, int &n_launch) {
  if (n == 0) return CB2_OK;
  const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 148 * 32);
  k_to_f32<<<blocks, 256, 0, s>>>(src, dst, n);
  ++n_launch;
  return check_launch();
}

}  // namespace cb2

namespace cb2 {

// ---- shock sensor (compute_shock_sensor, src/FieldOperation.cu:123-228) -------------------
// Computed on interior nodes once per step; the ghost values are never written (the
// reference's RK3 loop never exchanges them either), so the caller's zero fill stands there.
__global__ void __launch_bounds__(kPropThreads) k_shock_sensor(Zone z, Param p) {
  const int i = blockIdx.x * kPropThreads + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= z.mx) return;
  const Layout &L = z.L;
  const idx_t sz = L.sz, g = L.at(i, j, k);
  const idx_t st[3] = {1, L.disp2, L.disp1};
  const double *bv = z.bv;
  double sensor = 1;
  if (p.shock_sensor == 1) {  // modified Jameson (src/FieldOperation.cu:172-185)
    const double *pp = bv + 4 * sz + g;
    const double twoP = pp[0] * 2;
    double s = 0;
    for (int a = 0; a < 3; ++a) {
      const double pn = pp[st[a]] + pp[-st[a]];
      s += fabs(pn - twoP) / (pn + twoP);
    }
    sensor = s;
  } else if (p.shock_sensor == 2) {  // density / pressure jump (src/FieldOperation.cu:187-205)
    const double rho = bv[g], rhoI = 1.0 / rho, pr = bv[g + 4 * sz], pI = 1.0 / pr;
    double s = 0;
    for (int a = 0; a < 3; ++a) s = fmax(s, fabs(bv[g + st[a]] - rho) * rhoI);
    for (int a = 0; a < 3; ++a) s = fmax(s, fabs(bv[g + 4 * sz + st[a]] - pr) * pI);
    sensor = s;
  } else {  // modified Ducros (src/FieldOperation.cu:123-170)
    constexpr double c12 = 1.0 / 12.0, c23 = 2.0 / 3.0;
    double d[3][3];  // d[var u,v,w][dir]
    for (int c = 0; c < 3; ++c) {
      const double *f = bv + (1 + c) * sz + g;
      for (int a = 0; a < 3; ++a)
        d[c][a] = c12 * f[-2 * st[a]] - c23 * f[-st[a]] + c23 * f[st[a]] - c12 * f[2 * st[a]];
    }
    const double *M = z.metric + g;
    auto cart = [&](int c, int x) { return d[c][0] * M[x * sz] + d[c][1] * M[(3 + x) * sz] + d[c][2] * M[(6 + x) * sz]; };
    double div = cart(0, 0) + cart(1, 1) + cart(2, 2);
    if (div > 0) sensor = 0;
    else {
      const double duDy = cart(0, 1), duDz = cart(0, 2), dvDx = cart(1, 0), dvDz = cart(1, 2);
      const double dwDx = cart(2, 0), dwDy = cart(2, 1);
      div *= div;
      const double curl2 = (dwDy - dvDz) * (dwDy - dvDz) + (duDz - dwDx) * (duDz - dwDx) + (dvDx - duDy) * (dvDx - duDy);
      sensor = div / (div + curl2 + p.sensor_eps);
    }
  }
  z.shock[g] = sensor;
}

int launch_shock_sensor(const Zone &z, const Param &p, cudaStream_t s, int &n_launch) {
  dim3 grid((z.mx + kPropThreads - 1) / kPropThreads, z.my, z.mz);
  ProfScope prof("shock_sensor", s);
  k_shock_sensor<<<grid, kPropThreads, 0, s>>>(z, p);
  ++n_launch;
  return check_launch();
}

}  // namespace cb2
