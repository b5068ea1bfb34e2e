// Batched closed blocks: many 2-D / 3-D blocks of uneven size advanced by whole SSP-RK3 steps.  Every
// phase of a step runs over the tiles or nodes of all blocks in one launch, with the block path's
// per-node functions (the sweep tiles of inviscid_pv.cuh, stage_update_point, the periodic pair items
// of boundary.cuh, properties_point), and the phases follow one another in the block path's order
// (RK3<mix>, src/RK.cuh:107-237 for an inviscid air case with periodic faces), so a block's results
// are bitwise those of cb2_rk3_step on it.
//
// The blocks differ in size (a factor of 37 between 12^3 and 40^3 nodes), so one thread-block cluster
// per block left most of the GPU waiting for the largest: 96 such blocks, 1.7 M nodes, took 15.4 ms for
// two steps.  With the tiles of all blocks in one grid the work is even whatever the sizes; the price
// is a launch per phase (26 per step).
#include <algorithm>
#include <vector>
#include "point.cuh"
#include "inviscid_pv.cuh"
#include "boundary.cuh"
#include "sweep.cuh"
#include "block_batch.h"

namespace cb2 {

namespace {

constexpr int kBatchThreads = 256;

// Work item of a CTA: its block and its number among the block's CTAs of this phase.
struct BatchItem {
  int c, t;
};
__device__ __forceinline__ BatchItem batch_item(const int *owner, const int *first) {
  const int c = owner[blockIdx.x];
  return {c, (int)blockIdx.x - first[c]};
}

// The context's settings as one block of the batch sees them.
__device__ __forceinline__ Param block_param(const Param &p0, const Zone &z, BlockState *st) {
  Param p = p0;
  p.dim = z.mz == 1 ? 2 : 3;
  p.status = &st->flags;
  return p;
}

__global__ void k_batch_owner(const int *first, int n, int total, int *owner) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  int lo = 0, hi = n - 1;  // the last block whose first tile is <= t
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (first[mid] <= t) lo = mid; else hi = mid - 1;
  }
  owner[t] = lo;
}

// Closes the step just taken (if any) and opens the next one; all: for every block, whether or not it
// has reached its end time (a residual to be timed).
__global__ void k_batch_step(BlockState *state, int n, int close, int all, int *n_active) {
  chain_begin();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  BlockState &s = state[c];
  if (close && s.active) {
    if (s.bad) {
      s.status |= CB2_BLOCK_FAILED;
    } else {
      const double dt = __longlong_as_double((long long)s.dt_bits);
      s.time += dt;
      s.last_dt = dt;
      ++s.steps;
    }
  }
  s.active = all || (!(s.status & CB2_BLOCK_FAILED) && s.time < s.t_end);
  s.bad = 0;
  s.dt_bits = (unsigned long long)__double_as_longlong(s.dt_fixed > 0 ? s.dt_fixed : 1e+6);
  if (s.active) atomicAdd(n_active, 1);
}

// qn <- cv of the padded block, and the CFL step's minimum over its interior nodes.
__global__ void __launch_bounds__(kBatchThreads) k_batch_head(const BlockCase *cases, BlockState *state, const int *owner,
                                                              const int *first, const __grid_constant__ Param p0) {
  chain_begin();
  const BatchItem it = batch_item(owner, first);
  BlockState &st = state[it.c];
  if (!st.active) return;
  const Zone &z = cases[it.c].z;
  const long long e = (long long)it.t * kBatchThreads + threadIdx.x;
  const int g = z.ngg, px = z.mx + 2 * g, py = z.my + 2 * g;
  const idx_t sz = z.L.sz;
  double m = 1e+6;
  bool bad = false;
  if (e < sz) {
#pragma unroll
    for (int l = 0; l < 5; ++l) z.qn[e + l * sz] = z.cv[e + l * sz];
    const int i = (int)(e % px) - g;
    const long long r = e / px;
    const int j = (int)(r % py) - g, k = (int)(r / py) - g;
    if (!(st.dt_fixed > 0) && i >= 0 && i < z.mx && j >= 0 && j < z.my && k >= 0 && k < z.mz) {
      m = local_dt_point<0>(z, block_param(p0, z, &st), i, j, k);
      bad = !(m > 0) || !isfinite(m);
      if (bad) m = 1e+6;
    }
  }
  if (st.dt_fixed > 0) return;
  if (bad) st.bad = 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m < 1e+6) atomicMin(&st.dt_bits, (unsigned long long)__double_as_longlong(m));
}

// One sweep tile; the x sweep, the residual's first term, assigns dq (Param::assign_x).
template <int DIR, int REC, int SOLVER, int NI>
__global__ void __launch_bounds__(kSweepThreads, 4) k_batch_sweep(const BlockCase *cases, BlockState *state, const int *owner,
                                                               const int *first, const __grid_constant__ Param p0) {
  constexpr int TB = kSweepThreads;  // small blocks: 32 nodes along y, z at the default width
  extern __shared__ __align__(16) unsigned char bb_smem[];
  chain_begin();
  const BatchItem it = batch_item(owner, first);
  BlockState &st = state[it.c];
  if (!st.active || st.bad) return;
  const Zone z = cases[it.c].z;
  const Param p = block_param(p0, z, &st);
  if constexpr (DIR == 0) {
    const idx_t run = (idx_t)z.L.my * z.L.disp2;
    const int ntx = (int)((run + (TB - 2) - 1) / (TB - 2));
    pv_tile<double, 0, 0, REC, SOLVER, kNI, false, false, TB>(z, p, run, it.t % ntx, 0, it.t / ntx, bb_smem);
  } else {
    constexpr int NSW = TB / NI;
    const int nit = (z.mx + NI - 1) / NI, ms = DIR == 1 ? z.my : z.mz, nst = (ms + NSW - 3) / (NSW - 2);
    const int bx = it.t % nit, r = it.t / nit;
    pv_tile<double, 0, DIR, REC, SOLVER, NI, false, false, TB>(z, p, 0, bx, r % nst, r / nst, bb_smem);
  }
}

__global__ void __launch_bounds__(kBatchThreads) k_batch_update(const BlockCase *cases, BlockState *state, const int *owner,
                                                                const int *first, const __grid_constant__ Param p0, int rk) {
  chain_begin();
  const BatchItem it = batch_item(owner, first);
  BlockState &st = state[it.c];
  if (!st.active || st.bad) return;
  const Zone &z = cases[it.c].z;
  const long long e = (long long)it.t * kBatchThreads + threadIdx.x;
  if (e >= z.L0.sz) return;
  const int i = (int)(e % z.mx), r = (int)(e / z.mx);
  stage_update_point<0>(z, block_param(p0, z, &st), __longlong_as_double((long long)st.dt_bits), rk, i, r % z.my,
                        r / z.my);
}

__global__ void __launch_bounds__(kBatchThreads) k_batch_faces(const BlockCase *cases, BlockState *state, const int *owner,
                                                               const int *first, const __grid_constant__ Param p0, int d) {
  chain_begin();
  const BatchItem it = batch_item(owner, first);
  BlockState &st = state[it.c];
  if (!st.active || st.bad) return;
  const Zone &z = cases[it.c].z;
  bc_periodic_pair_item<0>(z, block_param(p0, z, &st), cases[it.c].pairs[d],
                           (long long)it.t * kBatchThreads + threadIdx.x);
}

__global__ void __launch_bounds__(kBatchThreads) k_batch_columns(const BlockCase *cases, BlockState *state, const int *owner,
                                                                 const int *first, const __grid_constant__ Param p0) {
  chain_begin();
  const BatchItem it = batch_item(owner, first);
  BlockState &st = state[it.c];
  if (!st.active || st.bad) return;
  const Zone &z = cases[it.c].z;
  const int g = z.ngg, px = z.mx + 2 * g, py = z.my + 2 * g;
  const long long e = (long long)it.t * kBatchThreads + threadIdx.x;
  if (e >= (long long)px * py) return;
  eliminate_k_gradient_point(z, block_param(p0, z, &st), (int)(e % px) - g, (int)(e / px) - g);
}

__global__ void __launch_bounds__(kBatchThreads) k_batch_properties(const BlockCase *cases, BlockState *state,
                                                                    const int *owner, const int *first,
                                                                    const __grid_constant__ Param p0) {
  chain_begin();
  const BatchItem it = batch_item(owner, first);
  BlockState &st = state[it.c];
  if (!st.active || st.bad) return;
  const Zone &z = cases[it.c].z;
  if (p0.mu_constant > 0 && !z.mach) return;  // nothing changes
  const int g = z.ngg, px = z.mx + 2 * g, py = z.my + 2 * g;
  const long long e = (long long)it.t * kBatchThreads + threadIdx.x;
  if (e >= z.L.sz) return;
  const long long r = e / px;
  properties_point<0>(z, block_param(p0, z, &st), (int)(e % px) - g, (int)(r % py) - g, (int)(r / py) - g);
}

// first: prefix sums on the host; off(ph): where phase ph's owners start.
struct Batch {
  const BatchStore &b;
  int n;
  const std::vector<int> &first;
  cudaStream_t s;
  int &nl;
  int count(int ph) const { return first[(size_t)ph * (n + 1) + n]; }
  const int *dfirst(int ph) const { return b.first + (size_t)ph * (n + 1); }
  const int *owner(int ph) const {
    long long o = 0;
    for (int q = 0; q < ph; ++q) o += count(q);
    return b.owner + o;
  }
};

template <int DIR, int REC, int SOLVER, int NI>
int sweep(const Batch &t, const Param &p) {
  const int ph = DIR == 0 ? kTilesX : (DIR == 1 ? kTilesY : kTilesZ);
  if (!t.count(ph)) return CB2_OK;
  const size_t smem = pv_tile_smem<double, 0, REC, SOLVER, false, kSweepThreads>(DIR, NI);
  auto kern = k_batch_sweep<DIR, REC, SOLVER, NI>;
  CB2_TRY(prepare_smem(kern, smem));
  ++t.nl;
  return launch_chain(kern, t.count(ph), kSweepThreads, smem, t.s, (const BlockCase *)t.b.cases, t.b.state, t.owner(ph),
                      t.dfirst(ph), p);
}

template <int REC, int SOLVER, int NI>
int residual(const Batch &t, const Param &p) {
  CB2_TRY((sweep<0, REC, SOLVER, kNI>(t, p)));
  CB2_TRY((sweep<1, REC, SOLVER, NI>(t, p)));
  return sweep<2, REC, SOLVER, NI>(t, p);
}

constexpr int kCheckSteps = 16;  // steps between looks at whether any block still runs

template <int REC, int SOLVER, int NI>
int run(const Batch &t, const Param &p0, int max_steps, int mode) {
  const BatchStore &b = t.b;
  Param p = p0;
  p.assign_x = 1;
  const int T = kBatchThreads, nb = (t.n + T - 1) / T;
  auto open = [&](int close) {
    CB2_TRY(check_cuda(cudaMemsetAsync(b.n_active, 0, sizeof(int), t.s)));
    CB2_TRY(launch_chain(k_batch_step, nb, T, 0, t.s, b.state, t.n, close, mode == 1 ? 1 : 0, b.n_active));
    ++t.nl;
    return check_launch();
  };
  CB2_TRY(open(0));
  if (mode == 1) return residual<REC, SOLVER, NI>(t, p);
  for (int step = 0; step < max_steps; ++step) {
    if (step > 0 && step % kCheckSteps == 0) {
      int active = 0;
      CB2_TRY(check_cuda(cudaMemcpyAsync(&active, b.n_active, sizeof(int), cudaMemcpyDeviceToHost, t.s)));
      CB2_TRY(check_cuda(cudaStreamSynchronize(t.s)));
      if (!active) break;
    }
    CB2_TRY(launch_chain(k_batch_head, t.count(kPadded), T, 0, t.s, (const BlockCase *)b.cases, b.state, t.owner(kPadded), t.dfirst(kPadded), p));
    ++t.nl;
    CB2_TRY(check_launch());
    for (int rk = 0; rk < 3; ++rk) {
      CB2_TRY((residual<REC, SOLVER, NI>(t, p)));
      CB2_TRY(launch_chain(k_batch_update, t.count(kNodes), T, 0, t.s, (const BlockCase *)b.cases, b.state, t.owner(kNodes), t.dfirst(kNodes), p, rk));
      ++t.nl;
      for (int d = 0; d < 3; ++d) {
        const int ph = kFacesX + d;
        if (!t.count(ph)) continue;
        CB2_TRY(launch_chain(k_batch_faces, t.count(ph), T, 0, t.s, (const BlockCase *)b.cases, b.state, t.owner(ph), t.dfirst(ph), p, d));
        ++t.nl;
      }
      if (t.count(kColumns)) {
        CB2_TRY(launch_chain(k_batch_columns, t.count(kColumns), T, 0, t.s, (const BlockCase *)b.cases, b.state, t.owner(kColumns), t.dfirst(kColumns), p));
        ++t.nl;
      }
      CB2_TRY(launch_chain(k_batch_properties, t.count(kPadded), T, 0, t.s, (const BlockCase *)b.cases, b.state, t.owner(kPadded), t.dfirst(kPadded), p));
      ++t.nl;
      CB2_TRY(check_launch());
    }
    CB2_TRY(open(1));
  }
  return CB2_OK;
}

template <int REC, int SOLVER>
int run_ni(const Batch &t, const Param &p, int max_steps, int mode, int ni) {
  if (ni == 4) return run<REC, SOLVER, 4>(t, p, max_steps, mode);
  if (ni == 16) return run<REC, SOLVER, 16>(t, p, max_steps, mode);
  return run<REC, SOLVER, 8>(t, p, max_steps, mode);
}

}  // namespace

bool batch_layout(const std::vector<BlockCase> &cases, int ni, std::vector<int> &first) {
  const int n = (int)cases.size();
  first.assign((size_t)kBatchPhases * (n + 1), 0);
  long long total[kBatchPhases] = {};
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  for (int c = 0; c < n; ++c) {
    const Zone &z = cases[c].z;
    const int g = z.ngg, nsw = kSweepThreads / ni;
    const long long px = z.mx + 2 * g, py = z.my + 2 * g;
    const long long pairs[3] = {(long long)z.my * z.mz, (long long)z.mx * z.mz, (long long)z.mx * z.my};
    long long k[kBatchPhases];
    k[kTilesX] = up((long long)z.my * z.L.disp2, kSweepThreads - 2) * z.mz;
    k[kTilesY] = up(z.mx, ni) * up(z.my, nsw - 2) * z.mz;
    k[kTilesZ] = z.mz > 1 ? up(z.mx, ni) * up(z.mz, nsw - 2) * z.my : 0;
    k[kNodes] = up(z.L0.sz, kBatchThreads);
    k[kPadded] = up(z.L.sz, kBatchThreads);
    for (int d = 0; d < 3; ++d) k[kFacesX + d] = d < 2 || z.mz > 1 ? up((2 * g + 1) * pairs[d], kBatchThreads) : 0;
    k[kColumns] = z.mz == 1 ? up(px * py, kBatchThreads) : 0;
    for (int ph = 0; ph < kBatchPhases; ++ph) {
      total[ph] += k[ph];
      if (total[ph] > 0x7fffffffLL) return false;
      first[(size_t)ph * (n + 1) + c + 1] = (int)total[ph];
    }
  }
  return true;
}

int launch_batch_owners(const BatchStore &b, int n, const std::vector<int> &first, cudaStream_t s, int &n_launch) {
  const Batch t{b, n, first, s, n_launch};
  for (int ph = 0; ph < kBatchPhases; ++ph) {
    if (!t.count(ph)) continue;
    k_batch_owner<<<(t.count(ph) + 255) / 256, 256, 0, s>>>(t.dfirst(ph), n, t.count(ph), const_cast<int *>(t.owner(ph)));
    ++n_launch;
  }
  return check_launch();
}

bool block_batch_supported(const Param &p) {
  return p.n_spec == 0 && p.i_eve < 0 && p.viscous_order == 0 && p.precision == CB2_PREC_FP64 && !p.limit_flow &&
         (p.reconstruction == CB2_REC_WENO5 || p.reconstruction == CB2_REC_WENO7) &&
         (p.inviscid_scheme == CB2_INV_AUSMP || p.inviscid_scheme == CB2_INV_HLLC);
}

int launch_block_batch(const BatchStore &b, int n, const std::vector<int> &first, const Param &p, int max_steps,
                       int mode, int ni, cudaStream_t s, int &n_launch) {
  if (n <= 0) return CB2_OK;
  if (!block_batch_supported(p)) return CB2_ERR_UNSUPPORTED;
  ProfScope prof(mode == 1 ? "block_batch_residual" : "block_batch", s);
  const Batch t{b, n, first, s, n_launch};
  const bool w7 = p.reconstruction == CB2_REC_WENO7, ausm = p.inviscid_scheme == CB2_INV_AUSMP;
  if (w7 && ausm) return run_ni<7, CB2_INV_AUSMP>(t, p, max_steps, mode, ni);
  if (w7) return run_ni<7, CB2_INV_HLLC>(t, p, max_steps, mode, ni);
  if (ausm) return run_ni<5, CB2_INV_AUSMP>(t, p, max_steps, mode, ni);
  return run_ni<5, CB2_INV_HLLC>(t, p, max_steps, mode, ni);
}

}  // namespace cb2
