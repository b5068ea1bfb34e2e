// Plain-form (FP64) dispatch of the primitive-variable sweep over reconstruction and Riemann solver.
// One translation unit per species count instantiates it (inviscid_pv*.cu), so that they compile
// side by side.
#pragma once
#include "inviscid_pv.cuh"

namespace cb2 {

template <int NS, int SOLVER, bool TT = false>
static int launch_pv_rec(const Zone &z, const Param &p, cudaStream_t s, int &nl) {
  switch (p.reconstruction) {
    case CB2_REC_MUSCL: return launch_pv_dirs<double, NS, 2, SOLVER, TT>(z, p, s, nl);
    case CB2_REC_NND2: return launch_pv_dirs<double, NS, 3, SOLVER, TT>(z, p, s, nl);
    case CB2_REC_WENO5: return launch_pv_dirs<double, NS, 5, SOLVER, TT>(z, p, s, nl);
    case CB2_REC_WENO7: return launch_pv_dirs<double, NS, 7, SOLVER, TT>(z, p, s, nl);
    default: return launch_pv_dirs<double, NS, 1, SOLVER, TT>(z, p, s, nl);
  }
}

// Two temperatures (FP64): AUSM+ and HLLC over the n_spec species and e_ve (NSC = n_spec + 1
// scalars); the reference's two-temperature build has no Roe or Lax-Friedrichs variant.
template <int NSC>
static int launch_pv_2t(const Zone &z, const Param &p, cudaStream_t s, int &nl) {
  switch (p.inviscid_scheme) {
    case CB2_INV_AUSMP: return launch_pv_rec<NSC, CB2_INV_AUSMP, true>(z, p, s, nl);
    case CB2_INV_HLLC: return launch_pv_rec<NSC, CB2_INV_HLLC, true>(z, p, s, nl);
    default: return CB2_ERR_UNSUPPORTED;
  }
}

template <int NS>
static int launch_pv_ns(const Zone &z, const Param &p, cudaStream_t s, int &nl) {
  switch (p.inviscid_scheme) {
    case CB2_INV_AUSMP: return launch_pv_rec<NS, CB2_INV_AUSMP>(z, p, s, nl);
    case CB2_INV_HLLC: return launch_pv_rec<NS, CB2_INV_HLLC>(z, p, s, nl);
    case CB2_INV_ROE: return launch_pv_rec<NS, CB2_INV_ROE>(z, p, s, nl);
    case 1:
      if constexpr (NS == 0) return launch_pv_rec<0, 1>(z, p, s, nl);
      else return CB2_ERR_UNSUPPORTED;
    default: return CB2_ERR_UNSUPPORTED;
  }
}

}  // namespace cb2
