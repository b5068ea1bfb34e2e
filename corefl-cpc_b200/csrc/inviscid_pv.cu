// Plain-form (FP64) air instantiations of the primitive-variable sweep and the precision dispatch.
// The kernels and Riemann solvers live in inviscid_pv.cuh; the FP32 (mixed-form) instantiations
// are compiled in inviscid_pv_f32.cu.
#include "inviscid_pv_f64.cuh"

namespace cb2 {

int launch_inviscid_pv(const Zone &z, const Param &p, cudaStream_t s, int &n_launch) {
  if (p.precision == CB2_PREC_MIXED) return launch_inviscid_pv_f32(z, p, s, n_launch);
  if (p.i_eve >= 0) {
    switch (p.n_spec) {
      case 5: return launch_inviscid_pv_2t5(z, p, s, n_launch);
      case 9: return launch_inviscid_pv_2t9(z, p, s, n_launch);
      default: return CB2_ERR_UNSUPPORTED;
    }
  }
  switch (p.n_spec) {
    case 0: return launch_pv_ns<0>(z, p, s, n_launch);
    case 5: return launch_inviscid_pv_mix5(z, p, s, n_launch);
    case 9: return launch_inviscid_pv_mix9(z, p, s, n_launch);
    default: return CB2_ERR_UNSUPPORTED;
  }
}

}  // namespace cb2
