#include "inviscid_pv_f64.cuh"

namespace cb2 {

int launch_inviscid_pv_mix9(const Zone &z, const Param &p, cudaStream_t s, int &n) { return launch_pv_ns<9>(z, p, s, n); }

}  // namespace cb2
