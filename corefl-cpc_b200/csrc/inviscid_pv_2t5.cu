#include "inviscid_pv_f64.cuh"

namespace cb2 {

int launch_inviscid_pv_2t5(const Zone &z, const Param &p, cudaStream_t s, int &n) { return launch_pv_2t<6>(z, p, s, n); }

}  // namespace cb2
