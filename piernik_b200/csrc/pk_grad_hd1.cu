// pk_grad_hd1.cu -- recording and adjoint sweeps for one fluid with energy, no B.
#include "pk_launch.cuh"

namespace pk {
const GradOps* grad_ops_hd1() { return make_grad_ops<Phys<K_NEU, K_NONE, K_NONE, false>>(); }
}  // namespace pk
