// pk_grad_mhd1.cu -- recording and adjoint sweeps for ionized fluid + B + psi.
#include "pk_launch.cuh"

namespace pk {
const GradOps* grad_ops_mhd1() { return make_grad_ops<Phys<K_ION, K_NONE, K_NONE, true>>(); }
}  // namespace pk
