// kernels_loss_bf16.cu -- see loss_instances.cuh.
#include "loss_instances.cuh"

namespace dsgdpp {

void* loss_kernel_bf16(LossShape s, bool mask) {
  return mask ? loss_instance<__nv_bfloat16, true>(s) : loss_instance<__nv_bfloat16, false>(s);
}

}  // namespace dsgdpp
