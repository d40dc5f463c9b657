// kernels_loss_bf16_long.cu -- see loss_instances.cuh.
#define DSGDPP_LONG_ROWS
#include "loss_instances.cuh"

namespace dsgdpp {

void* loss_kernel_bf16_long(LossShape s, bool mask) {
  return mask ? loss_instance<__nv_bfloat16, true>(s) : loss_instance<__nv_bfloat16, false>(s);
}

}  // namespace dsgdpp
