// kernels_loss_fp32_long.cu -- see loss_instances.cuh.
#define DSGDPP_LONG_ROWS
#include "loss_instances.cuh"

namespace dsgdpp {

void* loss_kernel_fp32_long(LossShape s, bool mask) {
  return mask ? loss_instance<float, true>(s) : loss_instance<float, false>(s);
}

}  // namespace dsgdpp
