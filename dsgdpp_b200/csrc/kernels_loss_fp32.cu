// kernels_loss_fp32.cu -- see loss_instances.cuh.
#include "loss_instances.cuh"

namespace dsgdpp {

void* loss_kernel_fp32(LossShape s, bool mask) {
  return mask ? loss_instance<float, true>(s) : loss_instance<float, false>(s);
}

}  // namespace dsgdpp
