// loss_instances.cuh -- included by the kernels_loss_*.cu files, each of which
// instantiates the loss kernel for one type and either the mappings of up to
// four lanes (ranks to 128 in FP32) or the longer ones, whose code is several
// times larger.  Each file is a module that a process loads when it first uses
// it, so a run loads the mappings of its own type and length only.
#include "loss_rows.cuh"

namespace dsgdpp {
namespace {

template <typename T, bool MASK>
void* loss_instance(LossShape s) {
#define DSGDPP_CASE(L, V, N) \
  if (s.lanes == L && s.vecs == V && s.words == N) \
    return reinterpret_cast<void*>(&loss_kernel<T, L, V, N, MASK>);
#ifdef DSGDPP_LONG_ROWS
  DSGDPP_CASE(8, 3, 8) DSGDPP_CASE(8, 4, 8) DSGDPP_CASE(16, 3, 8) DSGDPP_CASE(16, 4, 8)
  DSGDPP_CASE(8, 3, 4) DSGDPP_CASE(8, 4, 4) DSGDPP_CASE(16, 3, 4) DSGDPP_CASE(16, 4, 4)
  DSGDPP_CASE(32, 3, 4) DSGDPP_CASE(32, 4, 4)
#else
  DSGDPP_CASE(1, 1, 8) DSGDPP_CASE(2, 1, 8) DSGDPP_CASE(4, 1, 8) DSGDPP_CASE(4, 2, 8)
  DSGDPP_CASE(4, 3, 8) DSGDPP_CASE(4, 4, 8)
  DSGDPP_CASE(1, 1, 4) DSGDPP_CASE(4, 1, 4) DSGDPP_CASE(4, 2, 4) DSGDPP_CASE(4, 3, 4)
  DSGDPP_CASE(4, 4, 4)
#endif
#undef DSGDPP_CASE
  return nullptr;
}

}  // namespace
}  // namespace dsgdpp
