// Instances of fwd_tma_kernel for rank-1 contexts.
#include "mp_fwd_tma.cuh"

namespace mpl {

cudaError_t launch_forward_tma_rank1(const FwdParams& p, int dir, int stages, bool train, cudaStream_t st) {
  return launch_forward_tma_rank<true>(p, dir, stages, train, st);
}

}  // namespace mpl
