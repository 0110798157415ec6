// Instances of fwd_tma_kernel for rank-1 contexts.
#include "mp_fwd_tma.cuh"

namespace mpl {

cudaError_t launch_forward_tma_stride(const FwdParams& p, int dir, int stages, cudaStream_t st);  // mp_fwd_tma_stride.cu

cudaError_t launch_forward_tma_rank1(const FwdParams& p, int dir, int stages, bool train, cudaStream_t st) {
  // (21 labels have instances of their own)
  if (!train && !p.agg && p.D == 4 && p.L != 21 && (p.ls & 3) == 0 && p.ls <= 32) return launch_forward_tma_stride(p, dir, stages, st);
  return launch_forward_tma_rank<true>(p, dir, stages, train, st);
}

}  // namespace mpl
