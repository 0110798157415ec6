// Instances of fwd_tma_kernel for rank-1 contexts, four directions and no saved indices: one per stride of rows padded to
// a multiple of four.
#include "mp_fwd_tma.cuh"

namespace mpl {

namespace {

template <int LRT = 4>
cudaError_t launch_stride(const FwdParams& p, int dir, int stages, cudaStream_t st) {
  if constexpr (LRT > 32) {
    return cudaErrorNotSupported;
  } else {
    return p.ls == LRT ? launch_tma_d<LRT <= 16 ? 16 : 32, 0, false, 4, false, true, LRT>(p, dir, stages, st)
                       : launch_stride<LRT + 4>(p, dir, stages, st);
  }
}

}  // namespace

// Strides 4, 8 .. 32.
cudaError_t launch_forward_tma_stride(const FwdParams& p, int dir, int stages, cudaStream_t st) {
  return launch_stride(p, dir, stages, st);
}

}  // namespace mpl
