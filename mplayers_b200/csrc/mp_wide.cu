// Instances of fwd_wide_kernel without saved indices, and the dispatch (mp_wide_train.cu: with them).
#include "mp_wide.cuh"

namespace mpl {

cudaError_t launch_forward_wide_train(const FwdParams& p, cudaStream_t st);  // mp_wide_train.cu

// Dispatch on labels per lane and window width; the caller has checked that the windowed
// evaluation is exact (FwdParams::host_windowed) and that the staging alignment rules hold.
// `train`: the sweep also saves the argmin and normalisation indices (FwdParams::min_idx / norm_idx).
cudaError_t launch_forward_wide(const FwdParams& p, bool train, cudaStream_t st) {
  return train ? launch_forward_wide_train(p, st) : launch_wide_l<false>(p, st);
}

}  // namespace mpl
