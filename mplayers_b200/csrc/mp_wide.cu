// Instances of fwd_wide_kernel without saved indices, and the dispatch (mp_wide_train.cu: with them).
#include "mp_wide.cuh"

namespace mpl {

cudaError_t launch_forward_wide_train(const FwdParams& p, cudaStream_t st);  // mp_wide_train.cu

// Dispatch on labels per lane and window width; the caller has checked that the windowed
// evaluation is exact (FwdParams::host_windowed) and that the staging alignment rules hold.
// `train`: the sweep also saves the argmin and normalisation indices (FwdParams::min_idx / norm_idx).
cudaError_t launch_forward_wide(const FwdParams& p, bool train, cudaStream_t st) {
  if (train) return launch_forward_wide_train(p, st);
  // (a first TRWP iteration leaves out the slices that are still zero: only fwd_wide_kernel has that form)
  if (forward_team_eligible(p) && !(p.first && !p.agg && p.dir0 > 0)) return launch_forward_team(p, st);
  if (forward_many_eligible(p)) return launch_forward_many(p, st);
  return launch_wide_l<false>(p, st);
}

}  // namespace mpl
