// Instances of fwd_wide_kernel that save the argmin and normalisation indices.
#include "mp_wide.cuh"

namespace mpl {

cudaError_t launch_forward_wide_train(const FwdParams& p, cudaStream_t st) { return launch_wide_l<true>(p, st); }

}  // namespace mpl
