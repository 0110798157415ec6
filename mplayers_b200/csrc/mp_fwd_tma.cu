// Instances of fwd_tma_kernel for label-by-label tables, and the dispatch (mp_fwd_tma_rank1.cu,
// mp_fwd_tma_stride.cu: rank-1 contexts).
#include "mp_fwd_tma.cuh"

namespace mpl {

cudaError_t launch_forward_tma_rank1(const FwdParams& p, int dir, int stages, bool train, cudaStream_t st);

// Can direction `dir` of this problem use the bulk-copy kernel?  Needs 16-byte aligned row segments.
bool forward_tma_eligible(const FwdParams& p, int dir, bool train, int* stages) {
  if (dir > 3 || p.L > 32 || (!p.agg && p.D != 4 && p.D != 8)) return false;
  if (p.W & 3) return false;
  const uintptr_t bits = (uintptr_t)p.unary | (uintptr_t)p.msg_read | (uintptr_t)p.ew;
  if (bits & 15) return false;
  int ns = tma_stage_override() ? tma_stage_override() : 4;
  while (ns >= 2 && tma_smem_bytes(p.L, p.ls, p.agg ? 2 : p.D, ns, train) > (ns >= 3 ? 110 : 200) * 1024) --ns;
  if (ns < 2) return false;
  *stages = ns;
  return true;
}

cudaError_t launch_forward_tma(const FwdParams& p, int dir, int stages, bool train, cudaStream_t st) {
  return p.ctx_rank == 1 ? launch_forward_tma_rank1(p, dir, stages, train, st)
                         : launch_forward_tma_rank<false>(p, dir, stages, train, st);
}

}  // namespace mpl
