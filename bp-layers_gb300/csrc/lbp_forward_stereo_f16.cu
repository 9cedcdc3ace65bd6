// LBP forward instantiations for the stereo pairwise variant, FP16 storage:
// the lean kernel (lbp_forward_f16.cuh) for up to 256 labels, the general
// kernel for wider rows.
#include "lbp_forward_f16.cuh"

namespace bpl {
int lbp_forward_stereo_f16(const FwdArgs& a, cudaStream_t s) {
  if (a.L <= 64) return launch_f16_pairs<1>(a, s);
  if (a.L <= 128) return launch_f16_pairs<2>(a, s);
  if (a.L <= 192) return lbp_forward_f16_pairs3(a, s);
  if (a.L <= 256) return lbp_forward_f16_pairs4(a, s);
  return dispatch_stereo<__half, 12, 32>(a, s);
}
}  // namespace bpl
