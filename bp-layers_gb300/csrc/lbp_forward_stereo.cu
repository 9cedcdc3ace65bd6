// LBP forward instantiations for the stereo pairwise variant, up to 128
// labels, and the dispatch over the label-count ranges (several units, so
// that they compile side by side).
#include "lbp_forward.cuh"

namespace bpl {
int lbp_forward_stereo(const FwdArgs& a, cudaStream_t s) {
  if (a.L <= 128) return dispatch_stereo<float, 1, 4>(a, s);
  if (a.L <= 192) return lbp_forward_stereo_k5(a, s);
  if (a.L <= 256) return lbp_forward_stereo_k7(a, s);
  return lbp_forward_stereo_k12(a, s);
}
}  // namespace bpl
