// LBP forward instantiations for the stereo pairwise variant, 129 to 192 labels.
#include "lbp_forward.cuh"

namespace bpl {
int lbp_forward_stereo_k5(const FwdArgs& a, cudaStream_t s) { return dispatch_stereo<float, 5, 6>(a, s); }
}  // namespace bpl
