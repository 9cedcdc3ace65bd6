// LBP forward instantiations for the stereo pairwise variant, 193 to 256 labels.
#include "lbp_forward.cuh"

namespace bpl {
int lbp_forward_stereo_k7(const FwdArgs& a, cudaStream_t s) { return dispatch_stereo<float, 7, 8>(a, s); }
}  // namespace bpl
