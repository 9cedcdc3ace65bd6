// LBP forward instantiations for the stereo pairwise variant, 257 to 1024 labels.
#include "lbp_forward.cuh"

namespace bpl {
int lbp_forward_stereo_k12(const FwdArgs& a, cudaStream_t s) { return dispatch_stereo<float, 12, 32>(a, s); }
}  // namespace bpl
