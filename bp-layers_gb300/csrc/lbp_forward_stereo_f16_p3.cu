// LBP forward instantiations for the stereo pairwise variant, FP16 storage,
// 129 to 192 labels.
#include "lbp_forward_f16.cuh"

namespace bpl {
int lbp_forward_f16_pairs3(const FwdArgs& a, cudaStream_t s) { return launch_f16_pairs<3>(a, s); }
}  // namespace bpl
