// LBP forward instantiations for the stereo pairwise variant, FP16 storage,
// 193 to 256 labels.
#include "lbp_forward_f16.cuh"

namespace bpl {
int lbp_forward_f16_pairs4(const FwdArgs& a, cudaStream_t s) { return launch_f16_pairs<4>(a, s); }
}  // namespace bpl
