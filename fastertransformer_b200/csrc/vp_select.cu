// Local pass of the vocabulary-parallel step, half and bfloat16 logits.
#include "vp_select.cuh"

namespace ftb200 {
template int vp_select_launch<FTB200_F16>(const KParams&, const VpArgs&, size_t, int, cudaStream_t);
template int vp_select_launch<FTB200_BF16>(const KParams&, const VpArgs&, size_t, int, cudaStream_t);
}  // namespace ftb200
