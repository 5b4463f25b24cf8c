// Decode-sampling step with a row split over a cluster, f16 logits.
#include "split_sampling.cuh"

namespace ftb200 {
template int split_sampling_launch<FTB200_F16>(const KParams&, const SplitArgs&, cudaStream_t);
template int split_resident<FTB200_F16>(int, bool, size_t);
}  // namespace ftb200
