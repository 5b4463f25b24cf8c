// Single-pass decode-sampling kernels (top-k rows, top-p rows), half and bfloat16 logits.
#include "fast_sampling.cuh"

namespace ftb200 {
size_t fast_smem_for(int hash_slots, int vocab_padded, bool topp)
{
    return fast_smem_bytes(hash_slots, vocab_padded, topp);
}
int fast_rows_for(const KParams& K, int* list_k, int* list_p, cudaStream_t st)
{
    return fast_rows_launch(K, list_k, list_p, st);
}
int fast_max_history()
{
    return kFMaxHistAll;
}
bool fast_leaves_k(int k, int vocab)
{
    return fast_sample_rank(fast_topk_target(k), vocab & ~7) > (u32)kFMaxRank;
}
int fast_max_words()
{
    return kFMaxWords;
}
template int fast_sampling_occupancy<FTB200_F16, false>(size_t, int*);
template int fast_sampling_occupancy<FTB200_BF16, false>(size_t, int*);
template int fast_sampling_launch<FTB200_F16, false>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
template int fast_sampling_launch<FTB200_BF16, false>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
}  // namespace ftb200
