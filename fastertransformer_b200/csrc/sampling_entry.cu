// extern "C" entry of the fused decode-sampling step: argument checks, shared-memory plan, launch.
#include <atomic>
#include <chrono>

#include "device_once.cuh"
#include "sampling_params.cuh"
#include "spans.cuh"
#include "split_args.cuh"
#include "vp_args.cuh"

namespace ftb200 {

template<int DT>
int sampling_occupancy(size_t smem, int* per_sm);
template<int DT>
int sampling_launch(const KParams& K, const StopArgs& T, int grid, size_t smem, cudaStream_t st);
extern template int sampling_occupancy<FTB200_F32>(size_t, int*);
extern template int sampling_occupancy<FTB200_F16>(size_t, int*);
extern template int sampling_occupancy<FTB200_BF16>(size_t, int*);
extern template int sampling_launch<FTB200_F32>(const KParams&, const StopArgs&, int, size_t, cudaStream_t);
extern template int sampling_launch<FTB200_F16>(const KParams&, const StopArgs&, int, size_t, cudaStream_t);
extern template int sampling_launch<FTB200_BF16>(const KParams&, const StopArgs&, int, size_t, cudaStream_t);
template<int DT, bool TOPP, int VP = 0>
int fast_sampling_occupancy(size_t smem, int* per_sm);
template<int DT, bool TOPP, int VP = 0>
int fast_sampling_launch(const KParams& K, const StopArgs& T, int grid, size_t smem, bool beside, cudaStream_t st);
extern template int fast_sampling_occupancy<FTB200_F16, false, 1>(size_t, int*);
extern template int fast_sampling_occupancy<FTB200_BF16, false, 1>(size_t, int*);
extern template int fast_sampling_launch<FTB200_F16, false, 1>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
extern template int fast_sampling_launch<FTB200_BF16, false, 1>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
extern template int fast_sampling_occupancy<FTB200_F16, false>(size_t, int*);
extern template int fast_sampling_occupancy<FTB200_BF16, false>(size_t, int*);
extern template int fast_sampling_launch<FTB200_F16, false>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
extern template int fast_sampling_launch<FTB200_BF16, false>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
extern template int fast_sampling_occupancy<FTB200_F16, true>(size_t, int*);
extern template int fast_sampling_occupancy<FTB200_BF16, true>(size_t, int*);
extern template int fast_sampling_launch<FTB200_F16, true>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
extern template int fast_sampling_launch<FTB200_BF16, true>(const KParams&, const StopArgs&, int, size_t, bool, cudaStream_t);
template<int DT>
int split_sampling_launch(const KParams& K, const SplitArgs& A, cudaStream_t st);
extern template int split_sampling_launch<FTB200_F32>(const KParams&, const SplitArgs&, cudaStream_t);
extern template int split_sampling_launch<FTB200_F16>(const KParams&, const SplitArgs&, cudaStream_t);
extern template int split_sampling_launch<FTB200_BF16>(const KParams&, const SplitArgs&, cudaStream_t);
template<int DT>
int split_resident(int lgn, bool whole, size_t smem);
extern template int split_resident<FTB200_F32>(int, bool, size_t);
extern template int split_resident<FTB200_F16>(int, bool, size_t);
extern template int split_resident<FTB200_BF16>(int, bool, size_t);
size_t fast_smem_for(int hash_slots, int vocab_padded, bool topp);
int    fast_rows_for(const KParams& K, int* list_k, int* list_p, cudaStream_t st);
int    fast_max_history();
int    fast_max_words();
bool   fast_leaves_k(int k, int vocab);
template<int DT>
int vp_select_launch(const KParams& K, const VpArgs& V, size_t smem, int sms, cudaStream_t st);
extern template int vp_select_launch<FTB200_F16>(const KParams&, const VpArgs&, size_t, int, cudaStream_t);
extern template int vp_select_launch<FTB200_BF16>(const KParams&, const VpArgs&, size_t, int, cudaStream_t);
template<int DT>
int vp_merge_launch(const KParams& K, const u64* gathered, int nranks, int* overflow, int grid, cudaStream_t st);
extern template int vp_merge_launch<FTB200_F32>(const KParams&, const u64*, int, int*, int, cudaStream_t);
extern template int vp_merge_launch<FTB200_F16>(const KParams&, const u64*, int, int*, int, cudaStream_t);
extern template int vp_merge_launch<FTB200_BF16>(const KParams&, const u64*, int, int*, int, cudaStream_t);

static int sm_count()
{
    // per device (a process may drive several GPUs, one thread each)
    constexpr int           kMaxDev = 64;
    static std::atomic<int> n[kMaxDev];
    int                     dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDev) {
        dev = 0;
    }
    int v = n[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        if (v <= 0) {
            v = 148;
        }
        n[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

constexpr int kMaxCtasPerSm = 2;

static u64* g_row_trace = nullptr;  // diagnostic timeline buffer, see ftb200_set_row_trace

static size_t scratch_stride_for(int vocab_padded)
{
    return ((size_t)vocab_padded + 255) / 256 * 256;
}

// Workspace: 256-byte header (row tickets, length of the row list), the list of rows the single-pass kernel
// leaves to decode_sampling_kernel (one int per local row), then one candidate area per resident CTA.
static size_t redo_list_bytes(int local_batch)
{
    return ((size_t)local_batch * sizeof(int) + 255) / 256 * 256;
}

static int g_fast_path = 1;  // see ftb200_set_single_pass

// Clusters of the split kernel that are resident at once.  A cluster stays inside a group of SMs, and the groups' sizes are
// no multiples of eight: with one, two, three CTAs on an SM 15, 33 and 48 clusters of eight fit, not 18, 37 and 55.
static int resident_clusters(int dtype, int lgn, bool whole, size_t smem)
{
    switch (dtype) {
        case FTB200_F32: return split_resident<FTB200_F32>(lgn, whole, smem);
        case FTB200_F16: return split_resident<FTB200_F16>(lgn, whole, smem);
        default: return split_resident<FTB200_BF16>(lgn, whole, smem);
    }
}

constexpr size_t kRoomyTwoPerSm = 103 * 1024, kTwoPerSm = 107 * 1024 + 512, kThreePerSm = 69 * 1024;
constexpr size_t kOnePerSm = 190 * 1024;  // one CTA, in the largest split of an SM's memory but one: L1 keeps 60 KB

// Whether the split kernel (a row over a cluster of CTAs) serves a call, and in which form.  `single_pass`: the
// single-pass kernels could serve it too.  The lines come from timing both at 17000 .. 250000 columns and 6 .. 1024
// rows (us a step, split / single-pass): the split form ends a row in 6 us (arg-max) to 40 us (wide nucleus) however slow
// the row is for one CTA, but costs 2 to 4 times the SM time, so it loses once the single-pass kernels have the chip full.
// With both kinds of rows in a call those wait longest for their slowest rows: 128 x 128256 107 / 117, 160 x 128256 129 / 130,
// 256 x 128256 196 / 134, 96 x 250000 177 / 173 (at few columns the split form still wins above the line: 700 x 32000
// 128 / 178, 512 x 51200 174 / 199, 700 x 51200 228 / 210).  Rows of a small k are nearly as quick in one CTA: k = 50 64 x
// 32000 30 / 32, 128 x 32000 35 / 32; k = 1024 128 x 32000 48 / 76, 32 x 128256 48 / 74, 64 x 128256 79 / 78.
// Nucleus rows alone: with two CTAs a row all clusters have to be resident (148 x 17000 38 / 52, 148 x 32000 46 / 60, 192 x
// 32000 71 / 64), with four a third more may wait (64 x 51200 51 / 68, 80 x 51200 66 / 69, 96 x 41000 75 / 77, 112 x 51200
// 75 / 71), with eight, whose rows take one CTA longest, two rounds of them and more above 110000 columns (64 x 80000 81 / 80,
// 80 x 80000 100 / 83, 80 x 100000 123 / 111; 64 x 128256 99 / 113, 80 x 128256 117 / 114).
static bool choose_split(const ftb200_sampling_params* p, const KParams& K, bool single_pass, SplitArgs* A)
{
    const int rows = p->local_batch_size, vocab = p->vocab_size, sms = sm_count();
    if (vocab < 1024) {
        return false;  // (the denominator's chains are then not 1024)
    }
    const bool topk = K.topk_states != nullptr, topp = K.topp_states != nullptr, mixed = topk && topp;
    // Nucleus rows off a 16-byte boundary (an odd vocabulary) are none of the single-pass kernels': they would all end in the general
    // one.  us a step, general kernel / split form, bf16: nucleus rows alone, 300 x 17001 205 / 89, 1000 x 30001 613 / 290, 1000 x 50257
    // 866 / 479, 150 x 128257 564 / 192, 500 x 128257 1183 / 616, 200 x 250001 1216 / 774: always the split form; both kinds, 1000 x 17001
    // 218 / 160, 400 x 50257 316 / 137, 800 x 50257 352 / 309, 1000 x 50257 367 / 380, 150 x 128257 503 / 122, 300 x 128257 555 / 284, 1000 x
    // 128257 665 / 888.  (The line is coarse: above it 600 x 100001 is even, 507 / 500, and 600 x 128257, 606 / 546, and 300 x 250001, 924 /
    // 861, would be quicker in the split form; the two that are not have 1000 rows.)
    const bool off = topp && (((size_t)p->logits | (size_t)p->vocab_size_padded * 2) & 15) != 0;
    if (single_pass && off && mixed && (double)rows * vocab > 48e6) {
        return false;
    }
    if (single_pass && !off && (double)rows * vocab > (mixed ? 16.5e6 : (topp ? 9e6 : (K.max_top_k > 256 ? 4.2e6 : 2.1e6)))) {
        return false;
    }
    // CTAs per row: eight while they are all resident (and for rows so long that a slice would not leave room for
    // three CTAs on an SM), four or two when there are more rows or the rows are short: a CTA's fixed costs then weigh
    // more than its columns (1024 x 32000 fp32, k = 50: 445 us with eight, 184 us with two).  With both kinds of rows the
    // costliest are started first and a last few that wait for a place are short: there the SMs are counted alone.
    const auto most_rows = [&](int lg) { return mixed ? 2 * sms >> lg : resident_clusters(p->dtype, lg, false, kTwoPerSm); };
    const bool few       = rows * 16 <= sms;  // (no group of SMs is so small: resident, without a question)
    int        lgn       = vocab > 65536 || few || rows <= most_rows(3) ? 3 : (vocab > 40960 || rows <= most_rows(2) ? 2 : 1);
    for (; lgn <= 3; ++lgn) {
        A->slice = ((vocab + 1023) / 1024) << (10 - lgn);
        A->slice = A->slice < kSpMinSlice ? kSpMinSlice : A->slice;
        if (split_smem_bytes(A->slice, kSpAreaMin) <= kSpMaxSmem) {
            break;
        }
    }
    if (lgn > 3) {
        return false;
    }
    A->lgn             = lgn;
    const size_t least = split_smem_bytes(A->slice, kSpAreaMin);
    if (single_pass && !off && topp && !topk) {
        const int at_once = resident_clusters(p->dtype, lgn, false, lgn == 1 ? least : kTwoPerSm);
        const int most    = lgn == 1 ? at_once : (lgn == 2 ? at_once * 4 / 3 : (int)(2.0 * at_once * (vocab > 110000 ? vocab / 110000.0 : 1.0)));
        if (rows > most) {
            return false;
        }
    }
    // The roomy form is taken while its clusters are resident at once, with two CTAs on an SM where shared
    // memory allows (16 x 128256 bf16, one CTA on an SM: k = 50 60 us a step, 46 in the other form; 14 rows 39 / 45).  The
    // collection areas: a wide nucleus of a flat row takes half of the columns, so up to 5/8 of a slice is
    // provided for as far as that residency holds (a row beyond it costs milliseconds in the general code).
    const auto area_within = [&](size_t budget, int most) {
        int area = (A->slice * 5 / 8 + 1023) / 1024 * 1024;
        area     = area > most ? most : (area < kSpAreaMin ? kSpAreaMin : area);
        while (area > kSpAreaMin && split_smem_bytes(A->slice, area) > budget) {
            area -= 1024;
        }
        return area;
    };
    // With one CTA on an SM there is room for areas of half a slice up to 245000 columns, and no step needs the second launch for wider ones,
    // which costs 3 us where nothing is flagged (area of 10240 keys and that launch / so: 28 x 208295 fp32 of both kinds with
    // log-probabilities 77.7 / 74.1 us; with areas that leave L1 28 KB 75.5).
    const auto one_on_an_sm = [&] {
        const int area = area_within(kOnePerSm, kSpAreaWide);
        return area < A->slice / 2 ? area_within(kSpMaxSmem, kSpAreaWide) : area;
    };
    const int  ctas  = rows << lgn;
    const auto keeps = [&](int per_sm, size_t budget) {
        A->area = per_sm == 1 ? one_on_an_sm() : area_within(budget, kSpAreaMax);
        return mixed || few ? ctas <= per_sm * sms : rows <= resident_clusters(p->dtype, lgn, true, split_smem_bytes(A->slice, A->area));
    };
    A->roomy    = lgn >= 2 && (keeps(1, kSpMaxSmem) || (least <= kRoomyTwoPerSm && keeps(2, kRoomyTwoPerSm)));
    A->criteria = A->roomy;
    if (!A->roomy && lgn >= 2 && least > kThreePerSm) {
        // Shared memory holds two CTAs on an SM, or one, whatever the registers: the roomy form for more rows than are resident
        // too.  us a step without a length limit, 128 / 80 registers: with both kinds of rows, bf16, 40 x 128256 40 / 47, 128 x
        // 128256 77 / 93, 160 x 100000 86 / 109, 250 x 65000 71 / 85, 200 x 50257 65 / 78; fp32, 300 x 128256 178 / 214; nucleus
        // rows, 64 x 128256 bf16 70 / 83, 160 x 65000 fp32 80 / 97, 300 x 50257 fp32 118 / 150; k = 50, fp32, 96 x 128256 59 / 71.
        // The criteria in the launch (the last row does them wherever it runs) against a launch of their own, with a limit:
        // both kinds of rows 47 / 54, 87 / 91, 102 / 101, 80 / 84, 76 / 79, 195 / 192 for those six.  One kind of rows alone has
        // them apart: 78 / 85 at 64 x 128256 bf16, 87 / 95 at 160 x 65000 fp32, but 264 / 260 and (k = 50) 197 / 189 at 300 x
        // 128256 fp32, and no line between the two has been drawn.
        A->roomy    = 1;
        A->criteria = mixed;
        A->area     = least <= kTwoPerSm ? area_within(kTwoPerSm, kSpAreaMax) : one_on_an_sm();
    }
    else if (!A->roomy) {
        A->area = area_within(least <= kThreePerSm ? kThreePerSm : (least <= kTwoPerSm ? kTwoPerSm : kSpMaxSmem), kSpAreaMid);
    }
    // (a row's number then need not be looked up in the order before anything of the row can be sent for)
    A->at_once = few || rows <= resident_clusters(p->dtype, lgn, A->roomy != 0, split_smem_bytes(A->slice, A->area));
    return true;
}

// Slices and areas of the split kernel's second launch, over flagged rows: eight CTAs a row.
static bool wide_areas(int vocab, SplitArgs* A)
{
    A->lgn   = 3;
    A->roomy = 1;
    A->slice = ((vocab + 1023) / 1024) << 7;
    A->slice = A->slice < kSpMinSlice ? kSpMinSlice : A->slice;
    A->area  = kSpAreaWide;
    while (A->area > kSpAreaMin && split_smem_bytes(A->slice, A->area) > kSpMaxSmem) {
        A->area -= 1024;
    }
    return split_smem_bytes(A->slice, A->area) <= kSpMaxSmem;
}

}  // namespace ftb200

using namespace ftb200;

extern "C" int ftb200_sampling_workspace_bytes(int dtype, int local_batch_size, int vocab_size_padded, size_t* bytes)
{
    if (bytes == nullptr || local_batch_size < 0 || vocab_size_padded <= 0 || dtype < 0 || dtype > 2) {
        set_error("ftb200_sampling_workspace_bytes: invalid argument");
        return FTB200_INVALID_ARG;
    }
    size_t ctas = (size_t)sm_count() * kMaxCtasPerSm;
    if ((size_t)local_batch_size < ctas) {
        ctas = (size_t)local_batch_size;
    }
    *bytes = 256 + redo_list_bytes(local_batch_size) + ctas * scratch_stride_for(vocab_size_padded) * sizeof(u64);
    return FTB200_OK;
}

// Argument checks, translation to the kernel argument block, shared-memory plan and grid size, shared by
// the entry points below.  `need_workspace` is false for the vocabulary-parallel merge.
static int plan_sampling(const ftb200_sampling_params* p, KParams& K, size_t& smem, int& grid, bool need_workspace)
{
    if (p == nullptr || p->logits == nullptr || p->end_ids == nullptr || p->output_ids == nullptr) {
        set_error("ftb200_decode_step_sampling: null logits / end_ids / output_ids");
        return FTB200_INVALID_ARG;
    }
    if (p->dtype < 0 || p->dtype > 2 || p->local_batch_size < 0 || p->vocab_size <= 0
        || p->vocab_size_padded < p->vocab_size || p->batch_size < p->local_batch_size || p->step < 0) {
        set_error("ftb200_decode_step_sampling: bad shape or dtype");
        return FTB200_INVALID_ARG;
    }
    if (p->vocab_size_padded > (1 << 21)) {
        set_error("ftb200_decode_step_sampling: vocab_size_padded above 2^21 is not supported");
        return FTB200_UNSUPPORTED;
    }
    if (p->topk_states == nullptr && p->topp_states == nullptr) {
        set_error("ftb200_decode_step_sampling: neither a top-k nor a top-p layer state was given");
        return FTB200_INVALID_ARG;
    }
    if (p->topk_states != nullptr) {
        if (p->topk_ks == nullptr || p->topk_ps == nullptr) {
            set_error("ftb200_decode_step_sampling: top-k layer needs topk_ks and topk_ps");
            return FTB200_INVALID_ARG;
        }
        if (p->max_top_k < 1 || p->max_top_k > kMaxTopK) {
            set_error("top-k kernel supports 1<=k<=1024 but got k=" + std::to_string(p->max_top_k));
            return FTB200_DOMAIN_ERROR;
        }
    }
    if (p->topp_states != nullptr && p->topp_ps == nullptr) {
        set_error("ftb200_decode_step_sampling: top-p layer needs topp_ps");
        return FTB200_INVALID_ARG;
    }
    if ((p->apply_temperature && p->temperature == nullptr) || (p->apply_repetition && p->repetition_penalty == nullptr)
        || (p->apply_min_length && (p->min_lengths == nullptr || p->sequence_length == nullptr))) {
        set_error("ftb200_decode_step_sampling: a penalty is switched on without its per-row array");
        return FTB200_INVALID_ARG;
    }
    size_t need = 0;
    ftb200_sampling_workspace_bytes(p->dtype, p->local_batch_size, p->vocab_size_padded, &need);
    if (need_workspace && (p->workspace == nullptr || p->workspace_bytes < need)) {
        set_error("ftb200_decode_step_sampling: workspace too small, need " + std::to_string(need) + " bytes");
        return FTB200_WORKSPACE_SMALL;
    }

    K.vp_out       = nullptr;
    K.vp_cap       = 0;
    K.vocab_offset = 0;
    K.dtype            = p->dtype;
    K.batch_size       = p->batch_size;
    K.local_batch      = p->local_batch_size;
    K.ite              = p->ite;
    K.vocab            = p->vocab_size;
    K.vocab_padded     = p->vocab_size_padded;
    K.step             = p->step;
    K.max_input_len    = p->max_input_length;
    K.logits           = p->logits;
    K.bias             = p->embedding_bias;
    K.end_ids          = p->end_ids;
    K.input_lengths    = p->input_lengths;
    K.output_ids       = p->output_ids;
    K.bad_words        = p->bad_words_len > 0 ? p->bad_words : nullptr;
    K.bad_words_len    = p->bad_words_len;
    K.bad_words_shared = p->bad_words_shared;
    K.temperature      = p->temperature;
    K.apply_temp       = p->apply_temperature ? 1 : 0;
    K.rep_penalty      = p->repetition_penalty;
    K.penalty_type     = p->penalty_type;
    K.apply_rep        = (p->apply_repetition && p->penalty_type != FTB200_PENALTY_NONE) ? 1 : 0;
    K.min_lengths      = p->min_lengths;
    K.apply_minlen     = p->apply_min_length ? 1 : 0;
    K.topk_states      = (curandState_t*)p->topk_states;
    K.topk_ks          = p->topk_ks;
    K.topk_ps          = p->topk_ps;
    K.topk_skip        = p->topk_skip;
    K.max_top_k        = p->topk_states != nullptr ? p->max_top_k : 1;
    K.topp_states      = (curandState_t*)p->topp_states;
    K.topp_ps          = p->topp_ps;
    K.topp_skip        = p->topp_skip;
    K.topp_initial     = p->topp_initial_ps;
    K.topp_decay       = (p->topp_decay && p->topp_min && p->topp_reset_ids && p->topp_initial_ps) ? p->topp_decay : nullptr;
    K.topp_min         = p->topp_min;
    K.topp_reset       = p->topp_reset_ids;
    K.seq_len          = p->sequence_length;
    K.finished         = p->finished;
    K.cum_log_probs    = p->cum_log_probs;
    K.out_log_probs    = p->output_log_probs;
    K.whole_words      = whole_words(p->local_batch_size, (size_t)p->topk_skip, (size_t)p->topp_skip, (size_t)p->finished);
    K.row_order        = p->row_order;
    K.trace            = g_row_trace;

    // shared-memory plan: candidates, histogram, 1024 floats, vector flags, token hash with two values per slot
    const int epv      = p->dtype == FTB200_F32 ? 4 : 8;
    K.flag_words       = ((p->vocab_size_padded / epv + 32) / 32 + 1) & ~1;  // even: what follows stays 8-byte aligned
    int specials       = (K.apply_rep ? p->step : 0) + (K.bad_words ? p->bad_words_len : 0) + 2;
    int slots          = 64;
    while (slots < 2 * specials) {
        slots <<= 1;
    }
    // (a large table costs the kernels resident CTAs: above 2048 slots it may be three quarters full)
    if (slots > 2048 && 3 * (slots / 2) >= 4 * specials) {
        slots /= 2;
    }
    K.hash_slots = slots;
    int lg       = 0;
    while ((1 << lg) < slots) {
        ++lg;
    }
    K.hash_shift = 32 - lg;
    smem         = (size_t)kCap * 8 + (size_t)kNB * 4 + 1024 * 4 + (size_t)K.flag_words * 4 + (size_t)slots * 12 + 32
                   + (size_t)kThreads * 16 * 2;
    if (smem > 200 * 1024 || specials > 4096) {
        set_error("ftb200_decode_step_sampling: token history too long for the shared-memory hash");
        return FTB200_UNSUPPORTED;
    }

    int per_sm = 0, rc;
    switch (p->dtype) {
        case FTB200_F32: rc = sampling_occupancy<FTB200_F32>(smem, &per_sm); break;
        case FTB200_F16: rc = sampling_occupancy<FTB200_F16>(smem, &per_sm); break;
        default: rc = sampling_occupancy<FTB200_BF16>(smem, &per_sm); break;
    }
    if (rc != FTB200_OK) {
        return rc;
    }
    if (per_sm < 1) {
        set_error("ftb200_decode_step_sampling: kernel does not fit on an SM");
        return FTB200_UNSUPPORTED;
    }
    if (per_sm > kMaxCtasPerSm) {
        per_sm = kMaxCtasPerSm;
    }
    grid = sm_count() * per_sm;
    if (grid > p->local_batch_size) {
        grid = p->local_batch_size;
    }
    K.ticket         = (u32*)p->workspace;
    K.redo_count     = nullptr;
    K.redo_rows      = nullptr;
    K.row_count_dev  = nullptr;
    K.row_flags      = nullptr;
    K.early          = 0;
    K.stop_words     = nullptr;
    K.scratch        = (u64*)((char*)p->workspace + 256 + redo_list_bytes(p->local_batch_size));
    K.scratch_stride = scratch_stride_for(p->vocab_size_padded);
    return FTB200_OK;
}

extern "C" int ftb200_set_row_trace(uint64_t* device_buf)
{
    g_row_trace = (u64*)device_buf;
    return FTB200_OK;
}

// One fused step.
namespace ftb200 {
// What of a step's end the sampling launches see to: nothing, all of it unless rows are left (the host hears of them and sends
// what serves them), or all of it.
enum StepEnd : int { kStepEndNone, kStepEndRowsLeft, kStepEndAll };
struct StepTail {
    StepEnd  end = kStepEndNone;
    // the general kernel over the single-pass kernels' list of rows, which ends the step then; grid 0: there is no such list
    KParams  K;
    StopArgs S;
    int      grid = 0;
    size_t   smem = 0;
};
// Whether the general kernel has been launched on the current device.  Its first launch takes milliseconds (the kernel is loaded, and the
// device's memory for stack frames grows to its): where nothing else asks for it in the first steps, one of them does.
static std::atomic<bool>* general_known(int dtype)
{
    static std::atomic<bool> known[kDevicesKnown][3];
    int                      dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kDevicesKnown ? &known[dev][dtype] : nullptr;
}
static int general_launch(int dtype, const KParams& K, const StopArgs& S, int grid, size_t smem, cudaStream_t st)
{
    int rc;
    switch (dtype) {
        case FTB200_F32: rc = sampling_launch<FTB200_F32>(K, S, grid, smem, st); break;
        case FTB200_F16: rc = sampling_launch<FTB200_F16>(K, S, grid, smem, st); break;
        default: rc = sampling_launch<FTB200_BF16>(K, S, grid, smem, st); break;
    }
    if (rc == FTB200_OK) {
        std::atomic<bool>* const known = general_known(dtype);
        if (known != nullptr && !known->load(std::memory_order_relaxed)) {
            known->store(true, std::memory_order_relaxed);
        }
        note_launch(1);
    }
    return rc;
}
// left_only: the rows that the split kernel of the same step has flagged, by the general kernel.
int decode_step_sampling_impl(const ftb200_sampling_params* p, const StopArgs* stop = nullptr, StepTail* tail = nullptr,
                              bool left_only = false);
int stop_criteria_launch(const ftb200_sampling_params* p, const StopArgs& T, cudaStream_t st);
}

extern "C" int ftb200_decode_step_sampling(const ftb200_sampling_params* p)
{
    return decode_step_sampling_impl(p);
}

extern "C" int ftb200_decode_step(const ftb200_sampling_params* p, ftb200_stop_params* s, int timeout_ms, int* should_stop)
{
    if (s == nullptr || should_stop == nullptr || p == nullptr || p->finished == nullptr
        || (s->sequence_limit_length != nullptr && (s->result_host == nullptr || s->arrived_dev == nullptr))) {
        set_error("ftb200_decode_step: invalid argument");
        return FTB200_INVALID_ARG;
    }
    StopArgs T{};
    T.stop_words     = s->stop_words_len > 0 ? s->stop_words : nullptr;
    T.stop_words_len = s->stop_words_len;
    T.limit          = s->sequence_limit_length;
    T.finished       = p->finished - (size_t)p->ite * p->local_batch_size;
    T.arrived        = s->arrived_dev;
    T.result         = (u64*)s->result_host;
    T.sequence       = ++s->sequence;
    StepTail tail;
    int      rc = decode_step_sampling_impl(p, &T, &tail);
    if (rc == FTB200_OK && tail.end == kStepEndNone) {
        rc = stop_criteria_launch(p, T, (cudaStream_t)p->stream);
    }
    *should_stop = 0;
    if (rc != FTB200_OK || T.limit == nullptr) {
        return rc;
    }
    // Rare: rows that the single-pass kernels left, by the general kernel, which ends the step; or rows that the split kernel's
    // tables could not hold, then the criteria over the whole call.  The rows are found by their list or their flags on the
    // device, so that these launches do nothing new where none is left.
    bool       left_sent = tail.end != kStepEndRowsLeft;
    const auto send_left = [&] {
        left_sent = true;
        if (tail.grid != 0) {
            return general_launch(p->dtype, tail.K, tail.S, tail.grid, tail.smem, (cudaStream_t)p->stream);
        }
        const int e = decode_step_sampling_impl(p, nullptr, nullptr, true);
        return e == FTB200_OK ? stop_criteria_launch(p, T, (cudaStream_t)p->stream) : e;
    };
    // The last kernel of the step stores (sequence, count) into the page-locked word: no query of the stream, whose
    // answer comes several microseconds after the kernel's end.
    const volatile u64* w  = T.result;
    const auto          t0 = std::chrono::steady_clock::now();
    for (u32 spin = 1;; ++spin) {
        const u64 v = *w;
        if ((u32)(v >> 32) == T.sequence) {
            *should_stop = (u32)v == (u32)p->batch_size ? 1 : 0;
            return FTB200_OK;
        }
        if (v == rows_left(T.sequence) && !left_sent) {
            rc = send_left();
            if (rc != FTB200_OK) {
                return rc;
            }
            continue;
        }
        if ((spin & 1023u) == 0) {
            const cudaError_t e = cudaStreamQuery((cudaStream_t)p->stream);
            if (e != cudaSuccess && e != cudaErrorNotReady) {
                set_error(std::string("ftb200_decode_step: ") + cudaGetErrorString(e));
                return FTB200_CUDA_ERROR;
            }
            const auto ms = std::chrono::duration_cast<std::chrono::milliseconds>(std::chrono::steady_clock::now() - t0);
            if (timeout_ms >= 0 && ms.count() > timeout_ms) {
                // (nobody may be there to read that rows are left: behind the step in its stream, whether there are any or not)
                if (!left_sent && (rc = send_left()) != FTB200_OK) {
                    return rc;
                }
                set_error("ftb200_decode_step: the step did not end within the deadline");
                return FTB200_TIMEOUT;
            }
        }
    }
}

int ftb200::decode_step_sampling_impl(const ftb200_sampling_params* p, const StopArgs* stop, StepTail* tail, bool left_only)
{
    if (!left_only) {
        reset_launch_count();
    }
    KParams K;
    size_t  smem = 0;
    int     grid = 0;
    int     rc   = plan_sampling(p, K, smem, grid, true);
    if (rc != FTB200_OK) {
        return rc;
    }
    if (p->local_batch_size == 0) {
        return FTB200_OK;
    }
    cudaStream_t st = (cudaStream_t)p->stream;
    // 16-bit logits without a bias, log-probs or timeline: the single-pass kernel serves the rows first and
    // leaves a list of the rows it does not cover; decode_sampling_kernel then works that list off.
    const bool single_pass = (g_fast_path || left_only) && p->dtype != FTB200_F32 && K.bias == nullptr && K.cum_log_probs == nullptr
                             && K.out_log_probs == nullptr && p->vocab_size_padded <= (1 << 20)
                             && p->vocab_size >= 16384 + 16 && (K.apply_rep ? p->step : 0) <= fast_max_history()
                             && (K.bad_words != nullptr ? K.bad_words_len : 0) <= fast_max_words();
    SplitArgs A{};
    if ((g_fast_path || left_only) && choose_split(p, K, single_pass, &A)) {
        A.redo_flags      = (int*)((char*)p->workspace + 256);
        if (A.at_once) {
            K.row_order = nullptr;
        }
        const auto launch = [&](const SplitArgs& args) {
            switch (p->dtype) {
                case FTB200_F32: return split_sampling_launch<FTB200_F32>(K, args, st);
                case FTB200_F16: return split_sampling_launch<FTB200_F16>(K, args, st);
                default: return split_sampling_launch<FTB200_BF16>(K, args, st);
            }
        };
        if (!left_only) {
            SplitArgs F = A;
            if (A.criteria && stop != nullptr && (stop->limit != nullptr || stop->stop_words != nullptr)) {
                F.stop    = *stop;
                tail->end = kStepEndRowsLeft;
            }
            rc = launch(F);
            if (rc != FTB200_OK) {
                return rc;
            }
            note_launch(1);
            if (F.stop.limit != nullptr) {
                return FTB200_OK;  // (the host hears of rows that are left and asks for them)
            }
        }
        // Flat rows' wide nuclei that the areas do not hold go over eight CTAs with areas as large as shared memory allows: where the host
        // has heard of rows left and the areas are larger than the first launch's, and behind every step that does not wait where those
        // are below half a slice (above 98000 columns; above 49000, 24000 with four, two CTAs a row).  Where the large ones are below
        // half a slice too (above 245000 columns) the general kernel's many CTAs serve the several rows left sooner.
        const bool words = !left_only && tail != nullptr && tail->end != kStepEndNone;  // (no limit: who serves a row sees to its stop words)
        SplitArgs  B     = A;
        if (words) {
            B.stop = *stop;
        }
        if (wide_areas(p->vocab_size, &B) && K.topp_states != nullptr && (left_only ? A.area << A.lgn < B.area << B.lgn : A.area < A.slice / 2)
            && B.area >= B.slice / 2) {
            B.clusters = sm_count() / kSpMaxN < p->local_batch_size ? sm_count() / kSpMaxN : p->local_batch_size;
            rc         = launch(B);
            if (rc != FTB200_OK) {
                return rc;
            }
            note_launch(1);
        }
        K.row_flags = A.redo_flags;
        if (words) {
            K.stop_words = stop->stop_words, K.stop_words_len = stop->stop_words_len, K.stop_finished = stop->finished;
        }
    }
    StopArgs S{};
    if (single_pass && K.row_flags == nullptr) {
        const size_t fsmem = fast_smem_for(K.hash_slots, p->vocab_size_padded, false);
        const size_t psmem = fast_smem_for(K.hash_slots, p->vocab_size_padded, true);
        const bool   f16   = p->dtype == FTB200_F16;
        int          fper = 0, pper = 0;
        rc = f16 ? fast_sampling_occupancy<FTB200_F16, false>(fsmem, &fper) :
                   fast_sampling_occupancy<FTB200_BF16, false>(fsmem, &fper);
        if (rc == FTB200_OK && K.topp_states != nullptr) {
            rc = f16 ? fast_sampling_occupancy<FTB200_F16, true>(psmem, &pper) :
                       fast_sampling_occupancy<FTB200_BF16, true>(psmem, &pper);
        }
        if (rc != FTB200_OK) {
            return rc;
        }
        if (fper >= 1 && (K.topp_states == nullptr || pper >= 1)) {
            KParams F    = K;
            F.redo_count = K.ticket + 1;
            F.redo_rows  = (int*)((char*)p->workspace + 256);
            // The rows of the top-p layer have a kernel of their own (it wants more registers than the top-k rows'
            // kernel can spare); the two run side by side.
            const bool topp_only = K.topp_states != nullptr && K.topk_states == nullptr;  // one launch
            const bool both      = K.topp_states != nullptr && K.topk_states != nullptr;
            int* const list_k    = (int*)K.scratch;  // (the general kernel takes the scratch area once these have ended)
            int* const list_p    = list_k + p->local_batch_size;
            rc                   = fast_rows_for(F, both ? list_k : nullptr, list_p, st);
            if (rc != FTB200_OK) {
                return rc;
            }
            note_launch(1);
            const int rows  = p->local_batch_size;
            const int pgrid = K.topp_states == nullptr ? 0 : (sm_count() * pper < rows ? sm_count() * pper : rows);
            const int fgrid = topp_only ? 0 : (sm_count() * fper < rows ? sm_count() * fper : rows);
            if (stop != nullptr && stop->limit != nullptr) {
                // A host that waits goes on once the last CTA has counted, and may hand the workspace to another stream then, so nothing
                // that reads it may be queued behind: the host hears of rows left and sends the general kernel.  That costs
                // a round trip; where there are such rows in all likelihood - a k that the sample is too small for, nucleus rows off
                // a 16-byte boundary - the general kernel is queued and ends the step; so it does in the first such step on a
                // device.  us a step, queued always / so: 867 x 26268 half, k = 50 64.8 / 59.2; nucleus rows at temperature 1.2, nine left,
                // 260.4 / 267.6; 785 x 36096 bf16 of both kinds, 204 of them with k = 1024, 123.4 / 120.7; 1024 x 128256 166.2 / 165.6.
                const std::atomic<bool>* const known = general_known(p->dtype);
                const bool queue = (known != nullptr && !known->load(std::memory_order_relaxed))
                                   || (!topp_only && fast_leaves_k(K.max_top_k, p->vocab_size))
                                   || (K.topp_states != nullptr && (((size_t)p->logits | (size_t)p->vocab_size_padded * 2) & 15) != 0);
                S         = *stop;
                S.arrived = K.ticket + 4;
                S.ctas    = queue ? 0u : (u32)(pgrid + fgrid);
                tail->end = queue ? kStepEndAll : kStepEndRowsLeft;
            }
            if (K.topp_states != nullptr) {
                if (both) {
                    F.row_order = list_p, F.row_count_dev = K.ticket + 6;
                }
                rc = f16 ? fast_sampling_launch<FTB200_F16, true>(F, S, pgrid, psmem, true, st) :
                           fast_sampling_launch<FTB200_BF16, true>(F, S, pgrid, psmem, true, st);
                if (rc != FTB200_OK) {
                    return rc;
                }
                note_launch(1);
            }
            if (!topp_only) {
                if (both) {
                    F.row_order = list_k, F.row_count_dev = K.ticket + 5;
                }
                rc = f16 ? fast_sampling_launch<FTB200_F16, false>(F, S, fgrid, fsmem, true, st) :
                           fast_sampling_launch<FTB200_BF16, false>(F, S, fgrid, fsmem, true, st);
                if (rc != FTB200_OK) {
                    return rc;
                }
                note_launch(1);
            }
            if (S.limit != nullptr) {
                S.arrived    = K.ticket + 7;
                K.stop_words = S.stop_words, K.stop_words_len = S.stop_words_len, K.stop_finished = S.finished;
            }
            K.ticket        = K.ticket + 2;
            K.row_order     = F.redo_rows;
            K.row_count_dev = F.redo_count;
            K.early         = 1;
            if (K.trace != nullptr) {
                K.trace += (size_t)p->local_batch_size * 32;  // the general kernel's records follow the single-pass kernel's
            }
            if (S.ctas != 0) {
                tail->K = K, tail->S = S, tail->grid = grid, tail->smem = smem;
                return FTB200_OK;
            }
        }
    }
    if (K.row_flags == nullptr && K.row_count_dev == nullptr) {
        FTB_CUDA_CHECK(cudaMemsetAsync(K.ticket, 0, 256, st));
    }
    return general_launch(p->dtype, K, S, grid, smem, st);
}

extern "C" int ftb200_set_single_pass(int on)
{
    g_fast_path = on ? 1 : 0;
    return FTB200_OK;
}

// ---- vocabulary-parallel sampling (the logits of a row are split over several GPUs by column) ------
// Records of the shards [0, n) that this device holds: `p` describes them together (vocab_size columns from token id
// `offset` on, vocab_size_padded columns per shard in memory), `logits` is a host array.  Returns false when the
// select kernel does not serve the call: fp32 logits, a bias, a row that does not fit into shared memory, top-p rows
// (statistics form) on more than one shard, which need the general kernel's row list per shard.
static bool plan_vp_select(const ftb200_sampling_params* p, const KParams& K, const void* const* logits, int n, int offset,
                           int cap, u64* records, VpArgs* V, size_t* smem)
{
    if (!g_fast_path || p->dtype == FTB200_F32 || K.bias != nullptr || K.topk_states == nullptr || n > kVpMaxShards
        || (K.topp_states != nullptr && n > 1)) {
        return false;
    }
    vp_select_plan(*V, p->vocab_size_padded, cap, K.max_top_k, K.apply_rep ? p->step : 0, smem);
    if (*smem > (size_t)kVpMaxSmem) {
        return false;
    }
    for (int i = 0; i < n; ++i) {
        if (((size_t)logits[i] & 1) != 0) {
            return false;
        }
        V->logits[i] = logits[i];
    }
    V->out = records, V->n_shards = n, V->vocab = p->vocab_size, V->offset = offset;
    return true;
}

static int launch_vp_select(const KParams& K, const VpArgs& V, size_t smem, cudaStream_t st)
{
    const int rc = K.dtype == FTB200_F16 ? vp_select_launch<FTB200_F16>(K, V, smem, sm_count(), st) :
                                           vp_select_launch<FTB200_BF16>(K, V, smem, sm_count(), st);
    if (rc == FTB200_OK) {
        note_launch(1);
    }
    return rc;
}

// The local pass of one shard; the caller has reset the launch count.
static int vp_local(const ftb200_sampling_params* p, int vocab_offset, int cap, uint64_t* records)
{
    KParams K;
    size_t  smem = 0;
    int     grid = 0;
    int     rc   = plan_sampling(p, K, smem, grid, true);
    if (rc != FTB200_OK) {
        return rc;
    }
    if (p->local_batch_size == 0) {
        return FTB200_OK;
    }
    K.vp_out       = (u64*)records;
    K.vp_cap       = cap;
    K.vocab_offset = vocab_offset;
    cudaStream_t st = (cudaStream_t)p->stream;
    VpArgs       V;
    size_t       vsmem  = 0;
    const bool   select = plan_vp_select(p, K, &p->logits, 1, vocab_offset, cap, K.vp_out, &V, &vsmem);
    if (select && K.topp_states == nullptr) {
        return launch_vp_select(K, V, vsmem, st);
    }
    FTB_CUDA_CHECK(cudaMemsetAsync(K.ticket, 0, 256, st));
    if (select) {
        KParams F    = K;
        F.redo_count = K.ticket + 1;
        F.redo_rows  = (int*)((char*)p->workspace + 256);
        rc           = launch_vp_select(F, V, vsmem, st);
        if (rc != FTB200_OK) {
            return rc;
        }
        K.ticket        = K.ticket + 2;
        K.row_order     = F.redo_rows;
        K.row_count_dev = F.redo_count;
    }
    // wider 16-bit shards: the single-pass kernel in its record form serves the top-k rows and leaves a list of the
    // others (top-p rows of the statistics form, rows it cannot decide) to the kernel below
    const bool single_pass = !select && g_fast_path && p->dtype != FTB200_F32 && K.bias == nullptr
                             && p->vocab_size_padded <= (1 << 20) && p->vocab_size >= 16384 + 16 && (K.apply_rep ? p->step : 0) <= fast_max_history()
                             && (K.bad_words != nullptr ? K.bad_words_len : 0) <= fast_max_words();
    if (single_pass) {
        const size_t fsmem = fast_smem_for(K.hash_slots, p->vocab_size_padded, false);
        const bool   f16   = p->dtype == FTB200_F16;
        int          fper  = 0;
        rc = f16 ? fast_sampling_occupancy<FTB200_F16, false, 1>(fsmem, &fper) :
                   fast_sampling_occupancy<FTB200_BF16, false, 1>(fsmem, &fper);
        if (rc != FTB200_OK) {
            return rc;
        }
        if (fper >= 1) {
            KParams F    = K;
            F.redo_count = K.ticket + 1;
            F.redo_rows  = (int*)((char*)p->workspace + 256);
            int fgrid    = sm_count() * fper;
            fgrid        = fgrid < p->local_batch_size ? fgrid : p->local_batch_size;
            rc = f16 ? fast_sampling_launch<FTB200_F16, false, 1>(F, StopArgs{}, fgrid, fsmem, false, st) :
                       fast_sampling_launch<FTB200_BF16, false, 1>(F, StopArgs{}, fgrid, fsmem, false, st);
            if (rc != FTB200_OK) {
                return rc;
            }
            note_launch(1);
            K.ticket        = K.ticket + 2;
            K.row_order     = F.redo_rows;
            K.row_count_dev = F.redo_count;
        }
    }
    switch (p->dtype) {
        case FTB200_F32: rc = sampling_launch<FTB200_F32>(K, StopArgs{}, grid, smem, st); break;
        case FTB200_F16: rc = sampling_launch<FTB200_F16>(K, StopArgs{}, grid, smem, st); break;
        default: rc = sampling_launch<FTB200_BF16>(K, StopArgs{}, grid, smem, st); break;
    }
    if (rc == FTB200_OK) {
        note_launch(1);
    }
    return rc;
}

static int vp_check(const ftb200_sampling_params* p, int vocab_offset, int cap, const void* records)
{
    if (records == nullptr || cap < 1 || cap > kCap || vocab_offset < 0) {
        set_error("ftb200_vocab_parallel_local: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (p != nullptr && (p->cum_log_probs != nullptr || p->output_log_probs != nullptr)) {
        set_error("ftb200_vocab_parallel_local: log-probs are not available with a sharded vocabulary");
        return FTB200_UNSUPPORTED;
    }
    return FTB200_OK;
}

extern "C" int ftb200_vocab_parallel_local(const ftb200_sampling_params* p, int vocab_offset, int cap,
                                           uint64_t* records)
{
    reset_launch_count();
    const int rc = vp_check(p, vocab_offset, cap, records);
    return rc != FTB200_OK ? rc : vp_local(p, vocab_offset, cap, records);
}

extern "C" int ftb200_vocab_parallel_shards(const ftb200_sampling_params* p, const void* const* logits, int n_shards,
                                            int shard_size, int cap, uint64_t* records)
{
    reset_launch_count();
    int rc = vp_check(p, 0, cap, records);
    if (rc == FTB200_OK && (p == nullptr || logits == nullptr || n_shards < 1 || shard_size < 1)) {
        set_error("ftb200_vocab_parallel_shards: invalid argument");
        rc = FTB200_INVALID_ARG;
    }
    if (rc != FTB200_OK) {
        return rc;
    }
    // the argument block of a shard: its columns in memory, and of the vocabulary what lies in it
    ftb200_sampling_params q = *p;
    q.logits                 = logits[0];
    q.vocab_size_padded      = shard_size;
    const auto columns       = [&](int i) {
        const long long left = (long long)p->vocab_size - (long long)i * shard_size;
        return (int)(left < 1 ? 1 : (left < shard_size ? left : shard_size));
    };
    q.vocab_size = columns(0);
    KParams K;
    size_t  smem = 0, vsmem = 0;
    int     grid = 0;
    rc           = plan_sampling(&q, K, smem, grid, true);
    if (rc != FTB200_OK) {
        return rc;
    }
    if (p->local_batch_size == 0) {
        return FTB200_OK;
    }
    VpArgs V;
    K.vp_out = (u64*)records, K.vp_cap = cap;
    if (plan_vp_select(&q, K, logits, n_shards, 0, cap, K.vp_out, &V, &vsmem)) {
        V.vocab = p->vocab_size;
        return launch_vp_select(K, V, vsmem, (cudaStream_t)p->stream);
    }
    for (int i = 0; i < n_shards && rc == FTB200_OK; ++i) {
        q.logits     = logits[i];
        q.vocab_size = columns(i);
        rc           = vp_local(&q, i * shard_size, cap, records + (size_t)i * p->local_batch_size * (cap + 2));
    }
    return rc;
}

extern "C" int ftb200_vocab_parallel_merge(const ftb200_sampling_params* p, const uint64_t* gathered, int n_ranks,
                                           int cap, int* overflow_count)
{
    reset_launch_count();
    if (gathered == nullptr || overflow_count == nullptr || n_ranks < 1 || cap < 1 || cap > kCap) {
        set_error("ftb200_vocab_parallel_merge: invalid argument");
        return FTB200_INVALID_ARG;
    }
    KParams K;
    size_t  smem = 0;
    int     grid = 0;
    int     rc   = plan_sampling(p, K, smem, grid, false);
    if (rc != FTB200_OK) {
        return rc;
    }
    if (p->local_batch_size == 0) {
        return FTB200_OK;
    }
    K.vp_cap        = cap;
    cudaStream_t st = (cudaStream_t)p->stream;
    grid            = sm_count() * 4 < p->local_batch_size ? sm_count() * 4 : p->local_batch_size;
    switch (p->dtype) {
        case FTB200_F32: rc = vp_merge_launch<FTB200_F32>(K, (const u64*)gathered, n_ranks, overflow_count, grid, st); break;
        case FTB200_F16: rc = vp_merge_launch<FTB200_F16>(K, (const u64*)gathered, n_ranks, overflow_count, grid, st); break;
        default: rc = vp_merge_launch<FTB200_BF16>(K, (const u64*)gathered, n_ranks, overflow_count, grid, st); break;
    }
    if (rc == FTB200_OK) {
        note_launch(1);
    }
    return rc;
}
