// Caller-side steps either side of the per-step decode path: start-of-decoding state, back-tracking of beam
// parents into final sequences, ranking of archived hypotheses, and archiving of unfinished beams.
// Replaces invokeDecodingInitialize (kernels/decoding_kernels.cu:26-64), invokeGatherTree (:452-646),
// invokeFinalize (:698-804) and invokeInsertUnfinishedPath (kernels/beam_search_topk_kernels.cu:788-843).
//
// The reference walks every parent chain with one thread and dependent global loads (one thread per batch
// entry for the archive).  Here one CTA serves a batch entry: the whole CTA stages a tile of time levels of the
// id / parent tables in shared memory with coalesced loads, one thread per beam follows its chain through the
// tile in shared memory, and the CTA writes results back with coalesced stores.
#include <limits.h>

#include <mutex>

#include "chains.cuh"
#include "common.cuh"
#include "ftb200.h"

namespace ftb200 {

namespace {

constexpr int kDkThreads = 256;
constexpr int kStage     = 2048;  // table entries (levels x beams) staged per tile
constexpr int kMaxBeams  = 1024;  // the reference's launch shapes stop here as well (:636-645, :787-789)
constexpr int kMaxArchiveBeams = 512;  // 2 * beam_width slots per entry have to fit a block there (:787-789)

template<typename T>
__device__ __forceinline__ T start_score_floor();
template<>
__device__ __forceinline__ float start_score_floor<float>()
{
    return -1e20f;
}
template<>
__device__ __forceinline__ __half start_score_floor<__half>()
{
    return __float2half(-65504.0f);
}
template<>
__device__ __forceinline__ __nv_bfloat16 start_score_floor<__nv_bfloat16>()
{
    return __float2bfloat16(-1e20f);
}

template<typename T>
__global__ void decoding_initialize_kernel(uint8_t* finished, int* sequence_length, int* word_ids, T* cum_log_probs,
                                           const int* sentence_ids, int n, int beam_width, int max_input_length)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += blockDim.x * gridDim.x) {
        finished[i]        = 0;
        sequence_length[i] = max_input_length;
        if (word_ids != nullptr) {
            word_ids[i] = sentence_ids[i / beam_width];
        }
        cum_log_probs[i] = (i % beam_width == 0) ? T(0.0f) : start_score_floor<T>();
    }
}

// ---- gather tree ------------------------------------------------------------------------------------------
struct GatherTree {
    int*       beams;
    int*       max_sequence_lengths;
    int        final_step;
    const int* input_lengths;
    int*       response_input_lengths;
    int        max_time, batch_size, beam_width;
    const int* step_ids;
    const int* parent_ids;
    const int* end_tokens;
    int        max_input_length;
    const int* prefix_lengths;
    const int* virtual_lengths;
    int        max_input_without_prompt_length, max_prefix_length;
    int*       output_ids;
    int        by_maps;  // the tables of tree_by_maps() fit
};

__global__ void __launch_bounds__(kDkThreads) gather_tree_kernel(GatherTree p)
{
    wait_for_previous();
    __shared__ int     s_ids[kStage], s_par[kStage];
    __shared__ int     s_parent[kMaxBeams];
    __shared__ uint8_t s_bad[kMaxBeams];
    __shared__ int     s_maxlen;

    const int    b = blockIdx.x, K = p.beam_width, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t BK = (size_t)p.batch_size * K, col0 = (size_t)b * K;
    const int    max_input_length = p.input_lengths == nullptr ? 0 : p.max_input_length;
    const int    prompt_len = p.prefix_lengths == nullptr ? 0 : p.prefix_lengths[b];
    const int    virt = p.virtual_lengths == nullptr ? 0 : p.virtual_lengths[b];
    const int    trimmed = p.max_prefix_length + (p.max_input_length - p.max_input_without_prompt_length);
    const int    end = p.end_tokens[b];
    auto         at = [&](int time, int beam) { return BK * (size_t)time + col0 + beam; };
    auto         in_len = [&](int beam) { return (p.input_lengths == nullptr ? 0 : p.input_lengths[col0 + beam]) - virt; };

    if (tid == 0) {
        s_maxlen = -1;
    }
    __syncthreads();
    // Every reference thread of a batch entry rewrites all of its lengths from the values it read; in lockstep
    // that is one update per entry, which is what is done here.
    for (int j = tid; j < K; j += kDkThreads) {
        const int tmp_len               = p.max_sequence_lengths[col0 + j] + p.final_step;
        p.max_sequence_lengths[col0 + j] = tmp_len - trimmed;
        if (p.response_input_lengths != nullptr) {
            p.response_input_lengths[col0 + j] = in_len(j) - prompt_len;
        }
        atomicMax(&s_maxlen, tmp_len);
    }
    __syncthreads();
    const int max_len = s_maxlen, top = min(p.max_time, max_len);
    if (top <= 0) {
        return;
    }

    // level top-1: the beam's own last token
    for (int beam = tid; beam < K; beam += kDkThreads) {
        const int shift = max_input_length - in_len(beam) + prompt_len;
        const int tgt   = top - 1 - shift;
        if (tgt >= 0) {  // the reference writes without this check
            p.beams[at(tgt, beam)] = p.step_ids[at(top - 1, beam)];
        }
        s_parent[beam] = p.parent_ids == nullptr ? 0 : p.parent_ids[at(top - 1, beam)] % K;
        s_bad[beam]    = 0;
    }
    // levels top-2 .. 0 in tiles of `tl` levels
    const int tl = kStage / K;
    for (int hi = top - 1; hi > 0; hi -= tl) {
        const int lo = max(0, hi - tl), n = (hi - lo) * K;
        __syncthreads();
        for (int e = tid; e < n; e += kDkThreads) {
            const size_t g = BK * (size_t)(lo + e / K) + col0 + e % K;
            s_ids[e]       = p.step_ids[g];
            s_par[e]       = p.parent_ids == nullptr ? 0 : p.parent_ids[g];
        }
        __syncthreads();
        for (int beam = tid; beam < K; beam += kDkThreads) {
            const int input_len = in_len(beam), shift = max_input_length - input_len + prompt_len;
            int       parent = s_parent[beam];
            bool      bad    = s_bad[beam];
            for (int level = hi - 1; level >= lo; --level) {
                if (level < prompt_len || (level >= input_len && level < max_input_length)) {
                    continue;
                }
                const int tgt = level >= max_input_length ? level - shift : level - prompt_len;
                if (parent < 0 || parent > K) {
                    p.beams[at(tgt, beam)] = end;
                    parent                 = -1;
                    bad                    = true;
                }
                else {
                    const int e            = (level - lo) * K + parent;
                    p.beams[at(tgt, beam)] = s_ids[e];
                    const int v            = s_par[e];  // in [0, K) on a well-formed tree: skip the division
                    parent                 = (unsigned)v < (unsigned)K ? v : v % K;
                }
            }
            s_parent[beam] = parent;
            s_bad[beam]    = bad;
        }
    }
    __syncthreads();

    // One warp per beam: end tokens after the sequence, nothing but end tokens after the first one, transposition.
    const int out_len = p.max_time - trimmed;
    for (int beam = wid; beam < K; beam += kDkThreads / 32) {
        const int shift = max_input_length - in_len(beam) + prompt_len;
        for (int t = max(0, max_len - shift) + lane; t < p.max_time - p.max_prefix_length; t += 32) {
            p.beams[at(t, beam)] = end;
        }
        __syncwarp();
        if (!s_bad[beam]) {
            int first = INT_MAX;
            for (int t = (max_input_length == 0 ? 1 : max_input_length) + lane; t < top; t += 32) {
                if (p.beams[at(t, beam)] == end) {
                    first = t;
                    break;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
            }
            if (first != INT_MAX) {
                for (int t = first + 1 + lane; t < top; t += 32) {
                    p.beams[at(t, beam)] = end;
                }
            }
        }
        __syncwarp();
        if (p.output_ids != nullptr) {
            int* out = p.output_ids + (col0 + beam) * (size_t)out_len;
            for (int j = lane; j < out_len; j += 32) {
                out[j] = p.beams[at(j, beam)];
            }
        }
    }
}

// ---- the tree in registers --------------------------------------------------------------------------------------
// A level's parents are a map of at most eight values (the beams, and "no parent", which stays): eight nibbles of a word.
constexpr u32 kMapIdentity = 0x76543210u;
constexpr int kTreeBeams = 7, kTreeLevels = 4;  // beams of a map, levels of a thread, at most
// first f, then g: two byte selections, with g spread to bytes and the result packed again
__device__ __forceinline__ u32 map_then(u32 f, u32 g)
{
    auto spread = [](u32 x) {
        x = (x | (x << 8)) & 0x00ff00ffu;
        return (x | (x << 4)) & 0x0f0f0f0fu;
    };
    auto pack = [](u32 x) {
        x = (x | (x >> 4)) & 0x00ff00ffu;
        return (x | (x >> 8)) & 0xffffu;
    };
    const u32 lo = spread(g & 0xffffu), hi = spread(g >> 16);
    return pack(__byte_perm(lo, hi, f & 0xffffu)) | (pack(__byte_perm(lo, hi, f >> 16)) << 16);
}
__device__ __forceinline__ int map_of(u32 m, int x)
{
    return (int)((m >> (4 * x)) & 15u);
}

// Up to KB beams that have prompts of one length, and up to LV levels for each thread.  Parents and tokens go into shared memory,
// neighbouring lanes to neighbouring words (a level is 4 K bytes of a row of all entries, so the number of lines that a
// warp's load touches is what it costs); a thread holds the maps of its levels (consecutive ones, from the top down); one scan
// over their compositions says where each beam's chain enters them; the tokens found go to where the parents were, and from
// there into the tree and its transposed copy, each element written once.  Returns false, with nothing written, for entries of
// another form.
template<int KB, int LV>
__device__ __forceinline__ bool tree_by_maps(const GatherTree& p, unsigned char* smem)
{
    __shared__ int s_top_token[KB];  // position of a beam's first end token
    __shared__ u32 s_warp[kChainThreads / 32], s_broken;
    const int      b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, K = p.beam_width, T = p.max_time;
    const size_t   BK = (size_t)p.batch_size * K, col0 = (size_t)b * K;
    const int      L = (T + kChainThreads - 1) / kChainThreads, first = T - 1 - tid * L;  // the thread's highest level
    int* const     s_tok = (int*)smem;       // [T][K]
    int* const     s_par = s_tok + T * K;    // [T][K]; then the token of every position
    FTB_ASSUME_SHARED(s_tok);
    FTB_ASSUME_SHARED(s_par);
    const int step = kChainThreads / K, col = tid % K, t0 = tid / K;
    if (t0 < step) {
        constexpr int U = 8;
        for (int t = t0; t < T; t += U * step) {
            int v[U], w[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool   in = t + u * step < T;
                const size_t g  = BK * (size_t)(t + u * step) + col0 + col;
                v[u]            = in ? __ldg(p.step_ids + g) : 0;
                w[u]            = in && p.parent_ids != nullptr ? __ldg(p.parent_ids + g) : 0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (t + u * step < T) {
                    s_tok[(t + u * step) * K + col] = v[u];
                    s_par[(t + u * step) * K + col] = w[u];
                }
            }
        }
    }
    const int max_il = p.input_lengths == nullptr ? 0 : p.max_input_length;
    const int prompt_len = p.prefix_lengths == nullptr ? 0 : p.prefix_lengths[b];
    const int virt       = p.virtual_lengths == nullptr ? 0 : p.virtual_lengths[b];
    const int len        = (p.input_lengths == nullptr ? 0 : p.input_lengths[col0]) - virt;
    const int end        = p.end_tokens[b];
    const int trimmed    = p.max_prefix_length + (p.max_input_length - p.max_input_without_prompt_length);
    int       max_len    = -1;
    bool      even       = true;
#pragma unroll
    for (int k = 0; k < KB; ++k) {
        if (k < K) {
            max_len = max(max_len, p.max_sequence_lengths[col0 + k] + p.final_step);
            even    = even && (p.input_lengths == nullptr ? 0 : p.input_lengths[col0 + k]) - virt == len;
        }
    }
    const int top = min(T, max_len), shift = max_il - len + prompt_len;
    // (then positions 0 .. top - 1 - shift are those of the prompt's and the generated levels, one after the other)
    if (!(even && prompt_len >= 0 && prompt_len <= len && len <= max_il && top > max_il)) {
        __syncthreads();  // (the tables are laid out anew)
        return false;
    }
    if (tid < KB) {
        s_top_token[tid] = INT_MAX;
    }
    if (tid == 0) {
        s_broken = 0;
    }
    __syncthreads();

    // ---- the maps, and the composition of those of the threads in front ----
    auto skipped = [&](int level) { return level < prompt_len || (level >= len && level < max_il); };
    u32  m[LV], all = kMapIdentity;
#pragma unroll
    for (int l = 0; l < LV; ++l) {
        const int level = first - l;
        m[l]            = kMapIdentity;
        if (l < L && level >= 0 && level < top && (level == top - 1 || !skipped(level))) {
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                if (k < K) {
                    int v = s_par[level * K + k];
                    v     = (unsigned)v < (unsigned)K ? v : v % K;
                    v     = v < 0 ? K : v;
                    m[l]  = (m[l] & ~(15u << (4 * k))) | ((u32)v << (4 * k));
                }
            }
        }
        all = map_then(all, m[l]);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 before = __shfl_up_sync(0xffffffffu, all, o);
        all              = lane >= o ? map_then(before, all) : all;
    }
    u32 entry = __shfl_up_sync(0xffffffffu, all, 1);
    entry     = lane == 0 ? kMapIdentity : entry;
    if (lane == 31) {
        s_warp[wid] = all;
    }
    __syncthreads();
    if (wid == 0) {
        u32 w = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 before = __shfl_up_sync(0xffffffffu, w, o);
            w                = lane >= o ? map_then(before, w) : w;
        }
        s_warp[lane] = w;
    }
    else if (wid == 1 && lane < K) {
        // (one update of the lengths per entry: see gather_tree_kernel; all threads have read them)
        p.max_sequence_lengths[col0 + lane] = p.max_sequence_lengths[col0 + lane] + p.final_step - trimmed;
        if (p.response_input_lengths != nullptr) {
            p.response_input_lengths[col0 + lane] = len - prompt_len;
        }
    }
    __syncthreads();
    entry = map_then(wid > 0 ? s_warp[wid - 1] : kMapIdentity, entry);

    // ---- tokens along the chains; a chain that broke off gives the end token.  Positions behind the sequence: end tokens, or
    // what the caller left ----
    const int first_t = max_il == 0 ? 1 : max_il, fill = max(0, max_len - shift), fill_end = T - p.max_prefix_length;
    const int out_len = T - trimmed, behind = top - shift;
    auto      at      = [&](int t, int j) { return BK * (size_t)t + col0 + j; };
    u32       broken  = 0;
#pragma unroll
    for (int l = 0; l < LV; ++l) {
        const int level = first - l;
        if (l < L && level >= 0 && level < top && !skipped(level)) {
            const int t = level < max_il ? level - prompt_len : level - shift;
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                if (j < K) {
                    const int from = map_of(entry, j), w = from == K ? end : s_tok[level * K + from];
                    broken |= from == K ? 1u << j : 0u;
                    if (t >= first_t && t < top && w == end) {
                        atomicMin(&s_top_token[j], t);
                    }
                    s_par[t * K + j] = w;
                }
            }
        }
        entry = map_then(entry, m[l]);
    }
    if (broken != 0) {
        atomicOr(&s_broken, broken);
    }
    if (t0 < step) {
        for (int t = behind + t0; t < T; t += step) {
            const int w        = t >= fill && t < fill_end ? end : p.beams[at(t, col)];
            s_par[t * K + col] = w;
            if (t >= first_t && t < top && w == end) {
                atomicMin(&s_top_token[col], t);
            }
        }
    }
    __syncthreads();

    // ---- nothing but end tokens after the first one ----
    if (t0 < step) {
        const int cut_from = (s_broken >> col) & 1u ? INT_MAX : s_top_token[col];
        int*      out      = p.output_ids == nullptr ? nullptr : p.output_ids + (col0 + col) * (size_t)out_len;
#pragma unroll 4
        for (int t = t0; t < T; t += step) {
            const bool over = t > cut_from && t < top;
            const int  w    = over ? end : s_par[t * K + col];
            if (t < behind || over || (t >= fill && t < fill_end)) {
                p.beams[at(t, col)] = w;
            }
            if (out != nullptr && t < out_len) {
                out[t] = w;
            }
        }
    }
    return true;
}

// The tree with the whole parent table of an entry in shared memory.  Bound by latency: 8 levels of ids and parents in
// flight per thread, then the chains, then one pass that writes and one that cuts and transposes.
// 64 entries x 4 beams x 2048 levels: 245 us with one thread per chain, 14.8 us this way (parents 4.7, walks 3.5, tokens 4.5, end
// tokens 1.2), 18.4 a call; 12.7 a call by maps in registers, which serve up to seven beams and 4096 levels.
__global__ void __launch_bounds__(kChainThreads) gather_tree_chains_kernel(GatherTree p)
{
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    if (p.by_maps && tree_by_maps<kTreeBeams, kTreeLevels>(p, smem)) {
        return;
    }
    __shared__ int     s_start[kMaxBeams], s_from[kMaxBeams], s_first[kMaxBeams];
    __shared__ uint8_t s_bad[kMaxBeams];
    __shared__ int     s_maxlen, s_uneven;

    const int    b = blockIdx.x, K = p.beam_width, tid = threadIdx.x;
    const size_t BK = (size_t)p.batch_size * K, col0 = (size_t)b * K;
    const int    max_input_length = p.input_lengths == nullptr ? 0 : p.max_input_length;
    const int    prompt_len = p.prefix_lengths == nullptr ? 0 : p.prefix_lengths[b];
    const int    virt = p.virtual_lengths == nullptr ? 0 : p.virtual_lengths[b];
    const int    trimmed = p.max_prefix_length + (p.max_input_length - p.max_input_without_prompt_length);
    const int    end = p.end_tokens[b];
    auto         at = [&](int time, int beam) { return BK * (size_t)time + col0 + beam; };
    auto         in_len = [&](int beam) { return (p.input_lengths == nullptr ? 0 : p.input_lengths[col0 + beam]) - virt; };

    if (tid == 0) {
        s_maxlen = -1;
        s_uneven = 0;
    }
    __syncthreads();
    // (one update of the lengths per entry: see gather_tree_kernel)
    for (int j = tid; j < K; j += kChainThreads) {
        const int tmp_len                = p.max_sequence_lengths[col0 + j] + p.final_step;
        p.max_sequence_lengths[col0 + j] = tmp_len - trimmed;
        if (p.response_input_lengths != nullptr) {
            p.response_input_lengths[col0 + j] = in_len(j) - prompt_len;
        }
        atomicMax(&s_maxlen, tmp_len);
        if (in_len(j) != in_len(0)) {
            s_uneven = 1;
        }
    }
    __syncthreads();
    const int max_len = s_maxlen, top = min(p.max_time, max_len);
    if (top <= 0) {
        return;
    }
    const int levels = top - 1;  // levels below the beam's own last token
    auto      skipped = [&](int level, int len) { return level < prompt_len || (level >= len && level < max_input_length); };
    const Chains c = map_chains(smem, levels, K, s_start, s_from);
    const u32    row = 2u * (u32)(K + 1);
    // every thread keeps to one beam (no division in the loops) and takes every step-th level or position of it
    const int  step = kChainThreads / K, j = tid % K, t0 = tid / K;
    const bool busy = t0 < step;
    const int  len = in_len(j), len0 = in_len(0), shift = max_input_length - len + prompt_len;
    if (busy) {
#pragma unroll 8
        for (int level = t0; level < levels; level += step) {
            int v              = p.parent_ids == nullptr ? 0 : __ldg(p.parent_ids + at(level, j));
            v                  = (unsigned)v < (unsigned)K ? v : v % K;
            v                  = s_uneven == 0 && skipped(level, len0) ? j : (v < 0 ? K : v);  // a skipped level passes on
            sts_u16(c.par + (u32)level * row + 2u * (u32)j, 2u * (u32)v);
            if (j == 0) {
                sts_u16(c.par + (u32)level * row + 2u * (u32)K, 2u * (u32)K);
            }
        }
    }
    for (int k = tid; k < K; k += kChainThreads) {
        const int v = p.parent_ids == nullptr ? 0 : p.parent_ids[at(top - 1, k)] % K;
        s_start[k]  = levels;
        s_from[k]   = v < 0 ? K : v;
        s_bad[k]    = 0;
        s_first[k]  = INT_MAX;
    }
    __syncthreads();
    if (s_uneven == 0) {
        walk_chains(c);
    }
    else {
        // beams of different prompt lengths skip different levels: one chain after the other
        for (int k = tid; k < K; k += kChainThreads) {
            const int lk  = in_len(k);
            int       cur = s_from[k];
            for (int level = levels - 1; level >= 0; --level) {
                sts_u16(c.sel + 2u * (u32)(level * K + k), (u32)cur);
                if (!skipped(level, lk)) {
                    cur = (int)lds_u16(c.par + (u32)level * row + 2u * (u32)cur) / 2;
                }
            }
        }
        __syncthreads();
    }
    // Position t of the beam: end tokens after the sequence, else the token of the level that lands there (levels of the
    // prompt first, then the generated ones, then the beam's own last token), else what the caller left.  Where a chain
    // broke off everything below is the end token, and the cut after the first end token is left out.
    const int     first_t = max_input_length == 0 ? 1 : max_input_length;
    const int     fill = max(0, max_len - shift), fill_end = p.max_time - p.max_prefix_length;
    const int     out_len = p.max_time - trimmed;
    constexpr int U = 8, R = 2;  // positions in flight, batches of them kept in registers
    int           v[R][U];
    auto          batch = [&](int t1, int* w) {
        bool put[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t1 + u * step;
            put[u]      = false;
            if (t < p.max_time) {
                const int la = t + prompt_len, lb = t + shift;
                int       level = lb < levels && lb >= max_input_length && lb >= prompt_len ? lb : -1;
                level           = la < levels && la < max_input_length && la < len ? la : level;
                const int from  = level >= 0 ? (int)lds_u16(c.sel + 2u * (u32)(level * K + j)) : j;
                level           = level < 0 && t == top - 1 - shift ? top - 1 : level;
                put[u]          = true;
                if ((t >= fill && t < fill_end) || (level >= 0 && from == K)) {
                    w[u] = end;
                    if (level >= 0 && from == K) {
                        s_bad[j] = 1;
                    }
                }
                else if (level >= 0) {
                    w[u] = __ldg(p.step_ids + at(level, from));
                }
                else {
                    put[u] = false;
                    w[u]   = p.beams[at(t, j)];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int t = t1 + u * step;
            if (put[u]) {
                p.beams[at(t, j)] = w[u];
            }
            if (t < p.max_time && t >= first_t && t < top && w[u] == end) {
                atomicMin(&s_first[j], t);
            }
        }
    };
    if (busy) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            batch(t0 + r * U * step, v[r]);
        }
        for (int t1 = t0 + R * U * step; t1 < p.max_time; t1 += U * step) {
            int w[U];
            batch(t1, w);
        }
    }
    __syncthreads();
    // nothing but end tokens after the first one, and the transposed copy (each thread meets what it wrote itself)
    if (busy) {
        const int cut_from = s_bad[j] || s_first[j] == INT_MAX ? INT_MAX : s_first[j];
        int*      out = p.output_ids == nullptr ? nullptr : p.output_ids + (col0 + j) * (size_t)out_len;
        auto      finish = [&](int t, int w) {
            const bool cut = t > cut_from && t < top;
            if (cut) {
                p.beams[at(t, j)] = end;
            }
            if (out != nullptr && t < out_len) {
                out[t] = cut ? end : w;
            }
        };
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int t = t0 + (r * U + u) * step;
                if (t < p.max_time) {
                    finish(t, v[r][u]);
                }
            }
        }
        for (int t = t0 + R * U * step; t < p.max_time; t += step) {
            finish(t, p.beams[at(t, j)]);
        }
    }
}

// ---- finalize ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kDkThreads) finalize_kernel(int* output_ids, int* sequence_lengths,
                                                              float* cum_log_probs, float* output_log_probs,
                                                              const int* topk_output_ids,
                                                              const int* topk_sequence_lengths, const float* scores,
                                                              const float* topk_cum_log_probs,
                                                              const float* topk_log_probs, const int* num_beams,
                                                              int K, int max_seq_len)
{
    wait_for_previous();
    __shared__ float s_score[2 * kMaxBeams];
    __shared__ int   s_rank[kMaxBeams];
    const int        b = blockIdx.x, tid = threadIdx.x, n = max(0, min(num_beams[b], 2 * K));
    for (int j = tid; j < n; j += kDkThreads) {
        s_score[j] = scores[(size_t)b * 2 * K + j];
    }
    // The reference picks the largest remaining score K times, the first index winning ties; once the n
    // archived entries are used up it finds entry 0 again.
    for (int i = tid; i < K; i += kDkThreads) {
        s_rank[i] = 0;
    }
    __syncthreads();
    for (int j = tid; j < n; j += kDkThreads) {
        const float s = s_score[j];
        int         r = 0;
        for (int l = 0; l < n; ++l) {
            const float o = s_score[l];
            r += (o > s) || (o == s && l < j);
        }
        if (r < K) {
            s_rank[r] = j;
        }
    }
    __syncthreads();
    for (int beam = tid; blockIdx.y == 0 && beam < K; beam += kDkThreads) {
        const size_t src = (size_t)b * 2 * K + s_rank[beam];
        sequence_lengths[(size_t)b * K + beam] = topk_sequence_lengths[src];
        if (cum_log_probs != nullptr) {
            cum_log_probs[(size_t)b * K + beam] = topk_cum_log_probs[src];
        }
    }
    for (int beam = blockIdx.y; beam < K; beam += gridDim.y) {
        const size_t src = ((size_t)b * 2 * K + s_rank[beam]) * (size_t)(max_seq_len + 1);
        const size_t dst = ((size_t)b * K + beam) * (size_t)max_seq_len;
        const int    len = topk_sequence_lengths[(size_t)b * 2 * K + s_rank[beam]];
        for (int i = tid; i < len; i += kDkThreads) {  // position 0 of the archive is the start token
            output_ids[dst + i] = topk_output_ids[src + i + 1];
            if (output_log_probs != nullptr) {
                output_log_probs[dst + i] = topk_log_probs[src + i + 1];
            }
        }
    }
}

// ---- archive of unfinished beams ----------------------------------------------------------------------------
struct InsertPath {
    int*         output_ids_tgt;
    int*         sequence_lengths_tgt;
    float*       cum_log_probs_tgt;
    float*       normed_scores;
    float*       log_probs_tgt;
    int*         num_beams;
    const uint8_t* is_done;
    const int*   output_ids_src;
    const int*   parent_ids_src;
    const int*   sequence_lengths_src;
    const float* log_probs_src;
    int          max_seq_len;
    float        length_penalty;
    const uint8_t* finished;
    const float* cum_log_probs;
    int          batch_size, beam_width;
};

__global__ void __launch_bounds__(kDkThreads) insert_unfinished_path_kernel(InsertPath p)
{
    wait_for_previous();
    __shared__ int   s_ids[kStage], s_par[kStage], s_out[kStage];
    __shared__ float s_lp[kStage], s_lpout[kStage];
    __shared__ int   s_prev[kMaxArchiveBeams], s_len[kMaxArchiveBeams];
    __shared__ int   s_top;

    const int b = blockIdx.x, K = p.beam_width, tid = threadIdx.x;
    if (p.is_done[b]) {
        return;
    }
    const size_t BK = (size_t)p.batch_size * K, col0 = (size_t)b * K;
    const int    first_slot = p.num_beams[b];
    const size_t row = (size_t)p.max_seq_len + 1;
    const bool   with_lp = p.log_probs_tgt != nullptr && p.log_probs_src != nullptr;
    if (tid == 0) {
        s_top = -1;
    }
    __syncthreads();
    for (int beam = tid; beam < K; beam += kDkThreads) {
        const int    len = p.sequence_lengths_src[col0 + beam];
        const size_t tgt = (size_t)b * 2 * K + beam + first_slot;
        const size_t g   = (size_t)len * BK + col0 + beam;
        s_len[beam]      = len;
        p.output_ids_tgt[tgt * row + len] = p.output_ids_src[g];
        if (with_lp) {
            p.log_probs_tgt[tgt * row + len] = p.log_probs_src[g];
        }
        s_prev[beam]                = p.parent_ids_src[g];
        p.sequence_lengths_tgt[tgt] = len;
        const float cum   = p.cum_log_probs[col0 + beam];
        const int   n_tok = p.finished[col0 + beam] ? len + 1 : len;
        p.normed_scores[tgt] =
            (p.length_penalty == 0.0f || n_tok == 1) ? cum : cum / powf((float)n_tok, p.length_penalty);
        p.cum_log_probs_tgt[tgt] = cum;
        atomicMax(&s_top, len);
    }
    __syncthreads();
    const int top = s_top, tl = kStage / K;
    for (int hi = top; hi > 0; hi -= tl) {  // levels hi-1 .. lo
        const int lo = max(0, hi - tl), n = (hi - lo) * K;
        __syncthreads();
        for (int e = tid; e < n; e += kDkThreads) {
            const size_t g = BK * (size_t)(lo + e / K) + col0 + e % K;
            s_ids[e]       = p.output_ids_src[g];
            s_par[e]       = p.parent_ids_src[g];
            if (with_lp) {
                s_lp[e] = p.log_probs_src[g];
            }
        }
        __syncthreads();
        for (int beam = tid; beam < K; beam += kDkThreads) {
            int prev = s_prev[beam];
            for (int level = min(hi, s_len[beam]) - 1; level >= lo; --level) {
                prev        = min(max(prev, 0), K - 1);  // the reference follows an out-of-range parent unchecked
                const int e = (level - lo) * K + prev, o = (level - lo) * K + beam;
                s_out[o]    = s_ids[e];
                if (with_lp) {
                    s_lpout[o] = s_lp[e];
                }
                prev = s_par[e];
            }
            s_prev[beam] = prev;
        }
        __syncthreads();
        // rows of the archive are contiguous in the level: flush level-major per beam
        const int levels = hi - lo;
        for (int e = tid; e < levels * K; e += kDkThreads) {
            const int beam = e / levels, level = lo + e % levels;
            if (level < s_len[beam]) {
                const size_t tgt = (size_t)b * 2 * K + beam + first_slot;
                const int    o   = (level - lo) * K + beam;
                p.output_ids_tgt[tgt * row + level] = s_out[o];
                if (with_lp) {
                    p.log_probs_tgt[tgt * row + level] = s_lpout[o];
                }
            }
        }
    }
    if (tid == 0) {
        p.num_beams[b] = first_slot + K;
    }
}

// The archive with the whole parent table of an entry in shared memory (see walk_chains).
__global__ void __launch_bounds__(kChainThreads) insert_chains_kernel(InsertPath p)
{
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_start[kMaxArchiveBeams], s_from[kMaxArchiveBeams];
    __shared__ int s_top;

    const int b = blockIdx.x, K = p.beam_width, tid = threadIdx.x;
    if (p.is_done[b]) {
        return;
    }
    const size_t BK = (size_t)p.batch_size * K, col0 = (size_t)b * K;
    const int    first_slot = p.num_beams[b];
    const size_t row = (size_t)p.max_seq_len + 1;
    const bool   with_lp = p.log_probs_tgt != nullptr && p.log_probs_src != nullptr;
    if (tid == 0) {
        s_top = 0;
    }
    __syncthreads();
    for (int beam = tid; beam < K; beam += kChainThreads) {
        const int    len = p.sequence_lengths_src[col0 + beam];
        const size_t tgt = (size_t)b * 2 * K + beam + first_slot;
        const size_t g   = (size_t)len * BK + col0 + beam;
        p.output_ids_tgt[tgt * row + len] = p.output_ids_src[g];
        if (with_lp) {
            p.log_probs_tgt[tgt * row + len] = p.log_probs_src[g];
        }
        s_start[beam]               = min(len, p.max_seq_len);
        s_from[beam]                = min(max(p.parent_ids_src[g], 0), K - 1);  // the reference follows it unchecked
        p.sequence_lengths_tgt[tgt] = len;
        const float cum   = p.cum_log_probs[col0 + beam];
        const int   n_tok = p.finished[col0 + beam] ? len + 1 : len;
        p.normed_scores[tgt] =
            (p.length_penalty == 0.0f || n_tok == 1) ? cum : cum / powf((float)n_tok, p.length_penalty);
        p.cum_log_probs_tgt[tgt] = cum;
        atomicMax(&s_top, s_start[beam]);
    }
    __syncthreads();
    const int    levels = s_top;
    const Chains c = map_chains(smem, levels, K, s_start, s_from);
    const u32    row_bytes = 2u * (u32)(K + 1);
    const int  step = kChainThreads / K, j = tid % K, t0 = tid / K;  // one beam per thread, every step-th level of it
    const bool busy = t0 < step;
    if (busy) {
#pragma unroll 8
        for (int level = t0; level < levels; level += step) {
            const int v = min(max(__ldg(p.parent_ids_src + BK * (size_t)level + col0 + j), 0), K - 1);
            sts_u16(c.par + (u32)level * row_bytes + 2u * (u32)j, 2u * (u32)v);
            if (j == 0) {
                sts_u16(c.par + (u32)level * row_bytes + 2u * (u32)K, 2u * (u32)K);
            }
        }
    }
    __syncthreads();
    walk_chains(c);
    if (busy) {
        const size_t tgt = ((size_t)b * 2 * K + j + first_slot) * row;
        const int    n = s_start[j];
        constexpr int U = 8;
        for (int l0 = t0; l0 < n; l0 += U * step) {
            int   id[U];
            float lp[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int level = l0 + u * step;
                if (level < n) {
                    const size_t g = BK * (size_t)level + col0 + lds_u16(c.sel + 2u * (u32)(level * K + j));
                    id[u]          = __ldg(p.output_ids_src + g);
                    lp[u]          = with_lp ? __ldg(p.log_probs_src + g) : 0.0f;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int level = l0 + u * step;
                if (level < n) {
                    p.output_ids_tgt[tgt + level] = id[u];
                    if (with_lp) {
                        p.log_probs_tgt[tgt + level] = lp[u];
                    }
                }
            }
        }
    }
    if (tid == 0) {
        p.num_beams[b] = first_slot + K;
    }
}

}  // namespace
}  // namespace ftb200

using namespace ftb200;

extern "C" int ftb200_decoding_initialize(uint8_t* finished, int* sequence_length, int* word_ids,
                                          void* cum_log_probs, int dtype, const int* sentence_ids, int batch_size,
                                          int beam_width, int max_input_length, void* stream)
{
    if (finished == nullptr || sequence_length == nullptr || cum_log_probs == nullptr || batch_size <= 0
        || beam_width <= 0 || (word_ids != nullptr && sentence_ids == nullptr)) {
        set_error("ftb200_decoding_initialize: invalid argument");
        return FTB200_INVALID_ARG;
    }
    const int    n = batch_size * beam_width, grid = (n + 255) / 256;
    cudaStream_t st = (cudaStream_t)stream;
    switch (dtype) {
        case FTB200_F32:
            decoding_initialize_kernel<float><<<grid, 256, 0, st>>>(finished, sequence_length, word_ids,
                                                                    (float*)cum_log_probs, sentence_ids, n,
                                                                    beam_width, max_input_length);
            break;
        case FTB200_F16:
            decoding_initialize_kernel<__half><<<grid, 256, 0, st>>>(finished, sequence_length, word_ids,
                                                                     (__half*)cum_log_probs, sentence_ids, n,
                                                                     beam_width, max_input_length);
            break;
        case FTB200_BF16:
            decoding_initialize_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(
                finished, sequence_length, word_ids, (__nv_bfloat16*)cum_log_probs, sentence_ids, n, beam_width,
                max_input_length);
            break;
        default:
            set_error("ftb200_decoding_initialize: unknown dtype");
            return FTB200_INVALID_ARG;
    }
    FTB_CUDA_CHECK(cudaGetLastError());
    note_launch(1);
    return FTB200_OK;
}

extern "C" int ftb200_gather_tree(const ftb200_gather_tree_params* a)
{
    if (a == nullptr || a->beams == nullptr || a->max_sequence_lengths == nullptr || a->step_ids == nullptr
        || a->end_tokens == nullptr || a->batch_size <= 0 || a->beam_width <= 0 || a->max_time < 0) {
        set_error("ftb200_gather_tree: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (a->beam_width > kMaxBeams) {
        set_error("ftb200_gather_tree: beam_width above 1024");
        return FTB200_UNSUPPORTED;
    }
    GatherTree p;
    p.beams                           = a->beams;
    p.max_sequence_lengths            = a->max_sequence_lengths;
    p.final_step                      = a->max_sequence_length_final_step;
    p.input_lengths                   = a->input_lengths;
    p.response_input_lengths          = a->response_input_lengths;
    p.max_time                        = a->max_time;
    p.batch_size                      = a->batch_size;
    p.beam_width                      = a->beam_width;
    p.step_ids                        = a->step_ids;
    p.parent_ids                      = a->parent_ids;
    p.end_tokens                      = a->end_tokens;
    p.max_input_length                = a->max_input_length;
    p.prefix_lengths                  = a->prefix_soft_prompt_lengths;
    p.virtual_lengths                 = a->p_prompt_tuning_prompt_lengths;
    p.max_input_without_prompt_length = a->max_input_without_prompt_length;
    p.max_prefix_length               = a->max_prefix_soft_prompt_length;
    p.output_ids                      = a->output_ids;
    // the parent table of an entry in shared memory where it fits (50000 level-beams), else tile by tile
    size_t       smem   = chain_smem_bytes(a->max_time, a->beam_width);
    const size_t tables = (size_t)a->max_time * a->beam_width * 8;  // tokens and parents as they are
    p.by_maps = a->beam_width <= kTreeBeams && a->max_time <= kTreeLevels * kChainThreads && tables <= kChainMaxSmem;
    smem      = p.by_maps && tables > smem ? tables : smem;
    if (smem <= kChainMaxSmem) {
        static std::atomic<bool> opted_in[kDevicesKnown];
        FTB_CUDA_CHECK(opt_in_smem(gather_tree_chains_kernel, kChainMaxSmem, opted_in));
        FTB_CUDA_CHECK(launch_early(gather_tree_chains_kernel, dim3((unsigned)a->batch_size), dim3(kChainThreads), smem,
                                    (cudaStream_t)a->stream, p));
    }
    else {
        FTB_CUDA_CHECK(launch_early(gather_tree_kernel, dim3((unsigned)a->batch_size), dim3(kDkThreads), 0, (cudaStream_t)a->stream, p));
    }
    FTB_CUDA_CHECK(cudaGetLastError());
    note_launch(1);
    return FTB200_OK;
}

extern "C" int ftb200_finalize(int* output_ids, int* sequence_lengths, float* cum_log_probs, float* output_log_probs,
                               const int* topk_output_ids, const int* topk_sequence_lengths, const float* scores,
                               const float* topk_cum_log_probs, const float* topk_log_probs, const int* num_beams,
                               int beam_width, int max_seq_len, int batch_size, void* stream)
{
    if (output_ids == nullptr || sequence_lengths == nullptr || topk_output_ids == nullptr
        || topk_sequence_lengths == nullptr || scores == nullptr || num_beams == nullptr || beam_width <= 0
        || batch_size <= 0 || max_seq_len < 0 || (cum_log_probs != nullptr && topk_cum_log_probs == nullptr)
        || (output_log_probs != nullptr && topk_log_probs == nullptr)) {
        set_error("ftb200_finalize: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if ((beam_width * 2 + 31) / 32 * 32 >= 1024) {  // FT_CHECK(block.x < 1024), decoding_kernels.cu:789
        set_error("ftb200_finalize: 2 * beam_width rounded up to a warp must stay below 1024");
        return FTB200_UNSUPPORTED;
    }
    // a CTA per beam (each ranks the entry's few scores for itself): the copies of an entry's beams run side by side
    FTB_CUDA_CHECK(launch_early(finalize_kernel, dim3(batch_size, beam_width < 64 ? beam_width : 64), dim3(kDkThreads), 0,
                                (cudaStream_t)stream, output_ids, sequence_lengths, cum_log_probs, output_log_probs, topk_output_ids,
                                topk_sequence_lengths, scores, topk_cum_log_probs, topk_log_probs, num_beams, beam_width, max_seq_len));
    FTB_CUDA_CHECK(cudaGetLastError());
    note_launch(1);
    return FTB200_OK;
}

extern "C" int ftb200_insert_unfinished_path(const ftb200_beam_hyps* hyps, const int* output_ids_src,
                                             const int* parent_ids_src, const int* sequence_lengths_src,
                                             const float* log_probs_src, int max_seq_len, float length_penalty,
                                             const uint8_t* finished, const float* cum_log_probs, int batch_size,
                                             int beam_width, void* stream)
{
    if (hyps == nullptr || hyps->output_ids_tgt == nullptr || hyps->sequence_lengths_tgt == nullptr
        || hyps->cum_log_probs == nullptr || hyps->normed_scores == nullptr || hyps->num_beams == nullptr
        || hyps->is_done == nullptr || output_ids_src == nullptr || parent_ids_src == nullptr
        || sequence_lengths_src == nullptr || finished == nullptr || cum_log_probs == nullptr || batch_size <= 0
        || beam_width <= 0 || max_seq_len < 0) {
        set_error("ftb200_insert_unfinished_path: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (beam_width > kMaxArchiveBeams) {
        set_error("ftb200_insert_unfinished_path: beam_width above 512");
        return FTB200_UNSUPPORTED;
    }
    InsertPath p;
    p.output_ids_tgt       = hyps->output_ids_tgt;
    p.sequence_lengths_tgt = hyps->sequence_lengths_tgt;
    p.cum_log_probs_tgt    = hyps->cum_log_probs;
    p.normed_scores        = hyps->normed_scores;
    p.log_probs_tgt        = hyps->log_probs;
    p.num_beams            = hyps->num_beams;
    p.is_done              = hyps->is_done;
    p.output_ids_src       = output_ids_src;
    p.parent_ids_src       = parent_ids_src;
    p.sequence_lengths_src = sequence_lengths_src;
    p.log_probs_src        = log_probs_src;
    p.max_seq_len          = max_seq_len;
    p.length_penalty       = length_penalty;
    p.finished             = finished;
    p.cum_log_probs        = cum_log_probs;
    p.batch_size           = batch_size;
    p.beam_width           = beam_width;
    const size_t smem = chain_smem_bytes(max_seq_len, beam_width);
    if (smem <= kChainMaxSmem) {
        static std::atomic<bool> opted_in[kDevicesKnown];
        FTB_CUDA_CHECK(opt_in_smem(insert_chains_kernel, kChainMaxSmem, opted_in));
        FTB_CUDA_CHECK(launch_early(insert_chains_kernel, dim3((unsigned)batch_size), dim3(kChainThreads), smem, (cudaStream_t)stream, p));
    }
    else {
        FTB_CUDA_CHECK(launch_early(insert_unfinished_path_kernel, dim3((unsigned)batch_size), dim3(kDkThreads), 0,
                                    (cudaStream_t)stream, p));
    }
    FTB_CUDA_CHECK(cudaGetLastError());
    note_launch(1);
    return FTB200_OK;
}
