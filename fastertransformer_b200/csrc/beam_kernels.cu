// Beam search, one step in two launches (sm_100a).
//
// beam_rows_kernel, one CTA per (batch entry, beam): penalties on the fly, one read of the row from HBM that yields the
// online soft-max statistics (max, sum of exponentials), a second one from L1 for the row's best 2K columns.
// beam_merge_kernel, one CTA per batch entry: merges the K x 2K candidates, applies length penalty and diversity,
// archives finished hypotheses, picks the K live continuations, updates lengths / finished / parents and rewrites the
// KV-cache indirection - everything OnlineBeamSearchLayer<T>::forward launches
// (layers/beam_search_layers/BaseBeamSearchLayer.cu:181-289) in five kernels.  The second kernel starts while the first
// drains (programmatic dependent launch).  Two kernels and not one with a last-arrival counter: the merge reads flags
// of other entries as they were before the step, which the first kernel can simply write down.
#include "chains.cuh"
#include "common.cuh"
#include "ftb200.h"

namespace ftb200 {

constexpr int kBeamThreads = 256;
constexpr int kMaxBeam     = 64;
constexpr int kMergeRank   = 512;  // candidates of an entry that are ordered by counting

struct BeamK {
    int dtype, batch_size, local_batch, ite, K, vocab, vocab_padded, step, max_input_len, max_seq_len;
    const void* logits;
    const void* bias;
    const int*  end_ids;
    const int*  input_lengths;
    float       temperature, rep_penalty;
    int         penalty_type, min_length, apply_temp;
    float       diversity, length_penalty;
    int*        output_ids;
    int*        parent_ids;
    uint8_t*    finished;
    int*        seq_len;
    float*      cum_log_probs;
    float*      out_log_probs;
    const int*  src_indir;
    int*        tgt_indir;
    ftb200_beam_hyps hyps;
    int         has_hyps;
    // workspace
    int*   cand_id;   // [local_batch, K, 2K]
    float* cand_val;  // [local_batch, K, 2K]  (already rounded to the logits type)
    uint8_t* snap_finished;  // finished / sequence_length as they were before this step
    int*     snap_seq_len;
    int      flag_words;   // words of the bit map of penalised columns; 0: none in this call
    int      listed;       // 0: a bit per column; else the map is a filter over column numbers modulo its (power of two)
                           // size, and so many ids can stand in the list that decides
    int      chain_levels; // levels of the parent table in shared memory; 0: the chain is followed in global memory
};

template<int DT>
__device__ __forceinline__ float beam_round(float x)
{
    return DT == FTB200_F16 ? __half2float(__float2half_rn(x)) : x;
}

// logits value of column v with bias / temperature / pad mask applied in the logits type
// (kernels/beam_search_penalty_kernels.cu:24-87); bf16 goes the fp32 way on the up-cast value.
template<int DT>
__device__ __forceinline__ float beam_plain(u32 bits)
{
    return DT == FTB200_F16 ? __half2float(__ushort_as_half((unsigned short)bits)) :
                              (DT == FTB200_F32 ? __uint_as_float(bits) : __uint_as_float(bits << 16));
}
template<int DT>
__device__ __forceinline__ float beam_temp(const BeamK& P, u32 bits, int v, float inv, __half inv_h)
{
    if (DT == FTB200_F16) {
        __half h = __ushort_as_half((unsigned short)bits);
        if (P.bias != nullptr && v < P.vocab) {
            h = __hadd(h, ((const __half*)P.bias)[v]);
        }
        const float y = __half2float(__hmul(h, inv_h));
        return v < P.vocab ? y : -65504.0f;
    }
    const float x = beam_plain<DT>(bits);
    float       b = 0.0f;
    if (P.bias != nullptr && v < P.vocab) {
        b = DT == FTB200_F32 ? ((const float*)P.bias)[v] : __bfloat162float(((const __nv_bfloat16*)P.bias)[v]);
    }
    const float y = (x + b) * inv;
    return v < P.vocab ? y : -FLT_MAX;
}

template<int DT>
__device__ __forceinline__ u32 beam_load(const void* row, int v)
{
    return DT == FTB200_F32 ? __ldg((const u32*)row + v) : (u32)__ldg((const unsigned short*)row + v);
}

struct MD {
    float m, d;
};
__device__ __forceinline__ MD md_merge(MD a, MD b)
{
    // kernels/online_softmax_beamsearch_kernels.cu:270-279
    const bool a_bigger = a.m > b.m;
    const MD   hi = a_bigger ? a : b, lo = a_bigger ? b : a;
    MD         r;
    r.d = hi.d + lo.d * __expf(lo.m - hi.m);
    r.m = hi.m;
    return r;
}

// (value desc, column asc) as one ascending u64
__device__ __forceinline__ u64 order_key(float val, u32 col)
{
    return ((u64)(~fkey(val)) << 32) | col;
}

constexpr int kBeamTile    = 4096;  // columns of a tile: sixteen per thread
constexpr int kBeamStages  = 4;     // tiles in the ring
constexpr int kBeamCollect = 2048;  // columns at or above the row's bound that are sorted in shared memory

// Marks the tokens of row bb's ancestry (the ids that the repetition / presence penalty applies to,
// beam_search_penalty_kernels.cu:89-152) in the bit map.  The chain runs through every level's parents: it is cut into
// segments whose maps compose (see chains.cuh), so that a long history costs a few walks of a segment's length.
__host__ __device__ inline int list_words(int listed)
{
    return listed != 0 ? (listed + 4) / 4 * 4 : 0;  // (its length stands in front)
}
static __device__ __noinline__ void mark_ancestry(const BeamK& P, int bb, u32* bits, unsigned char* tables)
{
    const int    tid = threadIdx.x, K = P.K, b = bb / K, V = P.vocab_padded;
    const int    bbsize = P.batch_size * K, top = P.step - 1;
    const int    input_len = P.input_lengths != nullptr ? P.input_lengths[bb] : P.max_input_len;
    const int*   ids = P.output_ids + (size_t)b * K;
    const int*   par = P.parent_ids + (size_t)P.ite * K * P.local_batch + (size_t)b * K;
    u32* const   list = bits + P.flag_words;
    auto         mark = [&](int id) {
        if (id >= 0 && id < V) {
            const int at = P.listed != 0 ? id & (32 * P.flag_words - 1) : id;
            smem_or(&bits[at >> 5], 1u << (at & 31));
            if (P.listed != 0) {
                list[1 + atomicAdd(&list[0], 1u)] = (u32)id;  // (one entry a level at most)
            }
        }
    };
    auto skipped = [&](int level) { return level >= input_len && level < P.max_input_len; };
    if (tid == 0) {
        mark(P.output_ids[(size_t)top * bbsize + (size_t)P.ite * P.local_batch * K + bb]);
    }
    if (P.chain_levels == 0) {
        if (tid == 0) {
            int beam = bb % K;
            for (int i = top - 1; i >= 0; --i) {
                if (!skipped(i)) {
                    beam = par[(size_t)i * bbsize + beam];
                    mark(ids[(size_t)i * bbsize + beam]);
                }
            }
        }
        return;
    }
    const int levels = top, W = K + 1;
    const u32 row = 2u * (u32)W, t_par = (u32)__cvta_generic_to_shared(tables), t_sel = t_par + (u32)levels * row;
    int       segments = kBeamThreads / W;
    segments           = segments < 1 ? 1 : (segments > 32 ? 32 : segments);
    const int seglen   = (levels + segments - 1) / segments;
    const u32 t_comp   = t_sel + 2u * (u32)levels;
    __shared__ u32 s_entry[32];
    for (int e = tid; e < levels * K; e += kBeamThreads) {
        const int level = e / K, k = e - level * K;
        int       v = skipped(level) ? k : __ldg(par + (size_t)level * bbsize + k);  // a skipped level passes the chain on
        v           = v < 0 || v >= K ? k : v;
        sts_u16(t_par + (u32)level * row + 2u * (u32)k, 2u * (u32)v);
    }
    __syncthreads();
    for (int e = tid; e < segments * K; e += kBeamThreads) {
        const int seg = e / K, lo = min(seg * seglen, levels), hi = min(lo + seglen, levels);
        u32       cur = 2u * (u32)(e % K), at = t_par + (u32)hi * row;
        for (int i = lo; i < hi; ++i) {
            at -= row;
            cur = lds_u16(at + cur);
        }
        sts_u16(t_comp + (u32)seg * row + 2u * (u32)(e % K), cur);
    }
    __syncthreads();
    if (tid == 0) {
        u32 cur = 2u * (u32)(bb % K);
        for (int seg = segments - 1; seg >= 0; --seg) {
            s_entry[seg] = cur;
            cur          = lds_u16(t_comp + (u32)seg * row + cur);
        }
    }
    __syncthreads();
    if (tid < segments) {
        const int lo = min(tid * seglen, levels), hi = min(lo + seglen, levels);
        u32       cur = s_entry[tid], at = t_par + (u32)hi * row;
        for (int i = hi - 1; i >= lo; --i) {
            at -= row;
            cur = lds_u16(at + cur);  // the parent at this level is the beam whose token counts
            sts_u16(t_sel + 2u * (u32)i, cur);
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int level = tid; level < levels; level += kBeamThreads) {
        if (!skipped(level)) {
            mark(__ldg(ids + (size_t)level * bbsize + lds_u16(t_sel + 2u * (u32)level) / 2u));
        }
    }
}

// TEMP: temperature, bias or a padded vocabulary; PEN: penalised columns (1: a bit map of them; 2: of more columns than
// shared memory has bits for, about a million: a filter and a list of the ids).  A branch per column costs as much as the
// column's arithmetic, so the variants are compiled apart.  Bound by latency and issue (24 instructions a column, a
// running maximum and a sum as chains): one row of 32000 half columns 12 us, 256 of them 16 us; with a list search per
// column, sixteen sorted lists and a pass per winner of a wide beam it was 80 us and up.
template<int DT, bool TEMP, int PEN>
__global__ void __launch_bounds__(kBeamThreads, 3) beam_rows_kernel(const __grid_constant__ BeamK P)
{
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // layout: ring of row tiles | u64 collected[kBeamCollect] | u32 bits[flag_words] | u32 list[list_words(listed)] | chain tables
    const u32      ring = (u32)__cvta_generic_to_shared(smem_raw);
    u64*           col  = (u64*)(smem_raw + (size_t)kBeamStages * kBeamTile * (DT == FTB200_F32 ? 4 : 2));
    u32*           bits = (u32*)(col + kBeamCollect);
    __shared__ MD  s_md[kBeamThreads / 32];
    __shared__ __align__(16) u32 s_key[kBeamThreads];
    __shared__ u32 s_n, s_bound;
    FTB_ASSUME_SHARED(col);
    FTB_ASSUME_SHARED(bits);

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int bb  = blockIdx.x;  // local batch-beam row
    const int b = bb / P.K, K = P.K, twoK = 2 * K;
    const int    V   = P.vocab_padded;
    const size_t ES  = DT == FTB200_F32 ? 4 : 2;
    const char*  row = (const char*)P.logits + (size_t)bb * V * ES;
    const float  MAXT = DT == FTB200_F16 ? 65504.0f : FLT_MAX;

    const bool fin    = P.finished[bb] != 0;
    const int  end_id = P.end_ids[b];
    const float cum   = P.cum_log_probs[bb];
    if (tid == 0) {
        P.snap_finished[bb] = fin ? 1 : 0;
        P.snap_seq_len[bb]  = P.seq_len[bb];
        s_n                 = 0;
    }
    int*   my_id  = P.cand_id + (size_t)bb * twoK;
    float* my_val = P.cand_val + (size_t)bb * twoK;
    if (fin) {
        // every column but the end token is -MAX: the end token first, then the smallest columns (:410-432)
        const bool  has   = end_id >= 0 && end_id < V;
        const float m     = has ? MAXT : -MAXT;
        const float log_d = logf(has ? 1.0f : (float)V);
        for (int n = tid; n < twoK; n += kBeamThreads) {
            const int   v = has ? (n == 0 ? end_id : (n - 1 < end_id ? n - 1 : n)) : n;
            const float u = has && n == 0 ? MAXT : -MAXT;
            my_id[n]      = v < V ? bb * V + v : -1;
            my_val[n]     = beam_round<DT>(u - m - log_d + cum);
        }
        return;
    }

    // ---- columns with a value of their own: repetition / presence penalty along the beam's ancestry, min-length mask
    if (PEN) {
        for (int i = tid; i < P.flag_words + (PEN == 2 ? 1 : 0); i += kBeamThreads) {
            bits[i] = 0;  // (and the length of the list)
        }
        __syncthreads();
        mark_ancestry(P, bb, bits, (unsigned char*)(bits + P.flag_words + list_words(P.listed)));
        __syncthreads();
    }
    // rare: a column whose bit of the filter is set
    auto in_list = [&](int v) {
        const u32* list = bits + P.flag_words;
        const int  n    = (int)list[0];
        bool       hit  = false;
        for (int i = 1; i <= n && !hit; ++i) {
            hit = list[i] == (u32)v;
        }
        return hit;
    };
    const bool   minlen = (P.step - P.max_input_len < P.min_length) && (P.seq_len[bb] + 1 - P.max_input_len < P.min_length);
    const int    masked = minlen ? end_id : -1;
    const float  pen    = beam_round<DT>(P.rep_penalty);
    const float  inv    = 1.0f / (P.temperature + 1e-6f);
    const __half inv_h  = __float2half_rn(inv);
    // value of column v as the reference's stage-1 kernel sees it (:410-432)
    auto value_of = [&](int v, u32 raw) -> float {
        float y = TEMP ? beam_temp<DT>(P, raw, v, inv, inv_h) : beam_plain<DT>(raw);
        if (PEN) {
            // one word for the 32 columns of a warp
            const u32 w = bits[PEN == 2 ? (v >> 5) & (P.flag_words - 1) : v >> 5];
            if (((w >> (v & 31)) & 1u) && (PEN != 2 || in_list(v))) {
                if (P.penalty_type == FTB200_PENALTY_ADDITIVE) {
                    y = beam_round<DT>(y - pen);
                }
                else {
                    y = beam_round<DT>(y > 0.0f ? y / pen : y * pen);
                }
            }
        }
        return v == masked ? -MAXT : y;
    };

    // ---- one pass: soft-max statistics and the candidates ----
    // Thread t takes columns t, t + 256, ... one after the other (an online maximum and sum; the order is kept, so that
    // scores rounded to half do not depend on the launch); only the maximum and the sum themselves are chains.  The
    // threads' maxima over the first tile give a bound that every one of the row's best 2K reaches: later columns at or above it are kept, a few times 2K V / 4096.
    constexpr int U = 16;
    MD            md{-MAXT, 0.0f};
    float         bound = -INFINITY;
    auto          add = [&](float y) {
        // md_merge(md, {y, 1}) in fewer instructions: |difference| serves both orders
        const float t = md.m - y, e = __expf(-fabsf(t));
        const bool  keep = t > 0.0f;
        md.d             = fmaf(md.d, keep ? 1.0f : e, keep ? e : 1.0f);
        md.m             = fmaxf(md.m, y);
    };
    auto push = [&](int v, float y) {
        const u32 at = atomicAdd(&s_n, 1u);
        if (at < (u32)kBeamCollect) {
            col[at] = order_key(y, (u32)v);
        }
    };
    // The 2K-th largest of the threads' maxima: a value that at least 2K columns seen so far reach (CTA-wide).  Narrow
    // beams: every warp takes out its 2K largest, warp 0 goes through those; wide ones: every thread counts.
    auto thread_bound = [&]() {
        u32 mine = fkey(md.m);
        if (twoK <= 16) {
            for (int r = 0; r < twoK; ++r) {
                const u32 top     = __reduce_max_sync(0xffffffffu, mine);
                const u32 holders = __ballot_sync(0xffffffffu, mine == top);
                mine              = lane == __ffs(holders) - 1 ? 0u : mine;
                if (lane == 0) {
                    s_key[wid * twoK + r] = top;
                }
            }
            __syncthreads();
            if (wid == 0) {
                u32 k[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int at = i * 32 + lane;
                    k[i]         = at < twoK * (kBeamThreads / 32) ? s_key[at] : 0u;
                }
                u32 top = 0;
                for (int r = 0; r < twoK; ++r) {
                    const u32 best = max(max(k[0], k[1]), max(k[2], k[3]));
                    top            = __reduce_max_sync(0xffffffffu, best);
                    const u32 holders = __ballot_sync(0xffffffffu, best == top);
                    if (lane == __ffs(holders) - 1) {
                        bool gone = false;  // one of them, once
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const bool hit = (k[i] == top) & !gone;
                            gone |= hit;
                            k[i] = hit ? 0u : k[i];
                        }
                    }
                }
                if (lane == 0) {
                    s_bound = top;
                }
            }
        }
        else {
            s_key[tid] = mine;
            __syncthreads();
            int rk = 0;
#pragma unroll 8
            for (int i = 0; i < kBeamThreads; i += 4) {
                // larger, or equal and of an earlier thread (short-circuit forms of this compile to branches: 12 us, not 2)
                const uint4 o = *(const uint4*)(s_key + i);
                rk += o.x >= mine + (i + 0 >= tid ? 1u : 0u) ? 1 : 0;
                rk += o.y >= mine + (i + 1 >= tid ? 1u : 0u) ? 1 : 0;
                rk += o.z >= mine + (i + 2 >= tid ? 1u : 0u) ? 1 : 0;
                rk += o.w >= mine + (i + 3 >= tid ? 1u : 0u) ? 1 : 0;
            }
            if (rk == twoK - 1) {
                s_bound = mine;
            }
        }
        __syncthreads();
        return fkey_inv(s_bound);
    };
    // The row comes through a ring of tiles in shared memory, three tiles ahead (16-byte asynchronous copies; the few
    // columns before the first and after the last 16-byte boundary go through registers).
    const int sh   = (int)(((size_t)row & 15) / ES);  // the row's first column inside its 16 bytes
    auto      fill = [&](int k) {
        constexpr int EPC = 16 / (DT == FTB200_F32 ? 4 : 2);
        for (int c = tid; c < kBeamTile / EPC; c += kBeamThreads) {
            const int v    = k * kBeamTile + c * EPC - sh;
            const u32 slot = ring + (u32)((k % kBeamStages) * kBeamTile + c * EPC) * (u32)ES;
            if (v >= 0 && v + EPC <= V) {
                cp_async16(slot, row + (ptrdiff_t)v * (ptrdiff_t)ES);
            }
            else {
#pragma unroll
                for (int e = 0; e < EPC; ++e) {
                    if (v + e >= 0 && v + e < V) {
                        if (DT == FTB200_F32) {
                            sts_u32(slot + 4u * (u32)e, beam_load<DT>(row, v + e));
                        }
                        else {
                            sts_u16(slot + 2u * (u32)e, beam_load<DT>(row, v + e));
                        }
                    }
                }
            }
        }
    };
    constexpr u32 kRing = kBeamStages * kBeamTile;
    auto staged = [&](u32 at) { return DT == FTB200_F32 ? lds_u32(at) : lds_u16(at); };
    // (no branch per column: a mask of the sixteen, and the rare column that is kept is read again)
    auto keep_above = [&](const float* y, int v0, auto&& again) {
        u32 hits = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            hits |= (y[u] >= bound ? 1u : 0u) << u;
        }
        while (hits != 0) {
            const int v = v0 + (__ffs(hits) - 1) * kBeamThreads;
            hits &= hits - 1;
            push(v, value_of(v, again(v)));
        }
    };
    float     y[U];
    const int v_whole = V / kBeamTile * kBeamTile, tiles = (V + sh + kBeamTile - 1) / kBeamTile;
    for (int k = 0; k < kBeamStages - 1; ++k) {
        if (k < tiles) {
            fill(k);
        }
        cp_async_commit();
    }
    for (int k = 0; k * kBeamTile < V; ++k) {
        cp_async_wait<kBeamStages - 3>();  // tile k + 1 has arrived too: a row that starts off a 16-byte boundary reaches into it
        __syncthreads();                   // for every thread; and tile k - 1 has been used up
        if (k + kBeamStages - 1 < tiles) {
            fill(k + kBeamStages - 1);
        }
        cp_async_commit();
        const int v0 = k * kBeamTile + tid;
        const u32 at = (u32)(v0 + sh) % kRing;
        if (v0 - tid < v_whole) {
            u32 raw[U];
            if (sh == 0) {
                const u32 a0 = ring + at * (u32)ES;  // the tile does not wrap: one address for all sixteen
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    raw[u] = staged(a0 + (u32)(u * kBeamThreads) * (u32)ES);
                }
            }
            else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    raw[u] = staged(ring + (at + (u32)(u * kBeamThreads)) % kRing * (u32)ES);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                y[u] = value_of(v0 + u * kBeamThreads, raw[u]);
                add(y[u]);
            }
        }
        else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int v = v0 + u * kBeamThreads;
                y[u]        = __int_as_float(0x7fc00000);  // not a number: below every bound
                if (v < V) {
                    y[u] = value_of(v, staged(ring + (at + (u32)(u * kBeamThreads)) % kRing * (u32)ES));
                    add(y[u]);
                }
            }
        }
        if (k == 0) {
            bound = thread_bound();
        }
        keep_above(y, v0, [&](int v) { return staged(ring + (u32)(v + sh) % kRing * (u32)ES); });
    }
    bound = thread_bound();  // (also a barrier: everything has been collected)
    for (int off = 16; off > 0; off >>= 1) {
        MD o;
        o.m = __shfl_down_sync(0xffffffffu, md.m, off);
        o.d = __shfl_down_sync(0xffffffffu, md.d, off);
        md  = md_merge(md, o);
    }
    if (lane == 0) {
        s_md[wid] = md;
    }
    const int n_all = (int)s_n;
    __syncthreads();
    md = s_md[0];
    for (int i = 1; i < kBeamThreads / 32; ++i) {
        md = md_merge(md, s_md[i]);
    }
    const float log_d = logf(md.d);
    auto        score = [&](u64 e) { return beam_round<DT>(fkey_inv(~(u32)(e >> 32)) - md.m - log_d + cum); };
    // the bound of the whole row leaves a few more than 2K of them
    if (tid == 0) {
        s_n = 0;
    }
    __syncthreads();
    u64 kept[kBeamCollect / kBeamThreads];
    if (n_all <= kBeamCollect) {
#pragma unroll
        for (int i = 0; i < kBeamCollect / kBeamThreads; ++i) {
            const int at = i * kBeamThreads + tid;
            kept[i]      = at < n_all ? col[at] : ~0ull;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kBeamCollect / kBeamThreads; ++i) {
            if ((kept[i] != ~0ull) & ((u32)(~(u32)(kept[i] >> 32)) >= s_bound)) {
                col[atomicAdd(&s_n, 1u)] = kept[i];
            }
        }
    }
    else {
        // a wide beam over a long row: the columns at or above the final bound, in a second pass
        for (int v0 = tid; v0 < V; v0 += kBeamThreads * U) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int v = v0 + u * kBeamThreads;
                y[u]        = v < V ? value_of(v, beam_load<DT>(row, v)) : __int_as_float(0x7fc00000);
            }
            keep_above(y, v0, [&](int v) { return beam_load<DT>(row, v); });
        }
    }
    __syncthreads();
    const int n = (int)s_n;
    if (n <= kBeamCollect && n >= (twoK < V ? twoK : V)) {
        for (int i = tid; i < n; i += kBeamThreads) {
            const u64 e  = col[i];
            int       rk = 0;
#pragma unroll 4
            for (int j = 0; j < n; ++j) {
                rk += col[j] < e ? 1 : 0;
            }
            if (rk < twoK) {
                my_id[rk]  = bb * V + (int)(e & 0xffffffffu);
                my_val[rk] = score(e);
            }
        }
        for (int i = n + tid; i < twoK; i += kBeamThreads) {
            my_id[i]  = -1;
            my_val[i] = score(~0ull);
        }
        return;
    }
    // thousands of equal values at the bound, or columns that are not above -MAX: the winners one by one, each in a pass
    // over the row
    __syncthreads();
    __shared__ u64 s_prev;
    if (tid == 0) {
        s_prev = 0;
    }
    __syncthreads();
    for (int w = 0; w < twoK; ++w) {
        const u64 prev = s_prev;
        u64       mine = ~0ull;
        for (int v = tid; v < V; v += kBeamThreads) {
            const u64 kk = order_key(value_of(v, beam_load<DT>(row, v)), (u32)v);
            if ((w == 0 || kk > prev) && kk < mine) {
                mine = kk;
            }
        }
        col[tid] = mine;
        __syncthreads();
        for (int s = kBeamThreads / 2; s > 0; s >>= 1) {
            if (tid < s && col[tid + s] < col[tid]) {
                col[tid] = col[tid + s];
            }
            __syncthreads();
        }
        if (tid == 0) {
            const u64 e = col[0];
            s_prev      = e;
            my_id[w]    = e == ~0ull ? -1 : bb * V + (int)(e & 0xffffffffu);
            my_val[w]   = score(e);
        }
        __syncthreads();
    }
}

template<int DT>
__global__ void __launch_bounds__(kBeamThreads) beam_merge_kernel(const __grid_constant__ BeamK P)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64*             sortbuf = (u64*)smem_raw;  // [2 * ncand] below kMergeRank candidates, else [ncand]
    constexpr int    kTop    = 128;
    __shared__ float s_old_cum[kMaxBeam], s_y[kTop];
    __shared__ int   s_newseq[kMaxBeam], s_word[kTop];
    const int        tid = threadIdx.x, b = blockIdx.x, K = P.K, twoK = 2 * K, V = P.vocab_padded;
    wait_for_previous();  // the rows' kernel has ended and its results are visible

    const int    end_id  = P.end_ids[b];
    const int    ncand   = K * twoK;
    const int*   x       = P.cand_id + (size_t)b * ncand;
    const float* y       = P.cand_val + (size_t)b * ncand;
    const int    gbi     = P.ite * P.local_batch + b;
    int*         z       = P.output_ids + (size_t)P.step * P.batch_size * K + (size_t)P.ite * P.local_batch * K + b * K;
    int*         parents = P.parent_ids + (size_t)P.step * P.batch_size * K + (size_t)P.ite * P.local_batch * K + b * K;
    float*       v_cum   = P.cum_log_probs + b * K;
    float*       olp     = P.out_log_probs == nullptr ?
                               nullptr :
                               P.out_log_probs + (size_t)P.step * P.batch_size * K + (size_t)P.ite * P.local_batch * K;
    if (tid < K) {
        s_old_cum[tid] = v_cum[tid];
    }
    __syncthreads();
    bool skip_select = false;
    if (P.has_hyps) {
        // batch_topk_kernel, kernels/online_softmax_beamsearch_kernels.cu:129-138
        if (P.hyps.num_beams[gbi] == 0 && tid == 0) {
            P.hyps.min_normed_scores[gbi] = FLT_MAX;
        }
        else if (P.hyps.num_beams[gbi] == K) {
            skip_select = true;
        }
    }
    if (!skip_select) {
        // score of a candidate: length penalty with the length of the batch entry's FIRST indices, as the
        // reference indexes finished / sequence_lengths by the batch index (:148-156), plus diversity
        const int  len    = P.snap_finished[b] ? P.snap_seq_len[b] : P.snap_seq_len[b] + 1;
        const bool use_lp = !(P.length_penalty == 0.0f);
        for (int i = tid; i < ncand; i += kBeamThreads) {
            float e = y[i];
            if (use_lp && len != 1) {
                e = beam_round<DT>(e / beam_round<DT>(powf((float)len, P.length_penalty)));
            }
            if (DT == FTB200_F16) {
                // `elem += diversity_rate * (T)i` in half: the compiler contracts the half multiply and add of the
                // reference into one fused multiply-add, so the sum is rounded once (exact in double first)
                const double d = (double)beam_round<DT>(P.diversity) * (double)beam_round<DT>((float)(i % K)) + (double)e;
                e              = __half2float(__double2half(d));
            }
            else {
                e = e + P.diversity * (float)(i % K);
            }
            sortbuf[i] = x[i] < 0 ? ~0ull : order_key(e, (u32)i);
        }
        __syncthreads();
        if (ncand <= kMergeRank) {
            // a few hundred: by counting the smaller ones (missing ones in the order they stand)
            for (int i = tid; i < ncand; i += kBeamThreads) {
                const u64 e  = sortbuf[i];
                int       rk = 0;
#pragma unroll 4
                for (int j = 0; j < ncand; ++j) {
                    rk += (int)(sortbuf[j] < e) | ((int)(sortbuf[j] == e) & (int)(j < i));
                }
                sortbuf[ncand + rk] = e;
            }
            __syncthreads();
            sortbuf += ncand;
        }
        else {
            group_sort_u64(sortbuf, ncand, tid, kBeamThreads, CtaSync());
            __syncthreads();
        }
        const int top_n = ncand < 2 * 4 ? ncand : (twoK <= 8 ? 8 : (twoK <= 16 ? 16 : (twoK <= 32 ? 32 : (twoK <= 64 ? 64 : 128))));
        // what the choice reads, fetched together
        for (int i = tid; i < top_n && i < ncand; i += kBeamThreads) {
            const u64 e = sortbuf[i];
            s_word[i]   = e == ~0ull ? -1 : x[(u32)e];
            s_y[i]      = e == ~0ull ? 0.0f : y[(u32)e];
        }
        __syncthreads();
        if (!P.has_hyps) {
            // no archive: the K best go on
            if (tid < K && tid < top_n && tid < ncand && s_word[tid] >= 0) {
                z[tid] = s_word[tid];
                if (olp != nullptr) {
                    olp[b * K + tid] = s_y[tid] - s_old_cum[(s_word[tid] / V) % K];
                }
                v_cum[tid] = s_y[tid];
            }
        }
        else if (tid == 0) {
            int       selected = 0;
            for (int i = 0; i < top_n && i < ncand; ++i) {
                const u64 e = sortbuf[i];
                if (e == ~0ull) {
                    break;
                }
                const float normed_score = fkey_inv(~(u32)(e >> 32));
                const int   word         = s_word[i];
                if (word % V == end_id) {
                    if (i < K) {
                        const int num_beam = P.hyps.num_beams[gbi];
                        int       beam_idx = num_beam;
                        bool      stop     = false;
                        if (num_beam == K) {
                            if (normed_score < P.hyps.min_normed_scores[gbi]) {
                                selected = K;
                                stop     = true;
                            }
                            else {
                                for (int j = 0; j < K; j++) {
                                    if (P.hyps.normed_scores[gbi * twoK + j] == P.hyps.min_normed_scores[gbi]) {
                                        beam_idx = j;
                                        P.hyps.num_beams[gbi]--;
                                        P.hyps.min_normed_scores[gbi]       = FLT_MAX;
                                        P.hyps.normed_scores[gbi * twoK + j] = normed_score;
                                        for (int l = 0; l < K; l++) {
                                            P.hyps.min_normed_scores[gbi] =
                                                fminf(P.hyps.min_normed_scores[gbi], P.hyps.normed_scores[gbi * twoK + l]);
                                        }
                                        break;
                                    }
                                }
                            }
                        }
                        if (stop) {
                            break;
                        }
                        const size_t tgt = ((size_t)gbi * twoK + beam_idx) * P.max_seq_len;
                        P.hyps.output_ids_tgt[tgt + P.step] = end_id;
                        if (P.hyps.log_probs != nullptr) {
                            P.hyps.log_probs[tgt + P.step] = s_y[i] - s_old_cum[(word / V) % K];
                        }
                        int prev_id = (word / V) % K;
                        for (int j = P.step - 1; j >= 0; j--) {
                            const size_t src = (size_t)j * P.batch_size * K + (size_t)P.ite * P.local_batch * K + b * K + prev_id;
                            P.hyps.output_ids_tgt[tgt + j] = P.output_ids[src];
                            if (P.hyps.log_probs != nullptr && P.out_log_probs != nullptr) {
                                P.hyps.log_probs[tgt + j] = P.out_log_probs[src];
                            }
                            prev_id = P.parent_ids[src];
                        }
                        const int tb                      = gbi * twoK + beam_idx;
                        P.hyps.sequence_lengths_tgt[tb]   = P.step;
                        P.hyps.normed_scores[tb]          = normed_score;
                        P.hyps.min_normed_scores[gbi]     = fminf(P.hyps.min_normed_scores[gbi], normed_score);
                        P.hyps.num_beams[gbi]++;
                        P.hyps.cum_log_probs[tb]          = s_y[i];
                    }
                }
                else if (i < twoK) {
                    z[selected] = word;
                    if (olp != nullptr) {
                        olp[b * K + selected] = s_y[i] - s_old_cum[(word / V) % K];
                    }
                    v_cum[selected] = s_y[i];
                    selected++;
                }
                if (selected >= K) {
                    break;
                }
            }
            // the reference indexes by the local batch index here (:254-261)
            if (P.hyps.num_beams[b] < K) {
                P.hyps.is_done[b] = 0;
            }
            else if (P.hyps.early_stopping) {
                P.hyps.is_done[b] = 1;
            }
        }
        __syncthreads();
    }

    // ---- update_kernel (layers/beam_search_layers/OnlineBeamSearchLayer.cu:24-58): lengths follow the parent
    if (tid < K) {
        const int idx = b * K + tid;
        s_newseq[tid] = P.finished[idx] ? P.seq_len[idx] : P.seq_len[idx] + 1;
    }
    __syncthreads();
    if (tid < K) {
        const int idx     = b * K + tid;
        const int word    = z[tid];
        const int beam_id = (word / V) % K;
        const int word_id = word % V;
        P.seq_len[idx]    = s_newseq[beam_id];
        P.finished[idx]   = word_id == end_id ? 1 : 0;
        parents[tid]      = beam_id;
        z[tid]            = word_id;
    }
    __syncthreads();
    if (P.has_hyps && P.hyps.num_beams[gbi] == K && tid < K) {
        P.finished[b * K + tid] = 1;
    }
    __syncthreads();

    // ---- KV-cache indirection (layers/beam_search_layers/BaseBeamSearchLayer.cu:23-79)
    if (P.tgt_indir != nullptr && P.src_indir != nullptr) {
        const int L          = P.max_seq_len;
        const int start_step = P.step + 1 - L > 0 ? P.step + 1 - L : 0;
        const int num_steps  = P.step + 1 < L ? P.step + 1 : L;
        for (int i = tid; i < K * num_steps; i += kBeamThreads) {
            const int k = i / num_steps, t = i % num_steps + start_step;
            if (P.finished[b * K + k]) {
                continue;
            }
            const int    tc       = t % L;
            const int    src_beam = parents[k];
            const size_t base     = (size_t)b * K * L;
            P.tgt_indir[base + (size_t)k * L + tc] = t == P.step ? k : P.src_indir[base + (size_t)src_beam * L + tc];
        }
    }
}

constexpr size_t kBeamMaxSmem = 200 * 1024;

template<int DT, bool TEMP, int PEN>
static int beam_rows_launch(const BeamK& K, size_t smem, cudaStream_t st)
{
    static std::atomic<bool> opted[kDevicesKnown];
    FTB_CUDA_CHECK(opt_in_smem(beam_rows_kernel<DT, TEMP, PEN>, kBeamMaxSmem, opted));
    FTB_CUDA_CHECK(launch_early(beam_rows_kernel<DT, TEMP, PEN>, dim3((unsigned)(K.local_batch * K.K)), dim3(kBeamThreads), smem, st, K));
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

template<int DT>
static int beam_launch(const BeamK& K, size_t smem, cudaStream_t st)
{
    static std::atomic<bool> merge_opted[kDevicesKnown];
    FTB_CUDA_CHECK(opt_in_smem(beam_merge_kernel<DT>, kBeamMaxSmem, merge_opted));
    const int pen = K.flag_words == 0 ? 0 : (K.listed == 0 ? 1 : 2);
    int       rc;
    if (K.apply_temp) {
        rc = pen == 0 ? beam_rows_launch<DT, true, 0>(K, smem, st) :
                        (pen == 1 ? beam_rows_launch<DT, true, 1>(K, smem, st) : beam_rows_launch<DT, true, 2>(K, smem, st));
    }
    else {
        rc = pen == 0 ? beam_rows_launch<DT, false, 0>(K, smem, st) :
                        (pen == 1 ? beam_rows_launch<DT, false, 1>(K, smem, st) : beam_rows_launch<DT, false, 2>(K, smem, st));
    }
    if (rc != FTB200_OK) {
        return rc;
    }
    const int             ncand = K.K * 2 * K.K;
    cudaLaunchConfig_t    cfg{};
    cudaLaunchAttribute   attr[1];
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim          = dim3((unsigned)K.local_batch);
    cfg.blockDim         = dim3(kBeamThreads);
    cfg.dynamicSmemBytes = (size_t)ncand * (ncand <= kMergeRank ? 16 : 8);
    cfg.stream           = st;
    cfg.attrs            = attr;
    cfg.numAttrs         = 1;
    FTB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, beam_merge_kernel<DT>, K));
    note_launch(2);
    return FTB200_OK;
}

}  // namespace ftb200

using namespace ftb200;

extern "C" int ftb200_beam_workspace_bytes(int local_batch_size, int beam_width, size_t* bytes)
{
    if (bytes == nullptr || local_batch_size < 0 || beam_width < 1 || beam_width > kMaxBeam) {
        set_error("ftb200_beam_workspace_bytes: invalid argument (beam_width must be 1..64)");
        return FTB200_INVALID_ARG;
    }
    const size_t rows = (size_t)local_batch_size * beam_width;
    *bytes            = 256 + (((size_t)local_batch_size * 4 + 255) / 256) * 256 + rows * 2 * beam_width * 8
             + ((rows + 255) / 256) * 256 + rows * 4;
    return FTB200_OK;
}

extern "C" int ftb200_beam_search_step(const ftb200_beam_params* p)
{
    reset_launch_count();
    if (p == nullptr || p->logits == nullptr || p->end_ids == nullptr || p->output_ids == nullptr
        || p->parent_ids == nullptr || p->finished == nullptr || p->sequence_length == nullptr
        || p->cum_log_probs == nullptr) {
        set_error("ftb200_beam_search_step: a required pointer is null (cum_log_probs is required in beam search)");
        return FTB200_INVALID_ARG;
    }
    if (p->beam_width < 2 || p->beam_width > kMaxBeam) {
        set_error("Topk kernel of beam search does not support beam_width=" + std::to_string(p->beam_width));
        return FTB200_DOMAIN_ERROR;
    }
    if (p->dtype < 0 || p->dtype > 2 || p->local_batch_size < 0 || p->vocab_size <= 0
        || p->vocab_size_padded < p->vocab_size || p->step < 0 || p->max_seq_len <= p->step) {
        set_error("ftb200_beam_search_step: bad shape or dtype");
        return FTB200_INVALID_ARG;
    }
    if (p->local_batch_size == 0) {
        return FTB200_OK;
    }
    size_t need = 0;
    ftb200_beam_workspace_bytes(p->local_batch_size, p->beam_width, &need);
    if (p->workspace == nullptr || p->workspace_bytes < need) {
        set_error("ftb200_beam_search_step: workspace too small, need " + std::to_string(need) + " bytes");
        return FTB200_WORKSPACE_SMALL;
    }
    BeamK K{};
    K.dtype = p->dtype, K.batch_size = p->batch_size, K.local_batch = p->local_batch_size, K.ite = p->ite;
    K.K = p->beam_width, K.vocab = p->vocab_size, K.vocab_padded = p->vocab_size_padded, K.step = p->step;
    K.max_input_len = p->max_input_length, K.max_seq_len = p->max_seq_len;
    K.logits = p->logits, K.bias = p->embedding_bias, K.end_ids = p->end_ids, K.input_lengths = p->input_lengths;
    K.temperature = p->temperature, K.rep_penalty = p->repetition_penalty, K.penalty_type = p->penalty_type;
    K.min_length = p->min_length, K.diversity = p->diversity_rate, K.length_penalty = p->length_penalty;
    // invokeAddBiasApplyPenalties gate, kernels/beam_search_penalty_kernels.cu:197
    K.apply_temp = (p->embedding_bias != nullptr || p->temperature != 1.0f || p->vocab_size != p->vocab_size_padded) ? 1 : 0;
    K.output_ids = p->output_ids, K.parent_ids = p->parent_ids, K.finished = p->finished;
    K.seq_len = p->sequence_length, K.cum_log_probs = p->cum_log_probs, K.out_log_probs = p->output_log_probs;
    K.src_indir = p->src_cache_indirection, K.tgt_indir = p->tgt_cache_indirection;
    K.has_hyps = (p->beam_hyps != nullptr && p->beam_hyps->num_beams != nullptr) ? 1 : 0;
    if (p->beam_hyps != nullptr) {
        K.hyps = *p->beam_hyps;
    }
    // (the first 256 + 4 * local_batch_size bytes of the workspace are not used any more)
    char*        ws   = (char*)p->workspace;
    const size_t rows = (size_t)p->local_batch_size * p->beam_width;
    K.cand_id         = (int*)(ws + (((size_t)p->local_batch_size * 4 + 255) / 256) * 256 + 256);
    K.cand_val        = (float*)(K.cand_id + rows * 2 * p->beam_width);
    K.snap_finished   = (uint8_t*)(K.cand_val + rows * 2 * p->beam_width);
    K.snap_seq_len    = (int*)(K.snap_finished + ((rows + 255) / 256) * 256);

    const bool penalise = p->penalty_type != FTB200_PENALTY_NONE && p->step > 0
                          && p->repetition_penalty != (p->penalty_type == FTB200_PENALTY_MULTIPLICATIVE ? 1.0f : 0.0f);
    const size_t base   = (size_t)kBeamStages * kBeamTile * (p->dtype == FTB200_F32 ? 4 : 2) + (size_t)kBeamCollect * 8;
    K.flag_words        = penalise ? ((p->vocab_size_padded + 31) / 32 + 3) / 4 * 4 : 0;
    K.listed            = 0;
    if (base + (size_t)K.flag_words * 4 > kBeamMaxSmem) {
        // more columns than there is room for bits: the ids of the ancestry in a list, and as large a filter as that leaves
        K.listed     = p->step;
        K.flag_words = 16384;
        while (K.flag_words > 4096 && base + (size_t)(K.flag_words + list_words(K.listed)) * 4 > kBeamMaxSmem) {
            K.flag_words /= 2;
        }
    }
    size_t smem = base + (size_t)(K.flag_words + list_words(K.listed)) * 4;
    if (smem > kBeamMaxSmem) {
        set_error("ftb200_beam_search_step: step too large for the list of penalised columns");
        return FTB200_UNSUPPORTED;
    }
    // the parents of all levels in shared memory where they fit
    K.chain_levels = 0;
    if (penalise && p->step > 1) {
        const size_t table = (size_t)(p->step - 1) * (p->beam_width + 2) * 2 + 32 * (size_t)(p->beam_width + 1) * 2 + 16;
        if (smem + table <= kBeamMaxSmem) {
            K.chain_levels = p->step - 1;
            smem += table;
        }
    }
    switch (p->dtype) {
        case FTB200_F32: return beam_launch<FTB200_F32>(K, smem, (cudaStream_t)p->stream);
        case FTB200_F16: return beam_launch<FTB200_F16>(K, smem, (cudaStream_t)p->stream);
        default: return beam_launch<FTB200_BF16>(K, smem, (cudaStream_t)p->stream);
    }
}
