// Local pass of the vocabulary-parallel step for 16-bit logits: the exchange records of all shards a device holds, in
// one launch.
//
// A CTA takes one row of one shard at a time.  The row (up to 200 KB) goes into shared memory by bulk copies that one
// thread issues, and the next row is on its way as soon as the candidates of this one have been collected.  With the row
// at hand no sample and no estimate is needed:
//   1. every thread keeps the largest value of each of eight groups of its columns.  The k-th largest of all those maxima
//      (one per thread while k is small, the finer groups above that) is a threshold that at least k columns reach, and
//      hardly more: 74 of 32000 for k = 64, 300 for k = 256;
//   2. the columns at or above it are collected from the groups that reach it, and placed by counting how many of them
//      come before each (a few hundred broadcast reads, no sorting network and none of its barriers);
//   3. columns that a penalty or a ban touches are taken out of the copy first (an atomic OR makes them NaN, which no
//      comparison lets through, and returns the raw value to exactly one thread) and are collected with their final values.
// A row whose candidates do not fit (thousands of equal values), with fewer than k values to choose from, or with a
// temperature that turns the order round, gets its threshold by bisection over the final values, counting in the copy:
// rare, and still this kernel.
//
// Bound by the latency of the steps behind the copy: 5.9 us a row (copy and maxima 1.7, threshold 0.9, candidates 1.6,
// placing and record 1.4) with three CTAs on an SM, which is 4.0 TB/s.  2048 rows of 8 x 32000 bf16, k = 64: 265 us; 8 x 100
// with a sample, a streaming pass and a sorting network in a launch per shard; 370 with 16-byte asynchronous copies by
// all threads (a thread's 16 copies take 2 us to issue).
#pragma once
#include "fast_sampling.cuh"
#include "vp_args.cuh"

namespace ftb200 {

// ---- bulk copies and the barriers that count their bytes ----
__device__ __forceinline__ void bar_init(u32 bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// `bytes` (a multiple of 16, or none) from global to shared memory; both on 16-byte boundaries
__device__ __forceinline__ void bulk_copy(u32 dst, const void* src, u32 bytes, u32 bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    if (bytes != 0) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                     "l"(src), "r"(bytes), "r"(bar)
                     : "memory");
    }
}
// false when the copy did not come in (a limit on the wait, nothing else ends it)
__device__ __forceinline__ bool bar_wait(u32 bar, u32 parity)
{
    u32 done = 0;
    for (int i = 0; i < (1 << 20) && done == 0; ++i) {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
    }
    return done != 0;
}

template<int DT, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 4 : 1)
vp_select_kernel(const __grid_constant__ KParams P, const __grid_constant__ VpArgs V)
{
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned short s_max[NT], s_hot[NT * 4];
    __shared__ u32            s_n, s_nspec, s_nhot, s_thr, s_kv, s_m, s_cnt[3], s_lost, s_args[5];
    __shared__ u64            s_bar[4];
    constexpr u32             kDead2 = DT == FTB200_F16 ? 0xfc00fc00u : 0xff80ff80u;  // two columns of -infinity
    uint4* const              row    = (uint4*)smem_raw;
    u64* const                cand   = (u64*)(smem_raw + V.row_bytes);
    u64* const                spec   = cand + V.cand_cap;
    const int                 tid = threadIdx.x, lane = tid & 31;
    const int                 rows = P.local_batch, tasks = rows * V.n_shards;
    const bool                temp = P.apply_temp != 0;
    const float               neg_max = DT == FTB200_F16 ? -65504.0f : -FLT_MAX;
    const bool special_launch = P.apply_rep || P.bad_words != nullptr || P.apply_minlen;

    struct Task {
        const char* base;  // the row's first byte, rounded down to a vector
        int         r, sh, mis, nv, vocab, k;
        float       inv_t;
        bool        live, topp;
    };
    // A row's arguments are sent for (asynchronous copies of the words that hold them, by one thread) at the start of the
    // row before it, and looked at when that one has been collected.
    enum { kSkipK, kSkipP, kFin, kK, kTemp };
    auto send_args = [&](int t) {
        if (tid == 32 && t < tasks) {
            const int r    = t % rows;
            const u32 args = (u32)__cvta_generic_to_shared(s_args);
            auto      word = [&](int slot, const void* p) { cp_async4(args + 4u * (u32)slot, p); };
            auto      byte = [&](int slot, const uint8_t* p) {
                if (p == nullptr) {
                    return;
                }
                // (asynchronous whatever the alignment: a load that is waited for here cost rows of 12000 columns 4 %)
                const WordSpan W = word_span((size_t)p, rows, r);
                if (W.bytes != 0) {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(args + 4u * (u32)slot), "l"(p + W.from),
                                 "r"(W.bytes)
                                 : "memory");
                }
                else {
                    sts_u32(args + 4u * (u32)slot, (u32)p[r] << (8 * (r - W.from)));
                }
            };
            byte(kSkipK, P.topk_skip);
            byte(kSkipP, P.topp_skip);
            byte(kFin, P.finished);
            word(kK, P.topk_ks + r);
            if (temp) {
                word(kTemp, P.temperature + r);
            }
            cp_async_commit();
        }
    };
    auto args_here = [&]() {  // before the barrier that publishes them
        if (tid == 32) {
            cp_async_wait_all();
        }
    };
    auto task_of = [&](int t) {
        Task T;
        auto byte_of = [&](int slot, const uint8_t* p, u32 none) {
            return p != nullptr ? (s_args[slot] >> (8 * ((size_t)(p + T.r) & 3))) & 0xffu : none;
        };
        T.sh            = t < tasks ? t / rows : 0;
        T.r             = t - T.sh * rows;
        const u32 skip_k = byte_of(kSkipK, P.topk_skip, 0u), fin = byte_of(kFin, P.finished, 0u);
        const u32 skip_p = P.topp_states == nullptr ? 1u : byte_of(kSkipP, P.topp_skip, 0u);
        T.live           = (t < tasks) & ((skip_k | fin) == 0);
        T.topp           = (t < tasks) & (skip_k != 0) & ((fin | skip_p) == 0);
        const int k      = (int)s_args[kK];
        T.k              = k < 1 ? 1 : (k > kMaxTopK ? kMaxTopK : k);
        T.inv_t          = temp ? 1.0f / (__uint_as_float(s_args[kTemp]) + 1e-6f) : 1.0f;
        const int left  = V.vocab - T.sh * P.vocab_padded;
        T.vocab         = left < P.vocab_padded ? left : P.vocab_padded;
        T.vocab         = T.vocab < 1 ? 1 : T.vocab;
        const RowSpan S = row_span((size_t)V.logits[T.sh] + (size_t)T.r * P.vocab_padded * 2, T.vocab);
        T.base          = (const char*)S.base;
        T.mis           = S.mis;
        T.nv            = S.nv;
        return T;
    };
    // the row's vectors in four parts (of whole fours of vectors per thread: vector i of a thread belongs to group i % 4),
    // so that the first ones can be looked at while the last are on their way
    const u32 row_s = (u32)__cvta_generic_to_shared(row), bar_s = (u32)__cvta_generic_to_shared(s_bar);
    auto      inside = [&](const Task& T) { return whole_vectors(rows, P.vocab_padded, T.r, T.mis, T.nv); };
    auto      send   = [&](const Task& T) {
        if (tid == 0) {
            const VecRange W   = inside(T);
            const int      per = ((T.nv + NT - 1) / NT + 15) / 16 * 4 * NT;
            for (int g = 0; g < 4; ++g) {
                const int skip = g == 0 ? W.first : 0, left = W.last - g * per, n = left < 0 ? 0 : (left < per ? left : per);
                bulk_copy(row_s + 16u * (u32)(g * per + skip), T.base + 16 * (size_t)(g * per + skip), 16u * (u32)(n - skip),
                          bar_s + 8u * (u32)g);
            }
        }
    };
    send_args((int)blockIdx.x);
    args_here();
    if (tid == 0) {
        s_n = 0, s_nspec = 0, s_nhot = 0, s_m = 0, s_lost = 0;
        for (int g = 0; g < 4; ++g) {
            bar_init(bar_s + 8u * (u32)g);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    Task cur = task_of((int)blockIdx.x);
    if (cur.live) {
        send(cur);
    }
    __syncthreads();  // (the arguments are looked at by all threads before the next ones take their place)
    u32  parity = 0;  // of the row at hand, on all four barriers
    auto wait   = [&](int g) {
        if (!bar_wait(bar_s + 8u * (u32)g, parity)) {
            s_lost = 1;  // (the row is reported as undecided)
        }
    };
    for (int t = blockIdx.x; t < tasks; t += gridDim.x) {
        const Task T   = cur;
        u64* const rec = P.trace != nullptr ? P.trace + (size_t)(t % rows) * kTraceWords : nullptr;
        if (rec != nullptr && tid == 0) {
            rec[0] = (u64)T.r, rec[1] = (u64)blockIdx.x, rec[2] = global_timer_ns();
        }
        send_args(t + (int)gridDim.x);
        u64* const out = V.out + (size_t)t * (P.vp_cap + 2);
        if (!T.live) {
            // nothing to send, or a top-p row: the general kernel's (statistics form)
            if (tid == 0) {
                if (T.topp) {
                    P.redo_rows[atomicAdd(P.redo_count, 1u)] = T.r;
                }
                else {
                    out[0] = 0;
                }
            }
            args_here();
            __syncthreads();
            cur = task_of(t + (int)gridDim.x);
            if (cur.live) {
                send(cur);
            }
            __syncthreads();
            continue;
        }
        const __half inv_t_h = __float2half_rn(T.inv_t);
        const int    id0     = V.offset + T.sh * P.vocab_padded;  // token id of the shard's first column
        // columns of the first and the last vector that are not the row's, and those of a vector that was not copied
        auto edge = [&](int j, uint4& v) {
            const VecRange W0 = inside(T);
            if (j < W0.first || j >= W0.last) {
#pragma unroll 1
                for (int c = max(j * 8 - T.mis, 0); c < min(j * 8 + 8 - T.mis, T.vocab); ++c) {
                    sts_u16(row_s + 2u * (u32)(T.mis + c), (u32)__ldg((const unsigned short*)T.base + T.mis + c));
                }
                v = row[j];
            }
            u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int c = j * 8 + e - T.mis;
                if (c < 0 || c >= T.vocab) {
                    w[e >> 1] = e & 1 ? (w[e >> 1] & 0xffffu) | (kDead2 & 0xffff0000u) : (w[e >> 1] & 0xffff0000u) | (kDead2 & 0xffffu);
                }
            }
            v      = make_uint4(w[0], w[1], w[2], w[3]);
            row[j] = v;
        };
        const bool own_edge = (tid == 0 && T.mis != 0) || ((T.mis + T.vocab) % 8 != 0 && (T.nv - 1) % NT == tid);
        if (special_launch) {
            for (int g = 0; g < 4; ++g) {
                wait(g);
            }
            if (own_edge) {
                for (int j = tid; j < T.nv; j += NT) {
                    if (j == 0 || j == T.nv - 1) {
                        uint4 v = row[j];
                        edge(j, v);
                    }
                }
            }
            __syncthreads();
            // takes column `id` out of the copy; true for the one thread that gets its raw value
            auto take = [&](int id, u32& raw) {
                const int c = id - id0;
                if (c < 0 || c >= T.vocab) {
                    return false;
                }
                const int at  = T.mis + c;
                const u32 old = atomicOr((u32*)smem_raw + (at >> 1), at & 1 ? 0xffff0000u : 0xffffu);
                raw           = at & 1 ? old >> 16 : old & 0xffffu;
                return raw != 0xffffu;
            };
            u32          raw;
            const size_t col = (size_t)P.ite * rows + T.r;
            if (P.bad_words != nullptr) {
                // banned words (kernels/ban_bad_words.cu:35-85): the last token, when the tokens in front of it match
                const int  L     = P.bad_words_len;
                const int* words = P.bad_words_shared ? P.bad_words : P.bad_words + (size_t)T.r * 2 * L;
                for (int i = tid; i < L; i += NT) {
                    const int e1 = words[L + i];
                    if (e1 < 0) {
                        continue;
                    }
                    const int s1 = i > 0 ? words[L + i - 1] : 0, size = e1 - s1;
                    bool      b  = size == 1;
                    if (size > 1 && P.step >= size - 1) {
                        b = true;
                        for (int j = size - 2; j >= 0 && b; --j) {
                            b = P.output_ids[(size_t)(P.step - (size - 1) + j) * P.batch_size + col] == words[s1 + j];
                        }
                    }
                    if (b && 0 < words[e1 - 1]) {
                        take(words[e1 - 1], raw);
                    }
                }
            }
            if (P.apply_minlen && tid == 0 && P.seq_len[T.r] + 1 - P.max_input_len < P.min_lengths[T.r]) {
                take(P.end_ids[T.r], raw);
            }
            __syncthreads();
            if (P.apply_rep) {
                const int input_len = P.input_lengths != nullptr ? P.input_lengths[T.r] : P.max_input_len;
                Xf        X;
                X.theta = P.rep_penalty[T.r], X.apply_rep = 1, X.penalty_type = P.penalty_type;
                for (int h = tid; h < P.step; h += NT) {
                    if (h >= input_len && h < P.max_input_len) {
                        continue;
                    }
                    const int id = P.output_ids[(size_t)h * P.batch_size + col];
                    if (take(id, raw)) {
                        const float y = special_value<DT>(X, f_value<DT>(raw, temp, T.inv_t, inv_t_h), kFlagHist);
                        if (y > neg_max) {
                            spec[atomicAdd(&s_nspec, 1u)] = ((u64)(~fkey(y)) << 32) | (u32)(id - id0);
                        }
                    }
                }
            }
            __syncthreads();
        }
        if (rec != nullptr) {
            trace_mark(rec, 0);
        }

        // ---- 1. group maxima and the threshold ----
        const int ni = (T.nv + NT - 1) / NT;
        u32       mx[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            mx[u] = kDead2;
        }
        {
            const int q    = (ni + 15) / 16 * 4;
            auto      part = [&](int g) {
                const int i1 = (g + 1) * q < ni ? (g + 1) * q : ni;
                for (int i = g * q; i < i1; i += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int j = (i + u) * NT + tid;
                        if (i + u < i1 && j < T.nv) {
                            uint4 v = row[j];
                            if (own_edge && !special_launch && (j == 0 || j == T.nv - 1)) {
                                edge(j, v);  // (done above, and columns taken out since, where there are special ones)
                            }
                            mx[u] = max2<DT>(mx[u], max2<DT>(max2<DT>(v.x, v.y), max2<DT>(v.z, v.w)));
                        }
                    }
                }
            };
            for (int g = 0; g < 4; ++g) {
                wait(g);
                part(g);
            }
            parity ^= 1u;
        }
        if (rec != nullptr) {
            trace_mark(rec, 1);
        }
        u32 thr;
        if (T.k <= NT * 3 / 8) {
            const u32 a = max2<DT>(max2<DT>(mx[0], mx[1]), max2<DT>(mx[2], mx[3]));
            const u32 x = key16(a & 0xffffu), y = key16(a >> 16);
            s_max[tid]  = (unsigned short)(x > y ? x : y);
            __syncthreads();
            if (tid < 32) {
                u32 mine[NT / 32], lo = 0xffffu, hi = 0;
#pragma unroll
                for (int i = 0; i < NT / 32; ++i) {
                    mine[i] = s_max[i * 32 + lane];
                    lo      = mine[i] < lo ? mine[i] : lo;
                    hi      = mine[i] > hi ? mine[i] : hi;
                }
                lo = __reduce_min_sync(0xffffffffu, lo);
                hi = __reduce_max_sync(0xffffffffu, hi);
                // two bits a round: three bounds counted at once, ten bits each (a bound above the least one: at most NT - 1 reach it)
                // (one bit a round: 295.9 us for 2048 rows of 8 x 32000 bf16, 292.7 so and with the merge's arguments ahead)
                while (lo < hi) {
                    const u32 q = (hi - lo + 3) >> 2, m1 = lo + q, m2 = m1 + q, m3 = m2 + q;
                    u32       c = 0;
#pragma unroll
                    for (int i = 0; i < NT / 32; ++i) {
                        c += (mine[i] >= m1 ? 1u : 0u) + (mine[i] >= m2 ? 1u << 10 : 0u) + (mine[i] >= m3 ? 1u << 20 : 0u);
                    }
                    c            = __reduce_add_sync(0xffffffffu, c);
                    const bool a1 = (c & 1023u) >= (u32)T.k, a2 = (c >> 10 & 1023u) >= (u32)T.k, a3 = c >> 20 >= (u32)T.k;
                    const u32  up = a3 ? hi : (a2 ? m3 : (a1 ? m2 : m1)) - 1;
                    lo            = a3 ? m3 : (a2 ? m2 : (a1 ? m1 : lo));
                    hi            = up < hi ? up : hi;
                }
                if (lane == 0) {
                    s_thr = lo;
                }
            }
            __syncthreads();
            thr = s_thr;
        }
        else {
            u32 key[8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                key[2 * u]     = key16(mx[u] & 0xffffu);
                key[2 * u + 1] = key16(mx[u] >> 16);
            }
            if (tid < 3) {
                s_cnt[tid] = 0;
            }
            __syncthreads();
            u32 lo = 0, hi = 0xffffu;
            for (int it = 0; it < 16; ++it) {  // (three counters in turn: one barrier a round)
                const u32 mid = (lo + hi + 1) >> 1;
                u32       c   = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    c += key[i] >= mid ? 1u : 0u;
                }
                c = __reduce_add_sync(0xffffffffu, c);
                if (lane == 0) {
                    atomicAdd(&s_cnt[it % 3], c);
                }
                if (tid == 0) {
                    s_cnt[(it + 1) % 3] = 0;
                }
                __syncthreads();
                const u32 all = s_cnt[it % 3];
                lo            = all >= (u32)T.k ? mid : lo;
                hi            = all >= (u32)T.k ? hi : mid - 1;
            }
            thr = lo;
        }
        auto value_of = [&](u32 key) { return f_value<DT>(key16_inv(key), temp, T.inv_t, inv_t_h); };
        // patterns below the threshold whose value after temperature is the same belong to its class
        auto whole_class = [&](u32 key) {
            if (temp) {
                const float y = value_of(key);
                while (key > 0 && value_of(key - 1) == y) {
                    --key;
                }
            }
            return key;
        };
        const u32 thr0 = thr;
        thr            = whole_class(thr);
        if (rec != nullptr) {
            trace_mark(rec, 2);
        }

        // ---- 2. the columns at or above it ----
        auto take_specials = [&](u32 least) {
            for (u32 i = tid; i < s_nspec; i += NT) {
                if (~(u32)(spec[i] >> 32) >= least) {
                    const u32 at = atomicAdd(&s_n, 1u);
                    if (at < (u32)V.cand_cap) {
                        cand[at] = spec[i];
                    }
                }
            }
        };
        // the columns `pm` of vector j, `c` of them
        auto put = [&](const uint4& v, int j, u32 pm, u32 c) {
            u32 pos = c != 0 ? atomicAdd(&s_n, c) : 0u;
            while (pm != 0) {
                const int e = __ffs(pm) - 1;
                pm &= pm - 1;
                if (pos < (u32)V.cand_cap) {
                    const float y = f_value<DT>(raw_bits<DT>(v, e), temp, T.inv_t, inv_t_h);
                    cand[pos]     = ((u64)(~fkey(y)) << 32) | (u32)(j * 8 + e - T.mis);
                }
                ++pos;
            }
        };
        bool by_hand = !(T.inv_t > 0.0f && T.inv_t < 3.0e38f && value_of(thr0) > neg_max);
        if (!by_hand) {
            // only groups whose largest value reaches the threshold are looked at again, their vectors spread over all
            // threads: 70 to 100 groups of 1024 for k = 64 (every thread going over its own vectors: 3.0 us instead of 1)
            u32 at = 0, b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const u32 x = key16(mx[u] & 0xffffu), y = key16(mx[u] >> 16);
                b[u] = __ballot_sync(0xffffffffu, (x > y ? x : y) >= thr);
                at += __popc(b[u]);
            }
            if (at != 0) {
                if (lane == 0) {
                    at = atomicAdd(&s_nhot, at);
                }
                at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if ((b[u] >> lane) & 1u) {
                        s_hot[at + __popc(b[u] & ((1u << lane) - 1u))] = (unsigned short)(tid * 4 + u);
                    }
                    at += __popc(b[u]);
                }
            }
            __syncthreads();
            trace_mark(rec, 5);
            const u32 thr2  = key16_inv(thr) * 0x10001u;
            const int gs    = (ni + 3) / 4, items = (int)s_nhot * gs;
            for (int x0 = tid & ~31; x0 < items; x0 += NT) {
                const int  x  = x0 + lane;
                const int  h  = x / gs, i = 4 * (x - h * gs);
                const int  q  = h < (int)s_nhot ? (int)s_hot[h] : 0;
                const int  j  = (i + (q & 3)) * NT + (q >> 2);
                const bool in = (x < items) & (j < T.nv);
                u32        pm = 0, c = 0;
                uint4      v = make_uint4(0, 0, 0, 0);
                if (in) {
                    v            = row[j];
                    const u32 m0 = ge2_mask<DT>(v.x, thr2), m1 = ge2_mask<DT>(v.y, thr2);
                    const u32 m2 = ge2_mask<DT>(v.z, thr2), m3 = ge2_mask<DT>(v.w, thr2);
                    pm = ((m0 & 1u) | ((m0 >> 15) & 2u)) | (((m1 & 1u) | ((m1 >> 15) & 2u)) << 2)
                         | (((m2 & 1u) | ((m2 >> 15) & 2u)) << 4) | (((m3 & 1u) | ((m3 >> 15) & 2u)) << 6);
                    c = (u32)__popc(pm);
                }
                put(v, j, pm, c);
            }
            take_specials(fkey(value_of(thr)));
            args_here();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (what was written into the copy, before the next one)
            __syncthreads();
            by_hand = s_n > (u32)V.cand_cap;
            trace_mark(rec, 6);
        }
        if (by_hand) {
            // rare: the k-th largest final value itself, by bisection over the ordered 32-bit keys
            auto mask_of = [&](const uint4& v, u32 least, u32& pm) {
                pm = 0;
#pragma unroll 1
                for (int e = 0; e < 8; ++e) {
                    const float y = f_value<DT>(raw_bits<DT>(v, e), temp, T.inv_t, inv_t_h);
                    pm |= (y > neg_max && fkey(y) >= least ? 1u : 0u) << e;
                }
                return (u32)__popc(pm);
            };
            u32 lo = fkey(neg_max) + 1u, hi = fkey(INFINITY);
            for (bool first = true; first || lo < hi; first = false) {
                // (the first round looks at `lo` itself: with fewer than k values in all, every one of them goes)
                const u32 mid = first ? lo : lo + (hi - lo + 1u) / 2u;
                __syncthreads();
                if (tid == 0) {
                    s_cnt[0] = 0;
                }
                __syncthreads();
                u32 c = 0, pm;
                for (int i = 0; i < ni; ++i) {
                    const int j = i * NT + tid;
                    if (j < T.nv) {
                        c += mask_of(row[j], mid, pm);
                    }
                }
                for (u32 s = tid; s < s_nspec; s += NT) {
                    c += ~(u32)(spec[s] >> 32) >= mid ? 1u : 0u;
                }
                c = __reduce_add_sync(0xffffffffu, c);
                if (lane == 0) {
                    atomicAdd(&s_cnt[0], c);
                }
                __syncthreads();
                const bool enough = s_cnt[0] >= (u32)T.k;
                if (first) {
                    hi = enough ? hi : lo;
                }
                else if (enough) {
                    lo = mid;
                }
                else {
                    hi = mid - 1u;
                }
            }
            __syncthreads();
            if (tid == 0) {
                s_n = 0;
            }
            __syncthreads();
            for (int i = 0; i < ni; ++i) {
                const int j  = i * NT + tid;
                u32       pm = 0, c = 0;
                if (j < T.nv) {
                    c = mask_of(row[j], lo, pm);
                }
                put(j < T.nv ? row[j] : make_uint4(0, 0, 0, 0), j, pm, c);
            }
            take_specials(lo);
            args_here();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
        const int n = (int)s_n;
        cur = task_of(t + (int)gridDim.x);
        if (cur.live) {
            send(cur);  // (no thread looks at this row's copy again)
        }
        if (rec != nullptr) {
            trace_mark(rec, 3);
        }

        // ---- 3. order, and the record: everything down to the k-th value's last equal ----
        const int k_eff = T.k < n ? T.k : n;
        if (n > V.cand_cap) {
            __syncthreads();
            if (tid == 0) {
                out[0] = ~0ull;  // more equal values than the record holds
                s_n = 0, s_nspec = 0, s_nhot = 0, s_m = 0;
            }
            __syncthreads();
            continue;
        }
        auto emit = [&](u64 e, int at) {
            if ((u32)(e >> 32) <= s_kv) {
                if (at < P.vp_cap) {
                    out[1 + at] = (e & 0xffffffff00000000ull) | (u64)((u32)(e & 0xffffffffu) + (u32)id0);
                }
                if (at + 1 >= k_eff) {
                    atomicMax(&s_m, (u32)at + 1u);
                }
            }
        };
        if (n <= 2 * NT) {
            const u64 e0 = tid < n ? cand[tid] : ~0ull, e1 = tid + NT < n ? cand[tid + NT] : ~0ull;
            int       c0 = 0, c1 = 0;
            if ((tid & ~31) < n) {
                auto before = [&](auto two) {
#pragma unroll 4
                    for (int b = 0; b + 1 < n; b += 2) {
                        const ulonglong2 x = *(const ulonglong2*)(cand + b);
                        c0 += (x.x < e0 ? 1 : 0) + (x.y < e0 ? 1 : 0);
                        if (two) {
                            c1 += (x.x < e1 ? 1 : 0) + (x.y < e1 ? 1 : 0);
                        }
                    }
                    if (n & 1) {
                        const u64 x = cand[n - 1];
                        c0 += x < e0 ? 1 : 0;
                        c1 += x < e1 ? 1 : 0;
                    }
                };
                if (n > NT) {
                    before(std::true_type());
                }
                else {
                    before(std::false_type());
                }
                if (tid < n && c0 == k_eff - 1) {
                    s_kv = (u32)(e0 >> 32);
                }
                if (tid + NT < n && c1 == k_eff - 1) {
                    s_kv = (u32)(e1 >> 32);
                }
            }
            __syncthreads();
            if (tid < n) {
                emit(e0, c0);
            }
            if (tid + NT < n) {
                emit(e1, c1);
            }
        }
        else {
            group_sort_u64(cand, n, tid, NT, CtaSync());
            __syncthreads();
            if (tid == 0) {
                s_kv = (u32)(cand[k_eff - 1] >> 32);
            }
            __syncthreads();
            for (int a = tid; a < n; a += NT) {
                emit(cand[a], a);
            }
        }
        __syncthreads();
        trace_mark(rec, 7);
        if (tid == 0) {
            const u32 m = s_m;
            out[0]      = m > (u32)P.vp_cap || s_lost ? ~0ull : (u64)m;
            s_n = 0, s_nspec = 0, s_nhot = 0, s_m = 0;
            if (rec != nullptr) {
                rec[3] = global_timer_ns();
            }
        }
        __syncthreads();
    }
}

template<int DT>
int vp_select_launch(const KParams& K, const VpArgs& V, size_t smem, int sms, cudaStream_t st)
{
    // CTAs per SM by shared memory (3.7 KB more per CTA are the kernel's and the system's); the registers allow four of 256 threads.  A row
    // that leaves room for one CTA only gets 512 threads.
    int per_sm = (int)((228 * 1024) / (smem + 3 * 1024 + 768));
    per_sm     = per_sm < 1 ? 1 : (per_sm > 4 ? 4 : per_sm);
    static std::atomic<bool> ready_256[kDevicesKnown], ready_512[kDevicesKnown];
    FTB_CUDA_CHECK(per_sm == 1 ? opt_in_smem(vp_select_kernel<DT, 512>, kVpMaxSmem, ready_512) :
                                 opt_in_smem(vp_select_kernel<DT, 256>, kVpMaxSmem, ready_256));
    const long long tasks = (long long)K.local_batch * V.n_shards;
    int             grid  = sms * per_sm;
    grid                  = grid < tasks ? grid : (int)tasks;
    if (per_sm == 1) {
        FTB_CUDA_CHECK(launch_early(vp_select_kernel<DT, 512>, dim3((unsigned)grid), dim3(512), smem, st, K, V));
    }
    else {
        FTB_CUDA_CHECK(launch_early(vp_select_kernel<DT, 256>, dim3((unsigned)grid), dim3(256), smem, st, K, V));
    }
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

}  // namespace ftb200
