// Decode-sampling step with a row split over a cluster of CTAs (sm_100a thread-block clusters, distributed shared
// memory).  One cluster serves one row: CTA c of n owns the columns whose number modulo 1024 lies in
// [c * 1024 / n, (c + 1) * 1024 / n), keeps their final values (temperature, bias, penalties and bans applied) in its
// shared memory as fp32, and every later step - maximum, ordered soft-max denominator, histogram, selection, nucleus
// sort - reads shared memory only: the row is read from HBM once, whatever the logits type and options are.
//
// Why this split: the reference's soft-max denominator is a sum over 1024 strided chains (column modulo 1024, added
// chunk after chunk), so a CTA that owns whole chains can add them in the reference's order without talking to the
// others, and the special columns (history, bans) are scattered evenly.  What is exchanged per row is small: a bit per
// special column, one maximum and 1024 / 32 / n partial sums per CTA, a 2048-bin histogram, the candidates.
//
// What bounds it: latency.  A row takes cluster barriers of 0.5 us each - three for an arg-max row, six where few candidates are
// left, eight or ten for a nucleus that one or several CTAs sort, one more with special columns, the last one at its end -
// and about six sweeps over its shared memory; a CTA-per-row kernel walks eight times as many columns with the same 256 threads.  Measured on B200, one row
// alone on its SMs: arg-max of 32000 columns 4 us, k = 50 of 50257 fp32 13 us, a nucleus of 50257 fp32 19 us (the general
// kernel: 180 to 1100 us), 128256 bf16 with 2500 tokens of history 5 us (k = 1) to 45 us (the widest nucleus of 96 rows).  Batch
// of 64 x 50257 fp32 top-p: 42 us a step; 48 x 51200 half with bias and log-probs: 51 us; 24 steps of 16 x 128256 bf16: 1300 to
// 1390 us.  Before the nucleus was placed by bin, sorted by short loops and the general row code taken out: 60, 83, 1600 to 1930.
//
// Code size matters: a row runs through most of this code once, so a loop that is unrolled for the largest case waits for
// its instructions in every case.
//
// The results are those of sampling_kernels.cuh, bit for bit; rows that do not fit the fixed tables here (a nucleus
// above the collection areas, thousands of equal values around the k-th) go to the general row code.
#pragma once
#include "sampling_kernels.cuh"

namespace ftb200 {

// ---- distributed shared memory ----------------------------------------------------------------------------------
__device__ __forceinline__ u32 cluster_rank()
{
    u32 r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ u32 cluster_addr(u32 smem, u32 rank)
{
    u32 a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_arrive()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait()
{
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync()
{
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ void dst_u32(u32 a, u32 v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void dst_u64(u32 a, u64 v)
{
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ u32 dld_u32(u32 a)
{
    u32 v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ u32 datom_add(u32 a, u32 v)
{
    u32 o;
    asm volatile("atom.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ void dred_or(u32 a, u32 v)
{
    asm volatile("red.shared::cluster.or.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void dred_min(u32 a, u32 v)
{
    asm volatile("red.shared::cluster.min.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void dred_max(u32 a, u32 v)
{
    asm volatile("red.shared::cluster.max.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void dred_add(u32 a, u32 v)
{
    asm volatile("red.shared::cluster.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ u32 smem_addr(const void* p)
{
    return (u32)__cvta_generic_to_shared(p);
}

// ---- bins -------------------------------------------------------------------------------------------------------
// Distance d below the row maximum -> position on the scale of bins: 128 bins a logit for the first 8 (where nearly
// every selection ends), 32 up to 24, 8 beyond.  The least of three lines: monotone, no branch, and a distance that is
// not a number lands on the last bin.
__device__ __forceinline__ float sp_pos(float d)
{
    return fminf(fminf(fminf(d * 128.0f, d * 32.0f + 768.0f), d * 8.0f + 1344.0f), (float)(kSpBins - 1));
}
__device__ __forceinline__ int sp_bin(float d)
{
    return (int)sp_pos(d);
}
__device__ __forceinline__ float sp_edge(int b)  // near edge of bin b = far edge of bin b - 1
{
    return fmaxf(fmaxf((float)b * (1.0f / 128.0f), ((float)b - 768.0f) * (1.0f / 32.0f)), ((float)b - 1344.0f) * 0.125f);
}
// a value that every column of bins 0 .. b reaches (the exact test is the bin's)
__device__ __forceinline__ float sp_floor_value(float maxv, int b)
{
    return b + 1 < kSpBins ? maxv - sp_edge(b + 1) * 1.0001f - 1e-6f * fabsf(maxv) - 1e-6f : -INFINITY;
}

// Exclusive block-wide prefix of one value per thread; *total receives the sum.
static __device__ u32 block_excl_u32(u32 v, u32* total)
{
    __shared__ u32 s_w[kWarps];
    const int      lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    u32            incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, incl, off);
        incl += lane >= off ? t : 0u;
    }
    __syncthreads();  // (the previous call's sums have been read)
    if (lane == 31) {
        s_w[wid] = incl;
    }
    __syncthreads();
    u32 base = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) {
        const u32 w = s_w[i];
        base += i < wid ? w : 0u;
        tot += w;
    }
    *total = tot;
    return base + incl - v;
}

// Shared-memory map of a CTA, as 32-bit addresses and pointers.
struct SpMap {
    float* y;       // [slice] final values of this CTA's columns; local index = (column / 1024) * vt + column % vt
    u32*   area;    // [area_cap] nucleus keys received (all CTAs) or 64-bit candidates (leader)
    u32*   merged;  // [kSpBins] counts of the whole row, then their exclusive prefix
    u32*   sub;     // [area_cap / 4] pairs of 16-bit sub-bucket counters
    u32*   hist;    // [kSpBins] counts of this CTA's columns, then cursors
    int    area_cap;
};

struct SpShared {
    float wsum[32];        // warp sums of the soft-max denominator, written by all CTAs
    u32   max_key;         // of the row's largest value
    u32   first_max;       // smallest column that holds the maximum
    u32   n_cls;           // columns of the crossing class
    u32   verdict;         // 0 class found, 1 draw beyond the whole row (best token), 2 leave the row
    union {
        u32   p_sel;       // crossing: probability (bits),
        float per_y;       // (until it is looked for: raw value per unit of a final value, bfloat16 rows)
    };
    u32   j_sel;           // position in the sorted order
    u32   larger;          // columns of a larger probability than the crossing's
    u32    bad_order;
    u32    state[6];       // counter and words of the row's generator after its draw (nothing else of it moves)
    // (static and dynamic shared memory have to leave room for two CTAs with kTwoPerSm, which is asked for in whole kilobytes: at most 5120
    // bytes of static memory, which build.py checks)
    union {
        u64               best[kSpMaxN * kWarps];  // arg-max rows, a warp each: key of its largest value << 32 | the largest tie key of its columns
        alignas(16) float agg[(kSpMaxN * kSpAreaWide) / 256];  // nuclei: sums of 256 probabilities
    };
};

// Bias of a 32-bit word of logits in the logits type's arithmetic (half: two rounded sums; fp32: one).  bf16 sums stay
// fp32 in the reference's order of operations and do not fit the word: they are added per column.
template<int DT>
__device__ __forceinline__ u32 sp_add_bias(u32 x, u32 b)
{
    if (DT == FTB200_F16) {
        const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&x), *reinterpret_cast<const __half2*>(&b));
        return *reinterpret_cast<const u32*>(&r);
    }
    return __float_as_uint(__uint_as_float(x) + __uint_as_float(b));
}

// Loads this CTA's columns of row r and stores their values after temperature and bias.  Returns the thread's largest.
template<int DT>
__device__ __forceinline__ float sp_load_slice(const KParams& P, const Xf& X, const char* rowp, float* y, int rank, int lgvt,
                                              int nchunk)
{
    constexpr int ES = DT == FTB200_F32 ? 4 : 2, EPV = 16 / ES, LGE = DT == FTB200_F32 ? 2 : 3;
    const int     tid = threadIdx.x, vt = 1 << lgvt, col0 = rank << lgvt, vocab = P.vocab;
    float         best = -INFINITY;
    if (((size_t)rowp & 15) == 0 && lgvt >= LGE) {
        // a chunk of 1024 columns starts on a 16-byte boundary: whole vectors, eight in flight per thread (a slice of 16000
        // half-precision columns in one round)
        constexpr int U   = 8;
        const int     lgv = lgvt - LGE, nv = nchunk << lgv;
        const bool    bias = X.apply_temp && X.bias != nullptr, bias_vec = DT != FTB200_BF16 && bias && ((size_t)X.bias & 15) == 0;
        Xf            T    = X;  // (a bias that comes by the vector is added here)
        T.bias             = bias_vec ? nullptr : X.bias;
        for (int i0 = tid; i0 < nv; i0 += kThreads * U) {
            uint4 q[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * kThreads, v = ((i >> lgv) << 10) + col0 + ((i & ((1 << lgv) - 1)) << LGE);
                if (i < nv && v + EPV <= vocab) {
                    q[u] = ld_nc_v4(rowp + (size_t)v * ES);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = i0 + u * kThreads, v = ((i >> lgv) << 10) + col0 + ((i & ((1 << lgv) - 1)) << LGE);
                if (i >= nv) {
                    continue;
                }
                float f[EPV];
                if (v + EPV <= vocab) {
                    if (bias_vec) {
                        const uint4 b = ld_nc_v4((const char*)X.bias + (size_t)v * ES);
                        q[u]          = make_uint4(sp_add_bias<DT>(q[u].x, b.x), sp_add_bias<DT>(q[u].y, b.y),
                                                   sp_add_bias<DT>(q[u].z, b.z), sp_add_bias<DT>(q[u].w, b.w));
                    }
#pragma unroll
                    for (int e = 0; e < EPV; ++e) {
                        f[e] = temp_value<DT>(T, raw_bits<DT>(q[u], e), v + e);
                    }
                }
                else {
#pragma unroll
                    for (int e = 0; e < EPV; ++e) {
                        f[e] = -INFINITY;
                        if (v + e < vocab) {
                            const u32 bits = DT == FTB200_F32 ? __ldg((const u32*)rowp + v + e) :
                                                                (u32)__ldg((const unsigned short*)rowp + v + e);
                            f[e]           = temp_value<DT>(X, bits, v + e);
                        }
                    }
                }
                float4* dst = (float4*)(y + ((size_t)i << LGE));
#pragma unroll
                for (int e = 0; e < EPV; e += 4) {
                    dst[e / 4] = make_float4(f[e], f[e + 1], f[e + 2], f[e + 3]);
                    best       = fmaxf(best, fmaxf(fmaxf(f[e], f[e + 1]), fmaxf(f[e + 2], f[e + 3])));
                }
            }
        }
    }
    else {
        // A row that starts between two 16-byte boundaries: one column per load, a bias beside it (246 x 114514 bf16 with a bias that was
        // sent for once a column had come: 226 us a step, 162 so).  The next eight columns are on their way while eight are worked on, and no
        // load stands behind a branch: how many were in flight otherwise changed with the registers around the loop.  us a step, loads
        // behind a branch, as two builds of the same loop had them / eight, sixteen at a time without one / so: 28 x 208295 fp32 of both kinds
        // 64.5, 77.2 / 85.3, 75.1 / 63.1; 200 x 101001 fp32 145.8, 154.6 / 169.4, 156.5 / 142.2; 100 x 128257 bf16 118.5, 106.7 / 87.5, 88.0 /
        // 87.6; 300 x 39775 half nucleus rows 313, 182.2 / 172.5, 174.7 / 162.7; 246 x 114515 bf16, k = 40, with a bias 240, 219.6 / 184.0, 183.5 /
        // 180.3.  (Four columns ahead of four: 75.7, 155.7, 98.1, 176.3, 201.0.)
        constexpr int U    = 8;
        const int     ny   = nchunk << lgvt;
        Xf            T    = X;
        T.bias             = nullptr;  // (it is added here)
        auto walk = [&](auto with_bias) {
            constexpr bool kBias = decltype(with_bias)::value;
            u32            q[U], b[kBias ? U : 1];
            auto           send = [&](int i0, u32* qn, u32* bn) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * kThreads, v = ((i >> lgvt) << 10) + col0 + (i & (vt - 1));
                    const int at = i < ny && v < vocab ? v : 0;  // (no branch around a load)
                    qn[u]        = DT == FTB200_F32 ? __ldg((const u32*)rowp + at) : (u32)__ldg((const unsigned short*)rowp + at);
                    if (kBias) {
                        bn[u] = DT == FTB200_F32 ? __ldg((const u32*)X.bias + at) : (u32)__ldg((const unsigned short*)X.bias + at);
                    }
                }
            };
            send(tid, q, b);
#pragma unroll 1
            for (int i0 = tid; i0 < ny; i0 += kThreads * U) {
                u32 qn[U], bn[kBias ? U : 1];
                send(i0 + kThreads * U, qn, bn);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * kThreads, v = ((i >> lgvt) << 10) + col0 + (i & (vt - 1));
                    if (i < ny) {
                        if (!kBias) {
                            y[i] = v < vocab ? temp_value<DT>(T, q[u], v) : -INFINITY;
                        }
                        else if (v >= vocab) {
                            y[i] = -INFINITY;
                        }
                        else if (DT == FTB200_BF16) {
                            y[i] = (__uint_as_float(q[u] << 16) + __uint_as_float(b[kBias ? u : 0] << 16)) * X.inv_t;
                        }
                        else {
                            y[i] = temp_value<DT>(T, sp_add_bias<DT>(q[u], b[kBias ? u : 0]), v);
                        }
                        best = fmaxf(best, y[i]);
                    }
                    q[u] = qn[u];
                    if (kBias) {
                        b[kBias ? u : 0] = bn[kBias ? u : 0];
                    }
                }
            }
        };
        if (X.apply_temp && X.bias != nullptr) {
            walk(std::true_type{});
        }
        else {
            walk(std::false_type{});
        }
    }
    return best;
}

// History ids of the row that this CTA looks after, kHistRegs per thread: loaded before the row itself so that they are
// there when the bit maps are ready.  (-1: a padding position or none.)
constexpr int kHistRegs = 2;
__device__ __forceinline__ int sp_history_id(const KParams& P, size_t col, int input_len, int t)
{
    // sampling_penalty_kernels.cu:385-410
    return (t < P.step && !(t >= input_len && t < P.max_input_len)) ? P.output_ids[(size_t)t * P.batch_size + col] : -1;
}

// Marks the special columns of the row in the bit maps of the CTAs that own them: history ids (map 0) and banned words /
// the masked end token (map 1).  The CTAs of the cluster share the work.
template<int LGN>
__device__ __noinline__ void sp_mark_specials(const KParams& P, int r, u32 bits_addr, int words, int rank, int id0, int id1)
{
    constexpr int n = 1 << LGN, lgvt = 10 - LGN;
    const int     tid = threadIdx.x;
    const size_t  col = (size_t)P.ite * P.local_batch + r;
    auto          mark = [&](int v, int map) {
        if (v < 0 || v >= P.vocab) {
            return;
        }
        const int local = ((v >> 10) << lgvt) | (v & ((1 << lgvt) - 1));
        dred_or(cluster_addr(bits_addr + 4u * (u32)(map * words + (local >> 5)), (u32)((v & 1023) >> lgvt)), 1u << (local & 31));
    };
    if (P.apply_rep) {
        const int input_len = P.input_lengths != nullptr ? P.input_lengths[r] : P.max_input_len;
        mark(id0, 0);
        mark(id1, 0);
        for (int t = (kHistRegs * n + rank) * kThreads + tid; t < P.step; t += n * kThreads) {
            mark(sp_history_id(P, col, input_len, t), 0);
        }
    }
    if (P.bad_words != nullptr) {
        // a word bans its last token when the tokens before it match the tail of the sequence (ban_bad_words.cu:35-85)
        const int  L     = P.bad_words_len;
        const int* wbase = P.bad_words_shared ? P.bad_words : P.bad_words + (size_t)r * 2 * L;
        for (int i = rank * kThreads + tid; i < L; i += n * kThreads) {
            const int end = wbase[L + i];
            if (end < 0) {
                continue;
            }
            const int start = i > 0 ? wbase[L + i - 1] : 0, size = end - start;
            const int tok   = end > 0 ? wbase[end - 1] : 0;  // (an empty word stands in front of the list)
            bool      ban   = size == 1;
            if (size > 1 && P.step >= size - 1) {
                ban = true;
                for (int j = size - 2; j >= 0 && ban; --j) {
                    ban = P.output_ids[(size_t)(P.step - (size - 1) + j) * P.batch_size + col] == wbase[start + j];
                }
            }
            if (ban && tok > 0) {
                mark(tok, 1);
            }
        }
    }
    if (P.apply_minlen && rank == 0 && tid == 0 && P.seq_len[r] + 1 - P.max_input_len < P.min_lengths[r]) {
        mark(P.end_ids[r], 1);  // sampling_penalty_kernels.cu:493-499
    }
}

template<int DT>
__device__ __forceinline__ float sp_prob(float y, float maxv, float denom)
{
    return round_to_T<DT>(round_to_T<DT>(__expf(y - maxv)) / denom);
}

// Ordered pieces of the soft-max denominator: this CTA's virtual threads (columns modulo 1024) add their exponentials
// in chunk order, the butterfly over 32 of them follows, and the warp sums go to every CTA of the cluster.
template<int DT, int LGN>
__device__ __noinline__ void sp_chain_sums(const float* y, int nchunk, float maxv, u32 wsum_addr, int rank)
{
    constexpr int n = 1 << LGN, lgvt = 10 - LGN;
    FTB_ASSUME_SHARED(y);
    const int tid = threadIdx.x, vt = 1 << lgvt;
    for (int t = tid; t < vt; t += kThreads) {
        // the exponentials of the next eight chunks are on their way while those of the last eight are added
        float       a   = 0.0f, e[8];
        const int   m8  = nchunk & ~7;
        const float* yt = y + t;
        auto        eight = [&](int m, float* to) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                to[i] = round_to_T<DT>(__expf(yt[(m + i) << lgvt] - maxv));
            }
        };
        if (m8 > 0) {
            eight(0, e);
        }
#pragma unroll 1
        for (int m = 8; m < m8; m += 8) {
            float f[8];
            eight(m, f);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                a += e[i];
                e[i] = f[i];
            }
        }
        if (m8 > 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                a += e[i];
            }
        }
#pragma unroll 1
        for (int m = m8; m < nchunk; ++m) {
            a += round_to_T<DT>(__expf(yt[m << lgvt] - maxv));
        }
        // (vt is a multiple of 32: whole warps take part)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a = a + __shfl_xor_sync(0xffffffffu, a, o);
        }
        if ((tid & 31) == 0) {
            const u32 w = (u32)(((rank << lgvt) + t) >> 5);
#pragma unroll
            for (int q = 0; q < n; ++q) {
                dst_u32(cluster_addr(wsum_addr + 4u * w, (u32)q), __float_as_uint(a));
            }
        }
    }
}

// Per-thread walk over the CTA's values: f(local index, value) for every column not below thr, which has to lie above the
// values that cannot be selected.  Sixteen values a round become a mask without a branch; f stands in the loop over its
// bits once (inlined per value it was several times the instruction cache, and a branch per value cost more than the
// compare).
template<class F>
__device__ __forceinline__ void sp_sweep(const float* y, int ny, float thr, F&& f)
{
    FTB_ASSUME_SHARED(y);
    constexpr int U = 4;
    for (int i0 = 4 * (int)threadIdx.x; i0 < ny; i0 += 4 * kThreads * U) {
        u32 hits = 0;
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int    i = i0 + q * 4 * kThreads;
            const float4 v = i < ny ? *(const float4*)(y + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            hits |= (v.x >= thr ? 1u : 0u) << (4 * q);
            hits |= (v.y >= thr ? 2u : 0u) << (4 * q);
            hits |= (v.z >= thr ? 4u : 0u) << (4 * q);
            hits |= (v.w >= thr ? 8u : 0u) << (4 * q);
        }
        while (hits != 0) {
            const int e = __ffs(hits) - 1, i = i0 + (e >> 2) * 4 * kThreads + (e & 3);
            hits &= hits - 1;
            f(i, y[i]);
        }
    }
}

// The same for the columns with values in [lo, hi]; f returns a number to add.  Returns the thread's sum and its columns above hi.
template<class F>
__device__ __forceinline__ u32 sp_sweep_band(const float* y, int ny, float lo, float hi, F&& f)
{
    FTB_ASSUME_SHARED(y);
    constexpr int U = 4;
    u32           sum = 0;
    for (int i0 = 4 * (int)threadIdx.x; i0 < ny; i0 += 4 * kThreads * U) {
        u32 in = 0;
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int    i = i0 + q * 4 * kThreads;
            const float4 v = i < ny ? *(const float4*)(y + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            const u32    a = (v.x > hi ? 1u : 0u) | (v.y > hi ? 2u : 0u) | (v.z > hi ? 4u : 0u) | (v.w > hi ? 8u : 0u);
            const u32    b = (v.x >= lo ? 1u : 0u) | (v.y >= lo ? 2u : 0u) | (v.z >= lo ? 4u : 0u) | (v.w >= lo ? 8u : 0u);
            sum += __popc(a);
            in |= (b & ~a) << (4 * q);
        }
        while (in != 0) {
            const int e = __ffs(in) - 1, i = i0 + (e >> 2) * 4 * kThreads + (e & 3);
            in &= in - 1;
            sum += f(i, y[i]);
        }
    }
    return sum;
}

// The j-th smallest of n <= 512 columns.
static __device__ __noinline__ int sp_jth_of_few(const u32* cls, int n, int j)
{
    __shared__ u32 s_col;
    FTB_ASSUME_SHARED(cls);
    for (int i = threadIdx.x; i < n; i += kThreads) {
        const u32 c  = cls[i];
        int       rk = 0;
#pragma unroll 8
        for (int q = 0; q < n; ++q) {
            rk += cls[q] < c ? 1 : 0;
        }
        if (rk == j) {
            s_col = c;
        }
    }
    __syncthreads();
    return (int)s_col;
}

// Counts of the CTA's selectable columns per bin.
static __device__ __noinline__ void sp_count_bins(const float* y, int ny, float lowest, float maxv, u32 hist)
{
    FTB_ASSUME_SHARED(y);
    constexpr int U = 4;
    for (int i0 = 4 * (int)threadIdx.x; i0 < ny; i0 += 4 * kThreads * U) {
        float4 v[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int i = i0 + q * 4 * kThreads;
            v[q]        = i < ny ? *(const float4*)(y + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float x = e == 0 ? v[q].x : (e == 1 ? v[q].y : (e == 2 ? v[q].z : v[q].w));
                asm volatile("{\n .reg .pred p;\n setp.ge.f32 p, %0, %1;\n @p red.shared.add.u32 [%2], 1;\n}" ::"f"(x), "f"(lowest),
                             "r"(hist + 4u * (u32)sp_bin(maxv - x))
                             : "memory");
            }
        }
    }
}

// Columns of the nucleus (bins 0 .. b_thr) to their owners: `cursor` [kSpBins] holds, per bin, the cluster address of the next
// place of this CTA's keys.  No branch: at a tenth and more of the columns nearly every warp has a hit in every value, and
// four atomics are on their way before the first store waits for its place.
static __device__ __noinline__ void sp_scatter_keys(const float* y, int ny, float lowest, float maxv, u32 b_thr, u32 cursor)
{
    FTB_ASSUME_SHARED(y);
    constexpr int U = 2;
    for (int i0 = 4 * (int)threadIdx.x; i0 < ny; i0 += 4 * kThreads * U) {
        float4 v[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int i = i0 + q * 4 * kThreads;
            v[q]        = i < ny ? *(const float4*)(y + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
        u32 to[4 * U];
#pragma unroll
        for (int e = 0; e < 4 * U; ++e) {
            const float4& w = v[e >> 2];
            const float   x = (e & 3) == 0 ? w.x : ((e & 3) == 1 ? w.y : ((e & 3) == 2 ? w.z : w.w));
            const u32     b = (u32)sp_bin(maxv - x);
            asm volatile("{\n .reg .pred p;\n setp.le.u32 p, %1, %2;\n setp.ge.and.f32 p, %3, %4, p;\n mov.u32 %0, 0xffffffff;\n"
                         " @p atom.shared.add.u32 %0, [%5], 4;\n}"
                         : "=&r"(to[e])
                         : "r"(b), "r"(b_thr), "f"(x), "f"(lowest), "r"(cursor + 4u * b)
                         : "memory");
        }
#pragma unroll
        for (int e = 0; e < 4 * U; ++e) {
            const float4& w = v[e >> 2];
            const float   x = (e & 3) == 0 ? w.x : ((e & 3) == 1 ? w.y : ((e & 3) == 2 ? w.z : w.w));
            asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0xffffffff;\n @p st.shared::cluster.f32 [%0], %1;\n}" ::"r"(to[e]),
                         "f"(x)
                         : "memory");
        }
    }
}

// One nucleus owner's n keys (fp32 values, bin by bin) into descending order.  `excl` holds the first position of every bin in the
// row's order, `sub` counters for n / 2 sub-buckets.  A key's place inside its bin is guessed from
// its position between the bin's edges, so that a sub-bucket of two places receives two keys on average whatever the
// distribution is; inside it a key's place is the number of larger ones.
//
// The keys go to `tmp` by sub-bucket and come back in order: three short loops, because a row passes through this code once and
// an unrolled form waits for its instructions.  fp32 / bf16 logits, all steps of the sort: 900 keys 5.3 / 5.9 us, 3000 11.4 /
// 13.1, 4700 17 / 20 (keys held in registers by code unrolled for 10240 of them: 20 to 26 us).  Above half of the area it
// goes stretch by stretch: 5600 keys 24 / 27 us, 7500 33 / 38.  Returns false when a long sub-bucket of many values would
// have to be ordered.
constexpr int kSpShort = 24;   // keys of a sub-bucket that every thread orders for itself
constexpr int kSpLists = 256;  // words for the list of longer ones

// sub-bucket of a key, [0, (n + 1) / 2)
__device__ __forceinline__ u32 sp_sub_bucket(const u32* excl, float v, float maxv, u32 start, int n)
{
    const float t = sp_pos(maxv - v);
    const int   b = (int)t;
    const u32   e = excl[b], c = (b + 1 < kSpBins ? excl[b + 1] : start + (u32)n) - e;
    u32         o = (u32)((t - (float)b) * (float)c);
    o             = c > 0 && o >= c ? c - 1u : o;
    const u32 s = (e - start + o) >> 1, last = (u32)(n - 1) >> 1;
    return s < last ? s : last;
}
// the counts of `sub` (two 16-bit ones a word) become first positions
static __device__ __forceinline__ void sp_sub_prefix(u32* sub, int words)
{
    const int wpt = (words + kThreads - 1) / kThreads, w0 = (int)threadIdx.x * wpt, w1 = w0 + wpt < words ? w0 + wpt : words;
    u32       mine = 0, tot;
#pragma unroll 1
    for (int w = w0; w < w1; ++w) {
        mine += (sub[w] & 0xffffu) + (sub[w] >> 16);
    }
    u32 run = block_excl_u32(mine, &tot);
#pragma unroll 1
    for (int w = w0; w < w1; ++w) {
        const u32 c = sub[w];
        sub[w]      = run | ((run + (c & 0xffffu)) << 16);
        run += (c & 0xffffu) + (c >> 16);
    }
    __syncthreads();
}

// n <= 25 * kSpLists
// words behind the counters that sp_sort_keys needs for n keys (two bit maps)
__device__ __forceinline__ int sp_sort_bits(int n)
{
    return 2 * (n / 32 + 2);
}

static __device__ __noinline__ bool sp_sort_keys(float* a, float* tmp, u32* sub, u32* bits, const u32* excl, u32* list, u32 start, int n,
                                                 float maxv, bool ties)
{
    FTB_ASSUME_SHARED(bits);
    FTB_ASSUME_SHARED(a);
    FTB_ASSUME_SHARED(tmp);
    FTB_ASSUME_SHARED(sub);
    FTB_ASSUME_SHARED(excl);
    FTB_ASSUME_SHARED(list);
    __shared__ u32 s_nlong;
    const int      tid = threadIdx.x, lane = tid & 31, words = ((n + 1) / 2 + 1) / 2;
#pragma unroll 1
    for (int i = tid; i < words; i += kThreads) {
        sub[i] = 0;
    }
    u32* const edge = bits;              // a bit where a sub-bucket starts
    u32* const turn = bits + n / 32 + 2;  // a bit where a key differs from the one in front of it
#pragma unroll 1
    for (int i = tid; i < sp_sort_bits(n); i += kThreads) {
        bits[i] = i == 0 ? 1u : 0u;
    }
    if (tid == 0) {
        s_nlong = 0;
    }
    __syncthreads();
    // The 32 lanes of a warp take their keys from 32 places far apart: neighbours lie in the same sub-bucket.
    const int seg = ((n + 31) / 32) | 1;
    // Four keys at a time: their loads and atomics are on their way together.
    constexpr int kAtOnce = 4;
    float         v[kAtOnce];
    u32           s[kAtOnce];
    auto          take = [&](int j) {
        u32 in = 0;
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            const int  p  = lane * seg + j + q * kWarps;
            const bool ok = (j + q * kWarps < seg) & (p < n);
            v[q]          = ok ? a[p] : maxv;
            in |= ok ? 1u << q : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            s[q] = sp_sub_bucket(excl, v[q], maxv, start, n);
        }
        return in;
    };
#pragma unroll 1
    for (int j = tid >> 5; j < seg; j += kAtOnce * kWarps) {
        const u32 in = take(j);
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            if (in >> q & 1u) {
                smem_add(&sub[s[q] >> 1], 1u << (16 * (s[q] & 1u)));
            }
        }
    }
    __syncthreads();
    sp_sub_prefix(sub, words);
#pragma unroll 1
    for (int j = tid >> 5; j < seg; j += kAtOnce * kWarps) {
        const u32 in = take(j);
        u32       old[kAtOnce];
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            old[q] = in >> q & 1u ? atomicAdd(&sub[s[q] >> 1], 1u << (16 * (s[q] & 1u))) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
            if (in >> q & 1u) {
                tmp[(old[q] >> (16 * (s[q] & 1u))) & 0xffffu] = v[q];
            }
        }
    }
    __syncthreads();
    // The counters now hold where their sub-bucket ends.  16-bit logits fill most sub-buckets with equal keys, which stay where
    // they are: two bit maps tell (the place of every key looked for among up to 24: 16.7 us for the slowest row's sort of 48 x
    // 51200 half, 14.8 so).
#pragma unroll 1
    for (int i = tid; i < words; i += kThreads) {
        const u32 c = sub[i], e0 = c & 0xffffu, e1 = c >> 16;
        atomicOr(&edge[e0 >> 5], 1u << (e0 & 31u));
        atomicOr(&edge[e1 >> 5], 1u << (e1 & 31u));
    }
    if (ties) {
#pragma unroll 1
        for (int w = tid >> 5; w * 32 < n; w += kWarps) {
            const int   p = w * 32 + lane;
            const float x = tmp[p < n ? p : n - 1], y = tmp[p == 0 ? 0 : (p < n ? p - 1 : n - 1)];
            const u32   t = __ballot_sync(0xffffffffu, x != y);
            if (lane == 0) {
                turn[w] = t;
            }
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int w = tid >> 5; w * 32 < n; w += kWarps) {
        const int p = w * 32 + lane;
        if (p >= n) {
            break;
        }
        const float x  = tmp[p];
        const u64   up = (2ull << lane) - 1ull, down = (2ull << (32 + lane)) - 1ull;  // bits up to this key, from this word and the one before
        const u32   e0 = w > 0 ? edge[w - 1] : 0u, e1 = edge[w], e2 = edge[w + 1];
        const u32   t0 = w > 0 ? turn[w - 1] : 0u, t1 = turn[w], t2 = turn[w + 1];
        const u64   eb = (((u64)e1 << 32) | e0) & down, ea = (((u64)e2 << 32) | e1) & ~up;
        const u64   tb = (((u64)(t1 | e1) << 32) | (t0 | e0)) & down, ta = (((u64)(t2 | e2) << 32) | (t1 | e1)) & ~up;
        const int   lo = w * 32 + 31 - __clzll((long long)eb), hi = w * 32 - 1 + __ffsll((long long)ea);
        const bool  seen = eb != 0 && ea != 0;  // (both ends within the three words)
        if (seen && (hi - lo == 1
                     || (ties && __clzll((long long)tb) == __clzll((long long)eb) && __ffsll((long long)ta) == __ffsll((long long)ea)))) {
            a[p] = x;
            continue;
        }
        if (!seen || hi - lo > kSpShort) {
            if (e1 >> lane & 1u) {
                int to = w + 1;
                u32 e  = e2;
                if (ea != 0) {
                    to = hi;
                }
                else {
                    while (e == 0) {  // (position n has a bit)
                        e = edge[++to];
                    }
                    to = to * 32 + __ffs(e) - 1;
                }
                list[atomicAdd(&s_nlong, 1u)] = (u32)p | ((u32)(to - p) << 16);  // (at most n / 25 of them)
            }
            continue;
        }
        // the larger ones, and the equal ones in front
        int to = lo;
#pragma unroll 1
        for (int j = lo; j < hi; j += 4) {
            float y[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                y[q] = j + q < hi ? tmp[j + q] : -INFINITY;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                to += (y[q] > x ? 1 : 0) | (y[q] == x && j + q < p ? 1 : 0);
            }
        }
        a[to] = x;
    }
    __syncthreads();
    // A long sub-bucket holds few distinct values (16-bit logits: a run of equal ones, a penalised column's beside it): a warp
    // takes the largest value left, writes it as often as it occurs, and goes on.
    bool ok = true;
#pragma unroll 1
    for (u32 w = (u32)(tid >> 5); w < s_nlong; w += kWarps) {
        const int lo = (int)(list[w] & 0xffffu), m = (int)(list[w] >> 16);
        // (all equal, as a rule)
        const float first = tmp[lo];
        bool        same  = true;
        for (int i = lane; i < m; i += 32) {
            same &= tmp[lo + i] == first;
            a[lo + i] = first;
        }
        if (__all_sync(0xffffffffu, same)) {
            continue;
        }
        __syncwarp();
        u32 below = 0xffffffffu;
        int pos   = 0;
        for (int d = 0; d < 256 && pos < m; ++d) {
            u32 top = 0, c = 0;
            for (int i = lane; i < m; i += 32) {
                const u32 k = fkey(tmp[lo + i]);
                c           = k >= below || k < top ? c : (k > top ? 1u : c + 1u);
                top         = k < below && k > top ? k : top;
            }
            below = __reduce_max_sync(0xffffffffu, top);
            c     = __reduce_add_sync(0xffffffffu, top == below ? c : 0u);
            if (c == 0) {
                break;
            }
            for (int i = lane; i < (int)c; i += 32) {
                a[lo + pos + i] = fkey_inv(below);
            }
            pos += (int)c;
        }
        ok = ok && pos >= m;
    }
    return __syncthreads_and(ok) != 0;
}

// All of an owner's keys: at once while they fill at most half of the area (its other half is tmp), else stretches of whole bins
// one after the other, with tmp in the words behind the counters (`sub` to the end of `hist`).  A bin that is larger than a
// stretch holds few distinct values (16-bit logits); more than 32 of them are given up.
static __device__ __noinline__ bool sp_sort_area(float* a, u32* sub, const u32* excl, u32* hist, u32 start, int n, float maxv, int cap,
                                                 bool ties)
{
    __shared__ u32 s_end, s_top, s_cnt, s_val[32], s_num[32];
    FTB_ASSUME_SHARED(a);
    FTB_ASSUME_SHARED(excl);
    const int  tid = threadIdx.x, lane = tid & 31;
    u32* const list = hist + kSpBins - kSpLists;
    if (n <= cap / 2 && n <= 25 * kSpLists) {
        return sp_sort_keys(a, a + cap / 2, sub, hist, excl, list, start, n, maxv, ties);  // (the maps fit: n / 16 words)
    }
    // (a quarter of a word for the counters, a sixteenth for the maps, one for the key)
    const int most = (cap / 4 + kSpBins - kSpLists - 16) * 16 / 21;
    bool      ok   = true;
    for (int at = 0; at < n;) {
        int cnt = n - at;
        if (cnt > most) {
            // the last bin that starts within the stretch starts the next one
            __syncthreads();
            if (tid == 0) {
                s_end = 0;
                s_cnt = start + (u32)n;
            }
            __syncthreads();
            const u32 first = start + (u32)at;
            u32       last = 0, next = 0xffffffffu;
            for (int b = tid; b < kSpBins; b += kThreads) {
                const u32 e = excl[b];
                last        = e > first && e <= first + (u32)most && e > last ? e : last;
                next        = e > first && e < next ? e : next;
            }
            atomicMax(&s_end, last);
            atomicMin(&s_cnt, next);
            __syncthreads();
            const bool bin_alone = s_end == 0;
            cnt                  = (int)((bin_alone ? s_cnt : s_end) - first);
            if (bin_alone) {
                u32 below = 0xffffffffu;
                int left = cnt, d = 0;
                for (; d < 32 && left > 0; ++d) {
                    __syncthreads();
                    if (tid == 0) {
                        s_top = 0;
                        s_cnt = 0;
                    }
                    __syncthreads();
                    u32 top = 0;
                    for (int i = tid; i < cnt; i += kThreads) {
                        const u32 k = fkey(a[at + i]);
                        top         = k < below && k > top ? k : top;
                    }
                    top = __reduce_max_sync(0xffffffffu, top);
                    if (lane == 0) {
                        atomicMax(&s_top, top);
                    }
                    __syncthreads();
                    below = s_top;
                    u32 c = 0;
                    for (int i = tid; i < cnt; i += kThreads) {
                        c += fkey(a[at + i]) == below ? 1u : 0u;
                    }
                    c = __reduce_add_sync(0xffffffffu, c);
                    if (lane == 0) {
                        atomicAdd(&s_cnt, c);
                    }
                    __syncthreads();
                    if (tid == 0) {
                        s_val[d] = below;
                        s_num[d] = s_cnt;
                    }
                    left = s_cnt != 0 ? left - (int)s_cnt : -1;
                }
                __syncthreads();
                if (left == 0) {
                    for (int q = 0, pos = at; q < d; ++q) {
                        const float v = fkey_inv(s_val[q]);
                        const int   c = (int)s_num[q];
                        for (int i = tid; i < c; i += kThreads) {
                            a[pos + i] = v;
                        }
                        pos += c;
                    }
                }
                ok = ok && left == 0;
                at += cnt;
                continue;
            }
        }
        ok = sp_sort_keys(a + at, (float*)(sub + cnt / 4 + 2 + sp_sort_bits(cnt)), sub, sub + cnt / 4 + 2, excl, list, start + (u32)at, cnt, maxv,
                          ties) && ok;
        at += cnt;
    }
    __syncthreads();
    return ok;
}

// Up to N keys into descending order, in registers (odd-even merge sort).
template<int N>
__device__ __forceinline__ void sp_sort_few(float* k, int m)
{
    float x[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        x[i] = i < m ? k[i] : -INFINITY;
    }
#pragma unroll
    for (int p = 1; p < N; p *= 2) {
#pragma unroll
        for (int q = p; q >= 1; q /= 2) {
#pragma unroll
            for (int j = q % p; j + q < N; j += 2 * q) {
#pragma unroll
                for (int i = 0; i < q; ++i) {
                    if (i + j + q < N && (i + j) / (2 * p) == (i + j + q) / (2 * p)) {
                        const float a = x[i + j], b = x[i + j + q];
                        x[i + j]      = fmaxf(a, b);
                        x[i + j + q]  = fminf(a, b);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (i < m) {
            k[i] = x[i];
        }
    }
}

// bfloat16 values without a bias that fall into bin b, by the distance of its edges in bit patterns; `per_y` raw values make one final one.
__device__ __forceinline__ u32 sp_bf16_patterns(float maxv, int b, float per_y)
{
    return (fkey((maxv - sp_edge(b)) * per_y) >> 16) - (fkey((maxv - sp_edge(b + 1)) * per_y) >> 16);
}

// One nucleus owner's keys (bins b_lo .. b_hi, bin by bin in `a`) into descending order, in place, where a bin holds few values: bfloat16
// logits without a bias, 128 values an octave, and the penalised columns' beside them.  A thread takes a bin of up to eight keys, a
// warp a larger one: most hold one value; up to 32 keys are ordered by counting, more are written value by value, up to 32 of them.
// Nothing is counted, prefixed or moved through a second copy, and a full area goes like a half full one.  Returns false where
// sp_sort_area has to order the keys (the bins may be in any order within).  An owner's 3000 keys, 128256 columns: 11.2 us with
// sp_sort_area, 5.2 so.  fp32 and half rows have too many values in a bin: 11 to 42 us where sp_sort_area takes 7 to 11.
//
// So have bfloat16 rows whose nucleus comes near zero (flat ones): there a bin of more than 32 keys can hold more than kSpFewPatterns
// values, and the owner goes to sp_sort_area before a key has been looked at.  us a step, p 0.95, sp_sort_area always / without this
// test, every bin value by value / with it at 32 / 16 / 8 / 4: 8 x 32000, sigma 1 50.0 / 75.8 / 55.1 / 51.5 / 49.3 / 48.8; 16 x 50264, sigma 1.5
// 53.6 / 73.8 / 54.2 / 52.4 / 51.1 / 51.0; 32 x 128256, sigma 2 121.9 / 104.4 / 103.1 / 102.8 / 104.4 / 107.1, sigma 2.5 71.1 / 64.3 / 64.4 /
// 64.5 / 64.2 / 64.3.
constexpr u32 kSpFewPatterns = 8;
static __device__ __noinline__ bool sp_sort_bins(float* a, const u32* excl, u32 start, int n, int b_lo, int b_hi, float maxv, float per_y)
{
    FTB_ASSUME_SHARED(a);
    FTB_ASSUME_SHARED(excl);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    bool      ok   = true;
#pragma unroll 1
    for (int b = b_lo + (int)threadIdx.x; b <= b_hi; b += kThreads) {
        const u32 c = (b < b_hi ? excl[b + 1] : start + (u32)n) - excl[b];
        ok          = ok && (c <= 32u || sp_bf16_patterns(maxv, b, per_y) <= kSpFewPatterns);
    }
    if (!__syncthreads_and(ok)) {
        return false;
    }
    int       turn = 0;  // larger bins in front, the same in every warp
#pragma unroll 1
    for (int b0 = b_lo; b0 <= b_hi; b0 += 32) {
        const int b  = b0 + lane;
        const int lo = b <= b_hi ? (int)(excl[b] - start) : n, hi = b < b_hi ? (int)(excl[b + 1] - start) : n;
        if ((((b0 - b_lo) >> 5) & (kWarps - 1)) == wid && hi - lo > 1 && hi - lo <= 8) {
            sp_sort_few<8>(a + lo, hi - lo);
        }
        u32 todo = __ballot_sync(0xffffffffu, hi - lo > 8);
#pragma unroll 1
        while (todo != 0) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1;
            if ((turn++ & (kWarps - 1)) != wid) {
                continue;
            }
            const int    at = __shfl_sync(0xffffffffu, lo, q), m = __shfl_sync(0xffffffffu, hi, q) - at;
            float* const k     = a + at;
            const float  first = k[0];
            bool         same  = true;
#pragma unroll 4
            for (int i = lane; i < m; i += 32) {
                same &= k[i] == first;
            }
            if (__all_sync(0xffffffffu, same)) {
                continue;
            }
            if (m <= 32) {
                const u32 mine = lane < m ? fkey(k[lane]) : 0u;
                int       to   = 0;
#pragma unroll 4
                for (int j = 0; j < m; ++j) {
                    const u32 x = __shfl_sync(0xffffffffu, mine, j);
                    to += x > mine || (x == mine && j < lane) ? 1 : 0;
                }
                __syncwarp();
                if (lane < m) {
                    k[to] = fkey_inv(mine);
                }
                continue;
            }
            // each value with its count, the largest first
            float mine  = 0.0f;
            int   times = 0;
            u32   below = 0xffffffffu;
            int   d = 0, pos = 0;
#pragma unroll 1
            for (; d < 32 && pos < m; ++d) {
                u32 top = 0, c = 0;
                for (int i = lane; i < m; i += 32) {
                    const u32 key = fkey(k[i]);
                    c             = key >= below || key < top ? c : (key > top ? 1u : c + 1u);
                    top           = key < below && key > top ? key : top;
                }
                below = __reduce_max_sync(0xffffffffu, top);
                c     = __reduce_add_sync(0xffffffffu, top == below ? c : 0u);
                if (lane == d) {
                    mine  = fkey_inv(below);
                    times = (int)c;
                }
                pos += (int)c;
            }
            if (pos < m) {
                ok = false;
                continue;
            }
            __syncwarp();
            for (int v = 0, to = 0; v < d; ++v) {
                const float x = __shfl_sync(0xffffffffu, mine, v);
                const int   c = __shfl_sync(0xffffffffu, times, v);
                for (int i = lane; i < c; i += 32) {
                    k[to + i] = x;
                }
                to += c;
            }
        }
    }
    return __syncthreads_and(ok) != 0;
}

// Half: first bin whose inclusive count reaches `want` (kSpBins - 1 when the total stays below) with a probability at its far
// edge that cannot round to the one at `p_below`.
static __device__ int sp_bin_below(const u32* excl, u32 total, u32 want, float p_below, float inv_denom)
{
    __shared__ int s_b;
    constexpr int  PER = kSpBins / kThreads;
    const int      tid = threadIdx.x;
    FTB_ASSUME_SHARED(excl);
    if (tid == 0) {
        s_b = kSpBins - 1;
    }
    __syncthreads();
    int found = kSpBins;
#pragma unroll
    for (int i = PER - 1; i >= 0; --i) {
        const int b    = tid * PER + i;
        const u32 incl = b + 1 < kSpBins ? excl[b + 1] : total;
        found          = (incl >= want) & (__expf(-sp_edge(b)) * inv_denom <= p_below) ? b : found;
    }
    if (found < kSpBins) {
        atomicMin(&s_b, found);
    }
    __syncthreads();
    return s_b;
}

// The nucleus scan of the reference (topp_sampling: cub::BlockScan<float, 256> in raking order, 256 sorted
// probabilities per chunk, sampling_topp_kernels.cu:877-1004) over keys that lie in the areas of `owners` CTAs.
struct SpKeys {
    u32 area;            // 32-bit address of the area in this CTA
    int owners;
    u32 start[kSpMaxN + 1];  // first position of every owner, then the total
};
// owner of a position (loads that do not wait for one another: with a search the aggregates of a wide row's chunks took 4.5 us, 2.3
// so)
__device__ __forceinline__ int sp_key_owner(const SpKeys& K, u32 pos)
{
    int o = 0;
#pragma unroll
    for (int q = 1; q < kSpMaxN; ++q) {
        o += pos >= K.start[q] ? 1 : 0;
    }
    return o < K.owners ? o : K.owners - 1;
}
__device__ __forceinline__ float sp_key_at(const SpKeys& K, u32 pos)
{
    const int o = sp_key_owner(K, pos);
    return __uint_as_float(dld_u32(cluster_addr(K.area + 4u * (pos - K.start[o]), (u32)o)));
}
// eight keys of chunk c for this lane; `own`: this CTA's rank (0 where the keys lie in this CTA)
__device__ __forceinline__ void sp_load8(const SpKeys& K, u32 c, int lane, int own, float* x)
{
    const u32 total = K.start[K.owners], p0 = c * 256u + (u32)lane * 8u;
    const int o     = sp_key_owner(K, p0);
    const u32 end   = K.start[o + 1], at = K.area + 4u * (p0 - K.start[o]);
    if (p0 + 8u <= end) {
        if (o == own) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                x[i] = __uint_as_float(lds_u32(at + 4u * (u32)i));
            }
        }
        else {
            const u32 base = cluster_addr(at, (u32)o);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                x[i] = __uint_as_float(dld_u32(base + 4u * (u32)i));
            }
        }
    }
    else {
        u32 from[8];  // (all places first: their loads are on their way together)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const u32 p = p0 + (u32)i < total ? p0 + (u32)i : total - 1u;
            const int q = sp_key_owner(K, p);
            from[i]     = cluster_addr(K.area + 4u * (p - K.start[q]), (u32)q);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float y = __uint_as_float(dld_u32(from[i]));
            x[i]          = p0 + (u32)i < total ? y : 0.0f;
        }
    }
}
// inclusive sum of the lane's eight values and the Kogge-Stone scan of the lane totals
__device__ __forceinline__ float sp_rake(const float* x, int lane)
{
    float up = x[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        up = up + x[i];
    }
    float inc = up;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) {
            inc = inc + t;
        }
    }
    return inc;
}

// Warp 0 of the leader: running prefix over the chunk aggregates (`agg` 16-byte aligned, readable up to a multiple of eight),
// the crossing inside its chunk and the crossing's probability.  Returns the verdict (see SpShared).
static __device__ __noinline__ u32 sp_find_crossing(const SpKeys& K, const float* agg, float rand_num, bool complete, int own, u32* p_out,
                                                    u32* sel_out)
{
    FTB_ASSUME_SHARED(agg);
    const int lane = threadIdx.x & 31;
    const u32 N    = K.start[K.owners];
    const int nch  = (int)((N + 255u) / 256u);
    // chunk by chunk, as the reference's prefix functor accumulates; stopped a little early (inside a chunk the partial
    // sums differ from prefix + aggregate in the last bits only)
    float     R  = 0.0f;
    const int c1 = running_prefix(agg, nch, rand_num * (1.0f - 1e-4f), R);
    int sel = -1;
    for (int c = c1; c < nch; ++c) {
        float x[8];
        sp_load8(K, (u32)c, lane, own, x);
        const float inc = sp_rake(x, lane);
        const float ag  = __shfl_sync(0xffffffffu, inc, 31);
        const float ex  = __shfl_up_sync(0xffffffffu, inc, 1);
        float       o   = lane == 0 ? R : R + ex;
        u32         cnt = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            o = o + x[i];
            cnt += rand_num <= o ? 1u : 0u;
        }
        // a warp of the reference covers 4 of these lanes (32 consecutive probabilities)
        u32 c4 = cnt;
        c4 += __shfl_xor_sync(0xffffffffu, c4, 1);
        c4 += __shfl_xor_sync(0xffffffffu, c4, 2);
        const u32 any = __ballot_sync(0xffffffffu, c4 > 0);
        if (any) {
            const int g  = (__ffs(any) - 1) >> 2;
            const u32 pc = __shfl_sync(0xffffffffu, c4, g * 4);
            sel          = c * 256 + g * 32 + (32 - (int)pc);
            if (!complete && (u32)(c * 256 + g * 32 + 31) >= N) {
                return 2;  // the 32 probabilities of that warp are not all known
            }
            break;
        }
        R = R + ag;
    }
    if (sel < 0 || (u32)sel >= N) {
        if (!complete || N == 0) {
            return 2;
        }
        // the cumulative sum never reached the draw: the reference leaves the best token in place
        *p_out   = __float_as_uint(sp_key_at(K, 0));
        *sel_out = 0;
        return 1;
    }
    const float p = sp_key_at(K, (u32)sel), last = complete ? 0.0f : sp_key_at(K, N - 1);
    if (!complete && p == last) {
        return 2;  // the lowest class may have members that were not collected
    }
    *p_out   = __float_as_uint(p);
    *sel_out = (u32)sel;
    return 0;
}

// Note of why a row is left to decode_sampling_kernel (word 25 of its trace record).
__device__ __forceinline__ bool sp_leave(const RowOut& O, int why)
{
    if (O.trace != nullptr && threadIdx.x == 0) {
        O.trace[4 + 25] = (u64)why;
    }
    return false;
}

// Result of a top-p row (one thread).
template<int DT>
__device__ __forceinline__ void sp_write_topp(const KParams& P, const RowOut& O, int id, float prob, bool drawn, bool want_lp)
{
    *O.id_out = id;
    if (drawn) {
        if (want_lp) {
            const float lprob = logf(prob);
            if (P.cum_log_probs != nullptr) {
                P.cum_log_probs[O.r] = __fadd_rn(P.cum_log_probs[O.r], lprob);
            }
            if (P.out_log_probs != nullptr) {
                P.out_log_probs[O.r] = lprob;
            }
        }
        write_lengths(P, O, id);
    }
}

__device__ __forceinline__ SpMap sp_map(const SplitArgs& A, unsigned char* smem)
{
    SpMap M;
    M.y        = (float*)smem;
    M.area     = (u32*)(M.y + A.slice);
    M.area_cap = A.area;
    M.merged   = M.area + A.area;
    M.sub      = M.merged + kSpBins;
    M.hist     = M.sub + A.area / 4;
    return M;
}

// One row on the cluster.  Every branch that skips a cluster barrier depends on values that all CTAs hold alike.
// Returns (leader only) whether the row is decided.
template<int DT, int LGN>
__device__ __forceinline__ bool sp_row(const KParams& P, const SplitArgs& A, unsigned char* smem, SpShared& X, const RowOut& O, int mode,
                                    bool want_lp)
{
    FTB_ASSUME_SHARED(smem);
    const SpMap      M = sp_map(A, smem);
    __shared__ float s_u, s_denom;
    const int        tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int    n = 1 << LGN, lgvt = 10 - LGN;
    const int        rank = (int)cluster_rank(), r = O.r;
    const int        nchunk = (P.vocab + 1023) >> 10, ny = nchunk << lgvt;
    float* const     y = M.y;
    const bool       specials = P.apply_rep || P.bad_words != nullptr || P.apply_minlen;
    const bool       softmax  = mode == 2 || want_lp;
    const float      neg_max  = DT == FTB200_F16 ? -65504.0f : -FLT_MAX;
    const float      lowest   = __uint_as_float(__float_as_uint(neg_max) - 1u);  // smallest value above neg_max
    FTB_ASSUME_SHARED(y);

    // ---- set-up: counters, the row's slice, special columns ----
    const int words = ny >> 5;
    u32*      bits  = M.area;  // [2][words] bit maps of the special columns
    for (int i = tid; i < kSpBins; i += kThreads) {
        M.hist[i] = 0;
    }
    if (specials) {
        for (int i = tid; i < 2 * words; i += kThreads) {
            bits[i] = 0;
        }
    }
    if (tid == 0) {
        X.first_max = 0xffffffffu;
        X.n_cls     = 0;
        X.larger    = 0;
        X.bad_order = 0;
        X.max_key   = 0;
    }
    __syncthreads();
    cluster_arrive();  // this CTA's counters may be written by the others
    // the row's arguments, sent for before the row so that nobody waits for them
    const u32     k_row = mode == 1 ? P.topk_ks[r] : 0u;
    const float   p_row = mode == 1 ? P.topk_ps[r] : P.topp_ps[r];
    curandState_t draw;
    if (tid == 0) {
        draw = (mode == 1 ? P.topk_states : P.topp_states)[r];
    }
    Xf X0;
    X0.bias       = P.bias;
    X0.apply_temp = P.apply_temp;
    X0.inv_t      = P.apply_temp ? 1.0f / (P.temperature[r] + 1e-6f) : 1.0f;
    X0.inv_t_h    = __float2half_rn(X0.inv_t);
    X0.theta      = P.apply_rep ? P.rep_penalty[r] : 1.0f;
    X0.apply_rep = P.apply_rep, X0.penalty_type = P.penalty_type;
    X0.vocab     = P.vocab;
    const char* rowp = (const char*)P.logits + (size_t)r * P.vocab_padded * (DT == FTB200_F32 ? 4 : 2);
    int         hist0 = -1, hist1 = -1;
    if (P.apply_rep) {
        const size_t col       = (size_t)P.ite * P.local_batch + r;
        const int    input_len = P.input_lengths != nullptr ? P.input_lengths[r] : P.max_input_len;
        hist0                  = sp_history_id(P, col, input_len, rank * kThreads + tid);
        hist1                  = sp_history_id(P, col, input_len, (n + rank) * kThreads + tid);
    }
    float best = sp_load_slice<DT>(P, X0, rowp, y, rank, lgvt, nchunk);
    if (tid == 0) {
        s_u        = curand_uniform(&draw);
        X.per_y    = P.apply_temp ? P.temperature[r] + 1e-6f : 1.0f;
        X.state[0] = draw.d;  // (stored with the result)
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            X.state[1 + i] = draw.v[i];
        }
    }
    trace_mark(O.trace, 0);
    cluster_wait();
    if (specials) {
        sp_mark_specials<LGN>(P, r, smem_addr(bits), words, rank, hist0, hist1);
        cluster_sync();
        for (int w = tid; w < words; w += kThreads) {
            const u32 dead = bits[words + w];
            u32       any  = bits[w] | dead;
            while (any != 0) {
                const int b = __ffs(any) - 1;
                any &= any - 1;
                const int i = w * 32 + b;
                y[i]        = special_value<DT>(X0, y[i], (dead >> b) & 1u ? kFlagDead : kFlagHist);
            }
        }
    }
    __syncthreads();

    // ---- row maximum ----
    trace_mark(O.trace, 1);
    const bool arg_max = mode == 1 && !want_lp && k_row <= 1u;
    if (specials || arg_max) {
        // (some values have changed since they came in; an arg-max row wants the maximum of what each warp walks over below)
        best = -INFINITY;
        for (int i = 4 * tid; i < ny; i += 4 * kThreads) {
            const float4 v = *(const float4*)(y + i);
            best           = fmaxf(best, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
        }
    }
    const u32 warp_key = __reduce_max_sync(0xffffffffu, best > neg_max ? fkey(best) : 0u);
    if (arg_max) {
        // ---- arg-max: value, then the reference's tie order (CTA lane and thread descending, column ascending).  Every warp
        // looks for its own maximum's columns, so that one exchange brings the value and the tie together ----
        const u32 bs1 = P.max_top_k <= 16 ? 128 : 256;
        const int sh1 = bs1 == 128 ? 7 : 8;
        u32       tie = 0;
        if (warp_key != 0) {
            sp_sweep(y, ny, fkey_inv(warp_key), [&](int i, float x) {
                if (fkey(x) != warp_key) {
                    return;  // (a zero of the other sign)
                }
                const u32 v = (u32)(((i >> lgvt) << 10) | (rank << lgvt) | (i & ((1 << lgvt) - 1)));
                const u32 c = (((v >> sh1) & 7u) << 29) | ((v & (bs1 - 1)) << 21) | (0x1fffffu - v);
                tie         = c > tie ? c : tie;
            });
            tie = __reduce_max_sync(0xffffffffu, tie);
        }
        if (lane == 0) {
            dst_u64(cluster_addr(smem_addr(&X.best[rank * kWarps + wid]), 0), ((u64)warp_key << 32) | tie);
        }
        cluster_sync();
        trace_mark(O.trace, 2);
        if (rank != 0) {
            return true;
        }
        u64 b = 0;
        for (int i = lane; i < n * kWarps; i += 32) {
            const u64 w = X.best[i];
            b           = w > b ? w : b;
        }
        b = warp_max_u64(b);
        if (b != 0 && !(fkey_inv((u32)(b >> 32)) < INFINITY)) {
            return sp_leave(O, 1);
        }
        if (tid == 0) {
            // (nothing can be selected: token 0)
            const int id = b != 0 ? (int)(0x1fffffu - ((u32)b & 0x1fffffu)) : 0;
            *O.id_out    = id;
            write_lengths(P, O, id);
        }
        return true;
    }
    if (lane < n) {
        dred_max(cluster_addr(smem_addr(&X.max_key), (u32)lane), warp_key);
    }
    cluster_sync();
    const u32 kmax = X.max_key;
    trace_mark(O.trace, 2);
    const float u = s_u;
    if (kmax == 0) {
        // nothing can be selected: token 0
        if (rank == 0 && tid == 0) {
            *O.id_out = 0;
            write_lengths(P, O, 0);
        }
        return true;
    }
    const float maxv = fkey_inv(kmax);
    if (!(maxv < INFINITY)) {
        return sp_leave(O, 1);
    }

    // ---- counts per bin; for a soft-max row the ordered denominator ----
    sp_count_bins(y, ny, lowest, maxv, smem_addr(M.hist));
    trace_mark(O.trace, 3);
    if (softmax) {
        sp_chain_sums<DT, LGN>(y, nchunk, maxv, smem_addr(X.wsum), rank);
    }
    trace_mark(O.trace, 4);
    cluster_sync();
    trace_mark(O.trace, 16);
    {
        // this CTA adds its share of the bins over the cluster and hands the sums to everybody
        constexpr int share = kSpBins >> LGN;
        for (int i = tid; i < share; i += kThreads) {
            const int b = rank * share + i;
            const u32 a = smem_addr(&M.hist[b]), m = smem_addr(&M.merged[b]);
            u32       part[n], sum = 0;
#pragma unroll
            for (int q = 0; q < n; ++q) {
                part[q] = dld_u32(cluster_addr(a, (u32)q));
            }
#pragma unroll
            for (int q = 0; q < n; ++q) {
                // (what is selected is placed by bin: what the CTAs before this one have of the bin goes where its count stood)
                dst_u32(cluster_addr(a, (u32)q), sum);
                sum += part[q];
            }
#pragma unroll
            for (int q = 0; q < n; ++q) {
                dst_u32(cluster_addr(m, (u32)q), sum);
            }
        }
        if (softmax && wid == 0) {
            float v = X.wsum[lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v = v + __shfl_xor_sync(0xffffffffu, v, o);
            }
            if (lane == 0) {
                s_denom = v + 1e-6f;
            }
        }
    }
    cluster_sync();
    const float denom = softmax ? s_denom : 1.0f;
    trace_mark(O.trace, 5);
    if (softmax && !(denom > 0.0f && denom < INFINITY)) {
        return sp_leave(O, 2);
    }
    u32* const excl = M.merged;
    if (mode == 2) {
        const float p_max = round_to_T<DT>(round_to_T<DT>(1.0f) / denom);
        if (p_max >= p_row) {
            // arg-max shortcut of topp_beam_topk_kernel (sampling_topp_kernels.cu:801-860): first column of the maximum
            u32 col = 0xffffffffu;
            sp_sweep(y, ny, maxv, [&](int i, float v) {
                if (v == maxv) {
                    const u32 c = (u32)(((i >> lgvt) << 10) | (rank << lgvt) | (i & ((1 << lgvt) - 1)));
                    col         = c < col ? c : col;
                }
            });
            if (col != 0xffffffffu) {
                dred_min(cluster_addr(smem_addr(&X.first_max), 0), col);
            }
            cluster_sync();
            if (rank == 0 && tid == 0) {
                sp_write_topp<DT>(P, O, (int)X.first_max, p_max, true, want_lp);
            }
            return true;
        }
    }

    // ---- first position of every bin in the row's order, and how far down the selection can reach: every column of bins
    // 0 .. b_thr takes part.  A thread holds eight bins: who holds the wanted one says so, and nobody else looks ----
    constexpr int    PER      = kSpBins / kThreads;
    const int        k        = mode == 1 ? ((int)k_row < 1 ? 1 : ((int)k_row > kMaxTopK ? kMaxTopK : (int)k_row)) : 1;
    const float      rand_num = mode == 2 ? u * p_row : 0.0f;
    __shared__ uint4 s_wcnt[kWarps / 4];
    __shared__ float4 s_wmass[kWarps / 4];
    __shared__ u32   s_cutbin, s_thr;
    u32              total, run, mine = 0, c[PER];
    {
        const uint4 m0 = ((const uint4*)M.merged)[2 * tid], m1 = ((const uint4*)M.merged)[2 * tid + 1];
        c[0] = m0.x, c[1] = m0.y, c[2] = m0.z, c[3] = m0.w, c[4] = m1.x, c[5] = m1.y, c[6] = m1.z, c[7] = m1.w;
        float mass = 0.0f;  // lower bound of this thread's bins' probability (top-p rows)
        if (mode == 2) {
            const float scale = 0.99f / denom;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int b = tid * PER + i;
                if (c[i] != 0 && b + 1 < kSpBins) {
                    mass += (float)c[i] * __expf(-sp_edge(b + 1)) * scale;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            mine += c[i];
        }
        u32   incl  = mine;
        float mincl = mass;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const u32   t = __shfl_up_sync(0xffffffffu, incl, off);
            const float f = __shfl_up_sync(0xffffffffu, mincl, off);
            incl += lane >= off ? t : 0u;
            mincl += lane >= off ? f : 0.0f;
        }
        if (lane == 31) {
            ((u32*)s_wcnt)[wid]    = incl;
            ((float*)s_wmass)[wid] = mincl;
        }
        if (tid == 0) {
            s_cutbin = kSpBins - 1;
            s_thr    = kSpBins - 1;
        }
        __syncthreads();
        u32   base = 0;
        float mbase = 0.0f;
        total       = 0;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) {
            const u32 w = ((const u32*)s_wcnt)[i];
            base += i < wid ? w : 0u;
            total += w;
            mbase += i < wid ? ((const float*)s_wmass)[i] : 0.0f;
        }
        run = base + incl - mine;
        uint4 e0, e1;
        e0.x = run, e0.y = e0.x + c[0], e0.z = e0.y + c[1], e0.w = e0.z + c[2];
        e1.x = e0.w + c[3], e1.y = e1.x + c[4], e1.z = e1.y + c[5], e1.w = e1.z + c[6];
        ((uint4*)M.merged)[2 * tid]     = e0;
        ((uint4*)M.merged)[2 * tid + 1] = e1;
        if (mode == 2 && mbase + mincl >= rand_num) {
            // first bins down to which the lower bound of the mass covers the draw (the bin inside the thread's eight is not
            // looked for: the last of them is taken)
            atomicMin(&s_cutbin, (u32)(tid * PER + PER - 1));
        }
    }
    // the bin whose inclusive count reaches `want` first
    auto reaching = [&](u32 want) {
        if (run < want && run + mine >= want) {
            u32 r = run;
            int b = tid * PER;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                r += c[i];
                b += r < want ? 1 : 0;
            }
            s_thr = (u32)b;
        }
    };
    if (mode == 1) {
        reaching((u32)k);
    }
    __syncthreads();
    trace_mark(O.trace, 6);
    int b_thr;
    if (mode == 1) {
        b_thr = (int)s_thr;
        if (want_lp) {
            // equal probabilities may lie in different bins: a few more columns, so that the k-th is not in the last class
            const u32 incl = b_thr + 1 < kSpBins ? excl[b_thr + 1] : total;
            __syncthreads();
            if (tid == 0) {
                s_thr = kSpBins - 1;
            }
            __syncthreads();
            reaching(incl + 32u);
            __syncthreads();
            b_thr = (int)s_thr;
        }
    }
    else {
        const int b_star = (int)s_cutbin;
        // at least 64 columns more: the scan reads 32 entries past the crossing, and the crossing must not fall into
        // the lowest collected class; half-precision probabilities are equal over several bins
        const u32 have = b_star + 1 < kSpBins ? excl[b_star + 1] : total;
        if (DT == FTB200_F16) {
            const float p_at = __expf(-sp_edge(b_star + 1)) / denom;
            b_thr            = sp_bin_below(excl, total, have + 64u, p_at * (1.0f - 1.0f / 512.0f) - 1.3e-7f, 1.0f / denom);
        }
        else {
            reaching(have + 64u);
            __syncthreads();
            b_thr = (int)s_thr;
        }
    }
    const bool complete = b_thr == kSpBins - 1;
    const u32  N        = complete ? total : excl[b_thr + 1];
    trace_mark(O.trace, 9);

    if (N <= (u32)kSpCandCap) {
        // ---- few candidates: the leader gets them all, bin by bin, and finishes the row alone ----
        {
            const u32 base = cluster_addr(smem_addr(M.area), 0);
            u32       e    = run;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                // the place of this CTA's first entry of a bin
                const int b = tid * PER + i;
                if (b <= b_thr) {
                    M.hist[b] = base + 8u * (e + M.hist[b]);
                }
                e += c[i];
            }
        }
        __syncthreads();
        const float thr = fmaxf(sp_floor_value(maxv, b_thr), lowest);
        sp_sweep(y, ny, thr, [&](int i, float v) {
            const int b = sp_bin(maxv - v);
            if (b <= b_thr) {
                const u32 col = (u32)(((i >> lgvt) << 10) | (rank << lgvt) | (i & ((1 << lgvt) - 1)));
                dst_u64(atomicAdd(&M.hist[b], 8u), ((u64)(~fkey(v)) << 32) | col);
            }
        });
        cluster_sync();
        trace_mark(O.trace, 7);
        if (rank != 0) {
            return true;
        }
        // An entry's place inside its bin is the number of smaller ones there, a handful unless many columns are equal.  (The
        // leader's slice has been read for the last time: the sorted list goes there, and the draw's scratch where the
        // entries came in.)
        const int n_cand = (int)N;
        auto      key_of = [&](u64 e) { return fkey_inv(~(u32)(e >> 32)); };
        u64*      sorted = (u64*)M.y;
        {
            const u64* in = (const u64*)M.area;
            FTB_ASSUME_SHARED(in);
#pragma unroll 1
            for (int i = tid; i < n_cand; i += kThreads) {
                const u64 e  = in[i];
                const int b  = sp_bin(maxv - key_of(e));
                const int lo = (int)excl[b], hi = b + 1 < kSpBins ? (int)excl[b + 1] : n_cand;
                int       rk = lo;
                int       j  = lo;
#pragma unroll 1
                for (; j + 4 <= hi; j += 4) {
                    u64 o[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        o[q] = in[j + q];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        rk += o[q] < e ? 1 : 0;
                    }
                }
#pragma unroll 1
                for (; j < hi; ++j) {
                    rk += in[j] < e ? 1 : 0;
                }
                sorted[rk] = e;
            }
            __syncthreads();
        }
        trace_mark(O.trace, 8);
        __shared__ Smem s_S;
        const Smem&     S = s_S;
        if (tid == 0) {
            s_S.cand = (u64*)M.area;
            s_S.hist = M.area;
            s_S.val2 = (float*)(M.area + kNB);
        }
        __syncthreads();
        if (!softmax) {
            return topk_finish(P, S, O, sorted, n_cand, k, u, p_row, true, false);
        }
        // values -> probabilities; their order has to be that of the values
        float* const pr  = (float*)M.merged;
        bool         bad = false;
        for (int i = tid; i < n_cand; i += kThreads) {
            const u64   e = sorted[i];
            const float q = sp_prob<DT>(key_of(e), maxv, denom);
            pr[i]         = q;
            sorted[i]     = ((u64)(~fkey(q)) << 32) | (u32)e;
        }
        __syncthreads();
        for (int i = tid; i + 1 < n_cand; i += kThreads) {
            bad |= pr[i] < pr[i + 1];
        }
        if (__syncthreads_or(bad)) {
            return sp_leave(O, 3);
        }
        if (mode == 1) {
            return topk_finish(P, S, O, sorted, n_cand, k, u, p_row, false, true, !complete);
        }
        __shared__ SpKeys s_K1;
        __shared__ u32    s_res[3];
        if (tid == 0) {
            s_K1.area   = smem_addr(pr);
            s_K1.owners = 1;
        }
        if (tid <= kSpMaxN) {
            s_K1.start[tid] = tid == 0 ? 0u : N;
        }
        __syncthreads();
        for (int c = wid; c * 256 < n_cand; c += kWarps) {
            float x[8];
            sp_load8(s_K1, (u32)c, lane, 0, x);
            const float inc = sp_rake(x, lane);
            if (lane == 31) {
                X.agg[c] = inc;
            }
        }
        __syncthreads();
        if (wid == 0) {
            u32       p = 0, j = 0;
            const u32 v = sp_find_crossing(s_K1, X.agg, rand_num, complete, 0, &p, &j);
            if (lane == 0) {
                s_res[0] = v, s_res[1] = p, s_res[2] = j;
            }
        }
        __syncthreads();
        trace_mark(O.trace, 14);
        if (s_res[0] == 2) {
            return sp_leave(O, 4);
        }
        // equal probabilities stand in column order in the reference's stable sort
        const float p_sel = __uint_as_float(s_res[1]);
        const u32   key   = ~fkey(p_sel);
        for (int i = tid; i < n_cand; i += kThreads) {
            const u64 e = sorted[i];
            if ((u32)(e >> 32) != key) {
                continue;
            }
            u32 rk = 0;
            int j  = i;
            while (j > 0 && (u32)(sorted[j - 1] >> 32) == key) {
                --j;
                rk += sorted[j] < e ? 1u : 0u;
            }
            rk += (u32)j;  // (those of a larger probability)
            for (j = i + 1; j < n_cand && (u32)(sorted[j] >> 32) == key; ++j) {
                rk += sorted[j] < e ? 1u : 0u;
            }
            if (rk == s_res[2]) {
                sp_write_topp<DT>(P, O, (int)(u32)e, p_sel, s_res[0] == 0, want_lp);
            }
        }
        return true;
    }
    if (mode == 1) {
        return sp_leave(O, 5);
    }

    // ---- a large nucleus: sorted by several CTAs ----
    int owners = (int)((N + 1023u) / 1024u);
    owners     = owners < 1 ? 1 : (owners > n ? n : owners);
    __shared__ SpKeys s_K;
    __shared__ int    s_blo, s_bhi;  // this owner's bins
    const SpKeys&     K = s_K;
    if (tid == 0) {
        s_K.area   = smem_addr(M.area);
        s_K.owners = owners;
        s_blo      = kSpBins;
        s_bhi      = -1;
    }
    if (tid <= kSpMaxN) {
        s_K.start[tid] = tid == 0 ? 0u : N;
    }
    __syncthreads();
    // The owner of a bin follows from its first position (any rule will do that rises with it and is the same in all CTAs).
    const float per_key  = (float)owners / (float)N;
    auto        owner_of = [&](u32 e) {
        const int o = (int)((float)e * per_key);
        return o < owners ? o : owners - 1;
    };
    u32 owner_bits = 0;  // of this thread's bins, four bits each
    {
        u32 e = run;
        int before = tid == 0 ? 0 : owner_of(excl[tid * PER - 1]);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            // the first bin of an owner: where its keys start in the row's order
            const int o = tid * PER + i <= b_thr ? owner_of(e) : before;
            for (int q = before + 1; q <= o; ++q) {
                s_K.start[q] = e;
            }
            owner_bits |= (u32)o << (4 * i);
            before = o;
            e += c[i];
        }
        if (DT == FTB200_BF16) {
            int b_lo = kSpBins, b_hi = -1;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int b = tid * PER + i;
                if (b <= b_thr && c[i] != 0 && (int)((owner_bits >> (4 * i)) & 15u) == rank) {
                    b_lo = b < b_lo ? b : b_lo;
                    b_hi = b;
                }
            }
            b_lo = __reduce_min_sync(0xffffffffu, b_lo);
            b_hi = __reduce_max_sync(0xffffffffu, b_hi);
            if (lane == 0 && b_hi >= 0) {
                atomicMin(&s_blo, b_lo);
                atomicMax(&s_bhi, b_hi);
            }
        }
    }
    __syncthreads();
    const bool fits = N > 0 && __syncthreads_and(tid >= kSpMaxN || s_K.start[tid + 1] - s_K.start[tid] <= (u32)M.area_cap - 64u);
    if (!fits) {
        return sp_leave(O, 6);
    }
    trace_mark(O.trace, 10);
    // per bin the place of this CTA's first key of it: the bin's in its owner's area, after the keys of the CTAs before
    {
        u32 e = run;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int b = tid * PER + i, o = (int)((owner_bits >> (4 * i)) & 15u);
            if (b <= b_thr) {
                M.hist[b] = cluster_addr(K.area + 4u * (e - s_K.start[o] + M.hist[b]), (u32)o);
            }
            e += c[i];
        }
    }
    __syncthreads();
    sp_scatter_keys(y, ny, lowest, maxv, (u32)b_thr, smem_addr(M.hist));
    cluster_sync();
    trace_mark(O.trace, 11);
    if (rank < owners) {
        float* const a   = (float*)M.area;
        const int    cnt = (int)(K.start[rank + 1] - K.start[rank]);
        bool         bad = !(DT == FTB200_BF16 && P.bias == nullptr && sp_sort_bins(a, excl, K.start[rank], cnt, s_blo, s_bhi, maxv, X.per_y))
                   && !sp_sort_area(a, M.sub, excl, M.hist, K.start[rank], cnt, maxv, M.area_cap, DT != FTB200_F32);
#pragma unroll 4
        for (int i = tid; i < cnt; i += kThreads) {
            a[i] = sp_prob<DT>(a[i], maxv, denom);
        }
        __syncthreads();
        // the exponential has to be monotone over the keys for their order to be the sorted order
        for (int i = tid; i + 1 < cnt; i += kThreads) {
            bad |= a[i] < a[i + 1];
        }
        if (__syncthreads_or(bad) && tid == 0) {
            dst_u32(cluster_addr(smem_addr(&X.bad_order), 0), 1u);
        }
    }
    if (owners > 1) {
        cluster_sync();
        if (rank > 0 && rank < owners && tid == 0 && K.start[rank + 1] > K.start[rank]
            && sp_key_at(K, K.start[rank] - 1u) < ((const float*)M.area)[0]) {
            dst_u32(cluster_addr(smem_addr(&X.bad_order), 0), 1u);
        }
    }
    trace_mark(O.trace, 12);
    if (rank < owners) {
        // aggregates of the chunks that start in this owner's range
        const u32 c0 = (K.start[rank] + 255u) >> 8, c1 = (K.start[rank + 1] + 255u) >> 8;
        for (u32 c = c0 + (u32)wid; c < c1; c += kWarps) {
            float x[8];
            sp_load8(K, c, lane, rank, x);
            const float inc = sp_rake(x, lane);
            if (lane == 31) {
                dst_u32(cluster_addr(smem_addr(&X.agg[c]), 0), __float_as_uint(inc));
            }
        }
    }
    if (owners > 1) {
        cluster_sync();
    }
    else {
        __syncthreads();
    }
    trace_mark(O.trace, 13);
    if (rank == 0 && wid == 0) {
        u32 p = 0, j = 0, verdict = 2;
        if (!X.bad_order) {
            verdict = sp_find_crossing(K, X.agg, rand_num, complete, 0, &p, &j);
        }
        if (lane < n) {
            const u32 q = (u32)lane;
            dst_u32(cluster_addr(smem_addr(&X.verdict), q), verdict);
            dst_u32(cluster_addr(smem_addr(&X.p_sel), q), p);
            dst_u32(cluster_addr(smem_addr(&X.j_sel), q), j);
        }
    }
    cluster_sync();
    const u32 verdict = X.verdict;
    trace_mark(O.trace, 14);
    if (verdict == 2) {
        return sp_leave(O, 7);
    }
    // ---- columns whose probability is that of the crossing; the one of its rank is the id ----
    const float p_sel = __uint_as_float(X.p_sel);
    // (no column outside [y_lo, y_hi] has that probability: rounding of the exponential, the quotient and the logarithm,
    // in half also of the two stored results, are allowed for)
    const float slack = DT == FTB200_F16 ? 1.0f / 256.0f : 1e-4f, tiny = DT == FTB200_F16 ? 1.3e-7f * (1.0f + denom) : 0.0f;
    const float e_sel = p_sel * denom, e_lo = e_sel * (1.0f - slack) - tiny, pad = 1e-4f + 2e-6f * fabsf(maxv);
    const float y_lo  = e_lo > 1e-37f ? maxv + __logf(e_lo) * 1.00001f - pad : -INFINITY;
    const float y_hi  = maxv + __logf(fmaxf(e_sel * (1.0f + slack) + tiny, 1e-37f)) * 0.99999f + pad;
    const u32 larger = sp_sweep_band(y, ny, fmaxf(y_lo, lowest), y_hi, [&](int i, float v) {
        const float p = sp_prob<DT>(v, maxv, denom);
        if (p == p_sel) {
            const u32 pos = datom_add(cluster_addr(smem_addr(&X.n_cls), 0), 1u);
            if (pos < (u32)M.area_cap) {
                dst_u32(cluster_addr(K.area + 4u * pos, 0), (u32)(((i >> lgvt) << 10) | (rank << lgvt) | (i & ((1 << lgvt) - 1))));
            }
        }
        return p > p_sel ? 1u : 0u;
    });
    {
        // columns of a larger probability: the class's first position in the sorted order
        const u32 w = __reduce_add_sync(0xffffffffu, larger);
        if (lane == 0 && w != 0) {
            dred_add(cluster_addr(smem_addr(&X.larger), 0), w);
        }
    }
    cluster_sync();
    if (rank != 0) {
        return true;
    }
    const u32 n_cls = X.n_cls, j_sel = X.j_sel - X.larger;
    trace_mark(O.trace, 15);
    if (n_cls > (u32)M.area_cap || j_sel >= n_cls) {
        return sp_leave(O, 8);
    }
    const int id = n_cls <= 512 ? sp_jth_of_few(M.area, (int)n_cls, (int)j_sel) :
                                  select_jth_column(M.area, (int)n_cls, (int)j_sel, (u32*)M.y, P.vocab_padded);
    if (tid == 0) {
        sp_write_topp<DT>(P, O, id, p_sel, verdict == 0, want_lp);
    }
    return true;
}

// The step's stop criteria (stop words of row r, then - by the last row of the call - the length limit and the count of
// finished rows over the batch), by the CTA that finished row r.  Same results as stop_criteria_kernel.  With rows left to
// another launch (their flags are set) nothing is counted: the host is told, and sends that launch and the criteria.
static __device__ __noinline__ void sp_stop_criteria(const KParams& P, const StopArgs& T, int r, const int* flags, bool decided)
{
    const int tid = threadIdx.x;
    __syncthreads();
    if (T.stop_words != nullptr && decided) {
        row_stop_words(P, T.stop_words, T.stop_words_len, T.finished, r);
    }
    if (T.limit == nullptr) {
        return;
    }
    if (!arrived_last(T.arrived, (u32)P.local_batch)) {
        return;
    }
    if (tid == 0) {
        *T.arrived = 0;
    }
    count_finished(P, T, flags, false);
}

// ROOMY: 128 registers, two CTAs on an SM, and - when asked to - the step's stop criteria: one launch per decode step.
// Taken while all rows are resident at once, and beyond that where shared memory holds no third CTA on an SM; elsewhere 80
// registers and three CTAs on an SM are worth more (choose_split).  Either form flags the rows that its tables cannot hold for a second launch: decode_sampling_kernel, or - where the areas of the first
// launch are small - a few clusters of the roomy form with all the shared memory there is (A.clusters), because a nucleus of half
// of 127000 columns takes 0.2 ms here and 5 to 9 ms in the general code.  Those areas hold 16384 keys a CTA, all of 128000 columns, and
// 60 % of 200000; what is wider still ends in the general code, so a batch of such rows takes what its widest nucleus takes.  Mean of
// steps of fresh normal logits with areas of 10240 keys / so, ms: 100 x 127000 bf16 with log-probabilities 0.29 / 0.30 (sigma 2, p
// 0.95, temperature 1.2), 7.9 / 0.42 (sigma 1.5), 11.5 / 0.67 (sigma 0.8, p 0.98, temperature 1.1); 800 x 126959 (sigma 1.5) 14.1 /
// 2.7; 60 x 200000 fp32 8.5 / 0.30 (sigma 2), 13.4 / 11.2 (sigma 1.5); 20 x 60000 fp32 (sigma 0.8) 1.38 / 0.15.
//
// The general row code is not part of this kernel.  It was, in the roomy form, for the rows it leaves; its frames brought the
// stack to 1.7 to 1.9 KB a thread, and builds that differed in nothing but such sizes ended steps of two CTAs on an SM with an
// illegal address, or did not.  The cause is not known: its index arithmetic, the sizes of its tables and the pointers it
// takes for shared have been read through since and stay inside.  Without it the stack is 16 bytes, 152 in the other form.
template<int DT, int LGN, bool ROOMY>
__global__ void __launch_bounds__(kThreads, ROOMY ? 2 : 3) split_sampling_kernel(const __grid_constant__ KParams P,
                                                                     const __grid_constant__ SplitArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SpShared                           s_X;
    __shared__ RowOut                             s_O;
    const int  tid = threadIdx.x, rank = (int)cluster_rank();
    const bool want_lp = P.cum_log_probs != nullptr || P.out_log_probs != nullptr;
    const int  first = (int)blockIdx.x >> LGN, step = (int)gridDim.x >> LGN;
    const bool again = ROOMY && A.clusters > 0;
    // Launched while the kernel in front of it in the stream drains: nothing of memory is touched before that one has ended.
    // What serves the rows left here may come up in the same way.
    wait_for_previous();
    let_next_come_up();
    __shared__ u32 s_flagged[kWarps];
    int            base = -kThreads, w = kWarps;  // of the flagged rows: place in the search for the next one
    u32            word = 0;
    for (int t = first; t < P.local_batch; t += step) {
        if (again) {
            // (every thread looks at one of the cluster's next 256 rows)
            while (word == 0 && (w + 1 < kWarps || first + step * (base + kThreads) < P.local_batch)) {
                if (++w < kWarps) {
                    word = s_flagged[w];
                    continue;
                }
                base += kThreads;
                w              = -1;
                const int  at  = first + step * (base + tid);
                const bool set = at < P.local_batch && A.redo_flags[P.row_order != nullptr ? P.row_order[at] : at] != 0;
                const u32  b   = __ballot_sync(0xffffffffu, set);
                __syncthreads();
                if ((tid & 31) == 0) {
                    s_flagged[tid >> 5] = b;
                }
                __syncthreads();
            }
            if (word == 0) {
                break;
            }
            t = first + step * (base + w * 32 + __ffs(word) - 1);
            word &= word - 1;
        }
        const int r    = P.row_order != nullptr ? P.row_order[t] : t;
        int       mode = 0;
        if (P.topk_states != nullptr && !(P.topk_skip != nullptr && P.topk_skip[r])) {
            mode = 1;
        }
        else if (P.topp_states != nullptr && !(P.topp_skip != nullptr && P.topp_skip[r])) {
            mode = 2;
        }
        const bool fin = P.finished != nullptr ? P.finished[r] != 0 : false;
        __syncthreads();  // (the previous row's record has been read)
        if (tid == 0) {
            s_O.r      = r;
            s_O.end_id = P.end_ids[r];
            s_O.id_out = P.output_ids + (size_t)P.step * P.batch_size + (size_t)P.ite * P.local_batch + r;
            s_O.trace  = rank == 0 && P.trace != nullptr ? P.trace + (size_t)t * kTraceWords : nullptr;
            if (s_O.trace != nullptr) {
                s_O.trace[0] = (u64)r, s_O.trace[1] = (u64)blockIdx.x, s_O.trace[2] = global_timer_ns();
            }
        }
        __syncthreads();
        bool decided = true;
        if (mode != 0 && !fin) {
            decided = sp_row<DT, LGN>(P, A, smem_raw, s_X, s_O, mode, want_lp);
            __syncthreads();
        }
        if (rank == 0 && tid == 0) {
            if (decided) {
                if (mode == 1 && fin) {
                    *s_O.id_out = s_O.end_id;  // no draw, length unchanged (sampling_topk_kernels.cu:249-252)
                }
                else if (mode != 0 && !fin) {
                    curandState_t& st = (mode == 1 ? P.topk_states : P.topp_states)[r];
                    st.d              = s_X.state[0];
#pragma unroll
                    for (int i = 0; i < 5; ++i) {
                        st.v[i] = s_X.state[1 + i];
                    }
                }
                else if (mode != 0) {
                    finished_topp_row<DT>(P, s_O, draw_uniform(P.topp_states, r), want_lp);
                }
                topp_decay_row(P, r, *s_O.id_out);
            }
            A.redo_flags[r] = decided ? 0 : 1;
            if (s_O.trace != nullptr) {
                s_O.trace[3] = global_timer_ns();
            }
        }
        if (ROOMY && rank == 0 && (A.stop.limit != nullptr || A.stop.stop_words != nullptr)) {
            sp_stop_criteria(P, A.stop, r, A.redo_flags, decided);
        }
        if (again) {
            cluster_sync();  // (the next row starts with nobody inside this one)
        }
    }
    cluster_sync();  // no CTA leaves while another may still reach into its shared memory
}

template<int DT, int LGN, bool ROOMY>
cudaError_t split_opt_in()
{
    static std::atomic<bool> opted_in[kDevicesKnown];
    return opt_in_smem(split_sampling_kernel<DT, LGN, ROOMY>, kSpMaxSmem, opted_in);
}

static inline void split_launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int lgn, int clusters, size_t smem,
                                       cudaStream_t st)
{
    attr[0].id               = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << lgn;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim              = dim3((unsigned)clusters << lgn);
    cfg.blockDim             = dim3(kThreads);
    cfg.dynamicSmemBytes     = smem;
    cfg.stream               = st;
    cfg.attrs                = attr;
    cfg.numAttrs             = 1;
}

template<int DT, int LGN, bool ROOMY>
int split_sampling_launch_n(const KParams& K, const SplitArgs& A, size_t smem, cudaStream_t st)
{
    FTB_CUDA_CHECK((split_opt_in<DT, LGN, ROOMY>()));
    cudaLaunchConfig_t  cfg{};
    cudaLaunchAttribute attr[2];
    split_launch_config(cfg, attr, LGN, A.clusters > 0 ? A.clusters : K.local_batch, smem, st);
    attr[1].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs                                       = 2;
    FTB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, split_sampling_kernel<DT, LGN, ROOMY>, K, A));
    return FTB200_OK;
}

template<int DT, int LGN, bool ROOMY>
int split_resident_n(size_t smem)
{
    // asked once per device and kilobyte of shared memory (what a call needs moves in steps of the vocabulary)
    constexpr int             kMost = (int)(kSpMaxSmem / 1024) + 1;
    static std::atomic<short> known[kDevicesKnown][kMost];  // clusters + 1; 0: not asked yet
    const int                 kb  = (int)((smem + 1023) / 1024);
    int                       dev = 0;
    if (kb >= kMost || cudaGetDevice(&dev) != cudaSuccess) {
        return 0;
    }
    const bool keep = dev >= 0 && dev < kDevicesKnown;
    short      v    = keep ? known[dev][kb].load(std::memory_order_relaxed) : 0;
    if (v == 0) {
        cudaLaunchConfig_t  cfg{};
        cudaLaunchAttribute attr[1];
        int                 n = 0;
        split_launch_config(cfg, attr, LGN, 1, (size_t)kb * 1024, nullptr);
        if (split_opt_in<DT, LGN, ROOMY>() != cudaSuccess
            || cudaOccupancyMaxActiveClusters(&n, split_sampling_kernel<DT, LGN, ROOMY>, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
        v = (short)(n + 1);
        if (keep) {
            known[dev][kb].store(v, std::memory_order_relaxed);
        }
    }
    return v - 1;
}

// Clusters of 2^lgn CTAs with `smem` bytes of shared memory each that the current device holds at once.
template<int DT>
int split_resident(int lgn, bool roomy, size_t smem)
{
    if (roomy) {
        return lgn == 2 ? split_resident_n<DT, 2, true>(smem) : split_resident_n<DT, 3, true>(smem);
    }
    return lgn == 1 ? split_resident_n<DT, 1, false>(smem) : (lgn == 2 ? split_resident_n<DT, 2, false>(smem) : split_resident_n<DT, 3, false>(smem));
}

template<int DT>
int split_sampling_launch(const KParams& K, const SplitArgs& A, cudaStream_t st)
{
    const size_t smem = split_smem_bytes(A.slice, A.area);
    if (A.roomy) {
        return A.lgn == 2 ? split_sampling_launch_n<DT, 2, true>(K, A, smem, st) :
                            split_sampling_launch_n<DT, 3, true>(K, A, smem, st);
    }
    switch (A.lgn) {
        case 1: return split_sampling_launch_n<DT, 1, false>(K, A, smem, st);
        case 2: return split_sampling_launch_n<DT, 2, false>(K, A, smem, st);
        default: return split_sampling_launch_n<DT, 3, false>(K, A, smem, st);
    }
}

}  // namespace ftb200
