// Single-pass form of the fused decode-sampling step for 16-bit logits (half / bfloat16) without an
// embedding bias: the kernel that serves the rows of a step first.  What it cannot decide from one pass
// (and every row kind it does not cover) is put on a list that decode_sampling_kernel works off afterwards,
// so the results are those of that kernel - and therefore the reference's - for every row.
//
// One CTA serves one row at a time; several CTAs share an SM, so that the fixed work of one row (set-up,
// threshold search, the draw) runs under the streaming of the others.  Per row:
//   1. a strided sample of 4096 columns gives, by bisection over the ordered 16-bit keys, a raw threshold
//      that about 2k (at least 128) columns of the row are expected to reach;
//   2. ONE pass over the row (16-byte loads, eight in flight per thread, one packed compare per two logits)
//      queues the vectors that hold a column at or above the threshold;
//   3. the queued vectors give the candidate columns and the count of every value class (bit pattern) above
//      the threshold; penalised / banned columns (token history, bad words, min-length) are taken out and
//      come back with their final values from a short list, as do the columns outside the aligned vectors;
//   4. the draw of topk_stage2_sampling (kernels/sampling_topk_kernels.cu:255-311) walks the classes from the
//      top - equal values add the same exponential, so the sorted sequence is (value, count) runs and no
//      sort of the candidates is needed - and the tie order inside the class the draw lands in follows
//      the reference's two-stage reduction (see resolve_topk_class).
// A row whose candidates turn out to be fewer than k, or that overflows one of the fixed-size tables, is
// left untouched (its generator state included) and goes to the list.
#pragma once
#include "sampling_kernels.cuh"
#include "spans.cuh"

namespace ftb200 {

constexpr int kFCap      = 3840;  // candidate columns held in shared memory
constexpr int kFBins     = 2048;  // value classes (bit patterns) above the threshold
constexpr int kFSpecCap  = 128;   // listed columns (special or edge) at or above the threshold
constexpr int kFClsCap   = 768;   // members of the class the draw lands in
constexpr int kFRuns     = 1536;  // runs the draw may walk (classes + listed columns among the first k)
constexpr int kFRunBytes = kFRuns * 6 + kFBins * 2;  // top-k draw: value, count per run; class ranks
constexpr int kFPRuns    = 3584;  // top-p: runs of the replayed scan (probability, first position); a long history
                                  //        adds a run per listed column to the ~1500 patterns of a deep window
constexpr int kFPSpecCap = 2048;  // top-p: listed columns above the cut (a history of 2000 ids puts a thousand in a deep window)
constexpr int kFPClsCap  = 2048;  // top-p: members of the class the scan stops in
constexpr int kFSampleV  = 2;     // sampled vectors per thread (4096 columns per row)
constexpr int kFUnroll   = 8;     // 16-byte loads in flight per thread
constexpr int kFMaxRank  = 96;    // highest rank among the sampled columns that the threads' maxima are good for

// Shared-memory map of the single-pass kernel (dynamic shared memory, offsets fixed per launch).
struct FMap {
    u32*            cand;  // [kFCap]    (relative key << 20) | column
    u32*            emask; // [mask_words] per aligned vector one byte: which of its columns are special; after the
                           //              pass the same area holds the listed columns and the run arrays of the draw
    u32*            hash;  // [hash_slots] (id << 2) | flags, open addressing
    u32*            sval;  // [hash_slots] gathered raw word, then the final value of that column (float bits)
    u32*            hist;  // [kFBins]   columns per value class above the threshold
    u32*            stage; // [kFStageBytes / 4] token history, word list and last tokens of the row, as fetched
    u32*            lo;    // [kFBins]   top-p rows: columns per bit pattern below the threshold
    uint4*          wbuf;  // [kWarps * kFRing] vectors parked during a pass (static shared memory of the kernel)
    unsigned short* wj;    // [kWarps * kFRing]
};

constexpr int kFMaxHist    = 1024;  // token-history entries the single-pass kernel stages at a time
constexpr int kFMaxHistAll = 4094;  // and in all (the table of special columns: step + words + 2 <= 4096)
constexpr int kFMaxWords   = 128;   // bad-word list length it stages
constexpr int kFRow2Ring   = 16384; // top-p rows, second pass: pairs of 1024-column chunks on their way, four of them
constexpr int kFStageBytes = 8192;  // >= (kFMaxHist + 2 * kFMaxWords + 4) * 4; later kFPSpecCap listed columns of a top-p row
// Special columns that a row with this table has at most (see the plan of the table in sampling_entry.cu).
__host__ __device__ inline int fast_max_records(int hash_slots)
{
    return hash_slots < 2048 ? hash_slots / 2 : (hash_slots / 4 * 3 < 4096 ? hash_slots / 4 * 3 : 4096);
}
// Columns that a top-k row's threshold should let through: 2k, at least k + 256 (the estimate from a few sampled maxima
// scatters widely); for k = 1 a handful is enough.
__host__ __device__ inline int fast_topk_target(int k)
{
    return k == 1 ? 64 : (2 * k > k + 256 ? 2 * k : k + 256);
}
// Rank among the 4096 sampled columns of the value that `target` of ncols reach; a row with a higher one than kFMaxRank is left.
__host__ __device__ inline u32 fast_sample_rank(int target, int ncols)
{
    const u32 rank = (u32)(((long long)target * (kFSampleV * kThreads * 8) + ncols - 1) / ncols);
    return rank < 3u ? 3u : rank;
}
// bytes of the per-vector mask area: one byte per aligned vector, and room for what follows the pass
__host__ __device__ inline size_t fast_mask_bytes(int hash_slots, int vocab_padded, bool topp)
{
    const size_t need = ((size_t)vocab_padded / 8 + 16 + 15) / 16 * 16;
    size_t post = (size_t)kFSpecCap * 8 + (size_t)kFRunBytes;  // the top-k rows' kernel
    if (topp) {
        // The second pass: its ring, a bucket for every warp and 2048 columns, a record for every special column.  Then the runs and one
        // more first position, or the class's columns.
        const size_t pass2 = kFRow2Ring + ((size_t)(kThreads / 32) * (vocab_padded / 2048 + 1) + (size_t)fast_max_records(hash_slots) + 3) / 4 * 16;
        post = (size_t)kFPRuns * 8 + 16;
        post = post > pass2 ? post : pass2;
        static_assert((size_t)kFPRuns * 8 >= (size_t)kFPClsCap * 4, "area too small");
    }
    return need > post ? need : post;
}
__host__ __device__ inline size_t fast_smem_bytes(int hash_slots, int vocab_padded, bool topp)
{
    const size_t sv = topp || hash_slots > kFBins ? hash_slots : kFBins;  // (top-k rows: the value area doubles as a class table)
    return (size_t)kFCap * 4 + fast_mask_bytes(hash_slots, vocab_padded, topp) + (size_t)hash_slots * 4 + sv * 4 + (size_t)kFBins * 4
           + (topp ? (size_t)kFPSpecCap * 8 + (size_t)kFBins * 4 : (size_t)kFStageBytes);
}

__device__ __forceinline__ void cp_async4(u32 saddr, const void* g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async8(u32 saddr, const void* g)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Row constants of the single-pass kernel (shared memory, written by thread 0).
struct FRow {
    const char* rowp;
    int         head, nfull, r, end_id, k;
    float       inv_t, theta, top_p, u;
    __half      inv_t_h;
    int*        id_out;
    u64*        trace;  // this row's record of the diagnostic timeline, or null
};

static __device__ void f_hash_insert(u32* hash, int slots, int shift, int id, u32 flag, int vocab_padded)
{
    if (id < 0 || id >= vocab_padded) {
        return;
    }
    FTB_ASSUME_SHARED(hash);
    u32       h    = hash_slot(id, shift);
    const u32 want = ((u32)id << 2) | flag;
    for (int probe = 0; probe < slots; ++probe) {
        const u32 old = smem_cas(&hash[h], kHashEmpty, want);
        if (old == kHashEmpty) {
            break;
        }
        if ((old >> 2) == (u32)id) {
            smem_or(&hash[h], flag);
            break;
        }
        h = (h + 1) & (slots - 1);
    }
}

// Value of a raw 16-bit pattern after temperature (no bias on this path).
template<int DT>
__device__ __forceinline__ float f_value(u32 raw, bool temp, float inv_t, __half inv_t_h)
{
    if (DT == FTB200_F16) {
        __half h = __ushort_as_half((unsigned short)raw);
        if (temp) {
            h = __hmul(h, inv_t_h);
        }
        return __half2float(h);
    }
    float x = __uint_as_float(raw << 16);
    if (temp) {
        x = x * inv_t;
    }
    return x;
}

// Slot of column `id` in the hash, -1 when it has none.
__device__ __forceinline__ int f_hash_find(const u32* hash, int shift, int mask, int id)
{
    FTB_ASSUME_SHARED(hash);
    u32 h = hash_slot(id, shift);
    for (int probe = 0; probe <= mask; ++probe) {
        const u32 v = hash[h];
        if (v == kHashEmpty) {
            return -1;
        }
        if ((v >> 2) == (u32)id) {
            return (int)h;
        }
        h = (h + 1) & mask;
    }
    return -1;
}

// What the pass over the row leaves behind, all in shared memory.
struct FSink {
    u32*                 cand;   // [kFCap] (relative key << 20) | column of every ordinary column at or above the threshold
    u32*                 hist;   // [kFBins] columns per relative key
    u32*                 sval;   // per hash slot: raw bits of that special column
    const u32*           hash;
    const unsigned char* emask;  // per aligned vector: bit e set = column e of the vector is special
    u32*                 ncand;
    u32*                 bad;    // set when a relative key does not fit the class table
    uint4*               wbuf;   // [kWarps][kFRing] vectors parked by the lanes of a warp
    unsigned short*      wj;     // [kWarps][kFRing] their vector indices
    int                  shift, mask, cap;
};

// One dense step of the side path: every live lane takes one parked vector of its warp, finds the columns at or
// above the threshold from the packed compares, leaves the raw values of special ones next to their hash slots
// and turns the others into candidates (one reservation in the candidate list per step and warp).
// BAND: the columns whose raw value lies in [thr_key, hi_key] are listed by column only (special ones left out).
template<int DT, bool BAND>
__device__ __forceinline__ void f_side_step(const uint4& v, int jj, bool live, int head, u32 thr_key, u32 thr2, u32 hi2,
                                            const FSink& K, u32& relmax)
{
    const int lane = threadIdx.x & 31;
    u32       pm   = 0;
    if (live) {
        u32 m0 = ge2_mask<DT>(v.x, thr2), m1 = ge2_mask<DT>(v.y, thr2);
        u32 m2 = ge2_mask<DT>(v.z, thr2), m3 = ge2_mask<DT>(v.w, thr2);
        if (BAND) {
            m0 &= le2_mask<DT>(v.x, hi2), m1 &= le2_mask<DT>(v.y, hi2);
            m2 &= le2_mask<DT>(v.z, hi2), m3 &= le2_mask<DT>(v.w, hi2);
        }
        pm = ((m0 & 1u) | ((m0 >> 15) & 2u)) | (((m1 & 1u) | ((m1 >> 15) & 2u)) << 2)
             | (((m2 & 1u) | ((m2 >> 15) & 2u)) << 4) | (((m3 & 1u) | ((m3 >> 15) & 2u)) << 6);
        if (BAND) {
            u32 t = pm;
            while (t != 0) {
                const int e = __ffs(t) - 1;
                t &= t - 1;
                if (hash_lookup_raw(K.hash, K.shift, K.mask, head + jj * 8 + e) != 0) {
                    pm &= ~(1u << e);
                }
            }
        }
        else {
            const u32 em = K.emask[jj];
            u32       sp = pm & em;
            pm &= ~em;
            while (sp != 0) {  // rare: a special column at or above the threshold
                const int e = __ffs(sp) - 1;
                sp &= sp - 1;
                const int slot = f_hash_find(K.hash, K.shift, K.mask, head + jj * 8 + e);
                if (slot >= 0) {
                    K.sval[slot] = raw_bits<DT>(v, e);
                }
            }
        }
    }
    const u32 n    = (u32)__popc(pm);
    u32       incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
        incl += lane >= o ? t : 0u;
    }
    const u32 total = __shfl_sync(0xffffffffu, incl, 31);
    if (total == 0) {
        return;
    }
    u32 base = 0;
    if (lane == 0) {
        base = atomicAdd(K.ncand, total);
    }
    base    = __shfl_sync(0xffffffffu, base, 0);
    u32 pos = base + incl - n;
    while (pm != 0) {
        const int e = __ffs(pm) - 1;
        pm &= pm - 1;
        if (BAND) {
            if (pos < (u32)K.cap) {
                K.cand[pos] = (u32)(head + jj * 8 + e);
            }
        }
        else {
            const u32 rel = key16(raw_bits<DT>(v, e)) - thr_key;
            if (rel >= (u32)kFBins) {
                *K.bad = 1;  // (the slot stays unwritten: the row is given up)
            }
            else {
                relmax = rel > relmax ? rel : relmax;
                if (pos < (u32)K.cap) {
                    K.cand[pos] = (rel << 20) | (u32)(head + jj * 8 + e);
                }
                smem_add(&K.hist[rel], 1u);
            }
        }
        ++pos;
    }
}

// The one pass over the row.  Eight 16-byte loads in flight per thread, one packed compare per two logits.
// A vector with a column at or above the threshold is a rare event for a lane but a common one for a warp, so
// a lane does not look at its own hit: it parks the vector in a small ring of its warp, and whenever 32
// vectors are parked the warp takes them one per lane (f_side_step).  Nothing of the row is read a second time.
constexpr int kFRing = 64;  // parked vectors per warp
template<int DT, bool BAND, int UNROLL>
__device__ __noinline__ void f_stream(const uint4* vp, int nfull, int head, u32 thr_key, u32 hi_key, const FSink& Ks,
                                      u32* relmax_out)
{
    const FSink K = Ks;  // (a copy in registers)
    FTB_ASSUME_SHARED(K.cand);
    FTB_ASSUME_SHARED(K.hist);
    FTB_ASSUME_SHARED(K.sval);
    FTB_ASSUME_SHARED(K.emask);
    FTB_ASSUME_SHARED(K.ncand);
    FTB_ASSUME_SHARED(K.bad);
    FTB_ASSUME_SHARED(K.wbuf);
    FTB_ASSUME_SHARED(K.wj);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const u32 thr_raw = key16_inv(thr_key), hi_raw = key16_inv(hi_key);
    const u32 thr2 = thr_raw | (thr_raw << 16), hi2 = hi_raw | (hi_raw << 16);
    uint4* const          wbuf = K.wbuf + wid * kFRing;
    unsigned short* const wj   = K.wj + wid * kFRing;
    int  rd = 0, cnt = 0;  // ring read position and fill (the same in every lane)
    u32  relmax = 0;
    for (int jb = 0; jb < nfull; jb += kThreads * UNROLL) {
        uint4 q[UNROLL];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int j = jb + u * kThreads + tid;
            if (j < nfull) {
                q[u] = ld_nc_v4(vp + j);
            }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int j   = jb + u * kThreads + tid;
            bool      hit = false;
            if (j < nfull) {
                u32 m;
                if (BAND) {
                    m = ((ge2_mask<DT>(q[u].x, thr2) & le2_mask<DT>(q[u].x, hi2))
                         | (ge2_mask<DT>(q[u].y, thr2) & le2_mask<DT>(q[u].y, hi2)))
                        | ((ge2_mask<DT>(q[u].z, thr2) & le2_mask<DT>(q[u].z, hi2))
                           | (ge2_mask<DT>(q[u].w, thr2) & le2_mask<DT>(q[u].w, hi2)));
                }
                else {
                    m = (ge2_mask<DT>(q[u].x, thr2) | ge2_mask<DT>(q[u].y, thr2))
                        | (ge2_mask<DT>(q[u].z, thr2) | ge2_mask<DT>(q[u].w, thr2));
                }
                hit = m != 0;
            }
            const u32 hits = __ballot_sync(0xffffffffu, hit);
            if (hits == 0) {
                continue;
            }
            if (hit) {
                const int at = (rd + cnt + __popc(hits & ((1u << lane) - 1u))) & (kFRing - 1);
                wbuf[at]     = q[u];
                wj[at]       = (unsigned short)j;
            }
            cnt += __popc(hits);
            if (cnt >= 32) {
                __syncwarp();
                const int at = (rd + lane) & (kFRing - 1);
                f_side_step<DT, BAND>(wbuf[at], (int)wj[at], true, head, thr_key, thr2, hi2, K, relmax);
                rd = (rd + 32) & (kFRing - 1);
                cnt -= 32;
                __syncwarp();
            }
        }
    }
    __syncwarp();
    if (cnt > 0) {
        const int  at   = (rd + lane) & (kFRing - 1);
        const bool live = lane < cnt;
        uint4      v    = make_uint4(0u, 0u, 0u, 0u);
        int        jj   = 0;
        if (live) {
            v  = wbuf[at];
            jj = (int)wj[at];
        }
        f_side_step<DT, BAND>(v, jj, live, head, thr_key, thr2, hi2, K, relmax);
    }
    if (!BAND) {
        relmax = __reduce_max_sync(0xffffffffu, relmax);
        if (lane == 0 && relmax != 0) {
            atomicMax(relmax_out, relmax);
        }
    }
}

// The `want`-th largest of the CTA's per-thread sample maxima (ordered 16-bit keys in smax[kThreads]), by
// bisection inside one warp.  With `want` far below the number of threads it is, to within a few ranks, the
// `want`-th largest of all sampled columns - on the low side, which only lets a few more candidates through.
__device__ __forceinline__ u32 f_select_from_maxima(const unsigned short* smax, u32 want, u32* largest)
{
    FTB_ASSUME_SHARED(smax);
    const int lane = threadIdx.x & 31;
    u32       mine[kThreads / 32];
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
        mine[i] = smax[i * 32 + lane];
    }
    {
        u32 mx = 0;
#pragma unroll
        for (int i = 0; i < kThreads / 32; ++i) {
            mx = mine[i] > mx ? mine[i] : mx;
        }
        *largest = __reduce_max_sync(0xffffffffu, mx);
    }
    u32 lo = 0, hi = 0xffffu;
#pragma unroll 1
    for (int it = 0; it < 16; ++it) {
        const u32 mid = (lo + hi + 1) >> 1;
        u32       c   = 0;
#pragma unroll
        for (int i = 0; i < kThreads / 32; ++i) {
            c += mine[i] >= mid ? 1u : 0u;
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= want) {
            lo = mid;
        }
        else {
            hi = mid - 1;
        }
    }
    return lo;
}

// Tie order inside one value class for m <= kThreads members (the rules of resolve_topk_class, by counting
// instead of sorting): member a of lane l = (col / bs1) % 8 has stage-1 rank
//   lane_base[l] + #{b in lane l : t1(b) > t1(a), or t1 equal and col(b) < col(a)},  t1 = col % bs1;
// members whose rank reaches k do not leave stage 1; the others are ordered by ((lane * k + rank) % bs2
// descending, lane * k + rank ascending).  Returns the column at position `want` of that order, -1 when
// there is none.  CTA-collective.
static __device__ int f_resolve_small(const u32* cols, int m, int want, int k, int bs1, int bs2, const u32* lane_base,
                                      u32* key2, int* s_ans)
{
    const int tid = threadIdx.x;
    FTB_ASSUME_SHARED(cols);
    FTB_ASSUME_SHARED(key2);
    if (tid == 0) {
        *s_ans = -1;
    }
    if (tid < m) {
        const u32 c = cols[tid], lane = (c / (u32)bs1) & 7u, t1 = c % (u32)bs1;
        u32       rk = 0;
        for (int b = 0; b < m; ++b) {
            const u32 cb = cols[b], lb = (cb / (u32)bs1) & 7u, tb = cb % (u32)bs1;
            rk += (lb == lane && (tb > t1 || (tb == t1 && cb < c))) ? 1u : 0u;
        }
        const u32 r = lane_base[lane] + rk;
        u32       key = 0xffffffffu;
        if (r < (u32)k) {
            const u32 i2 = lane * (u32)k + r;  // < 8 * 1024
            key          = (((u32)bs2 - 1u - (i2 % (u32)bs2)) << 16) | i2;
        }
        key2[tid] = key;
    }
    __syncthreads();
    if (tid < m) {
        const u32 mine = key2[tid];
        if (mine != 0xffffffffu) {
            int rk = 0;
            for (int b = 0; b < m; ++b) {
                rk += key2[b] < mine ? 1 : 0;
            }
            if (rk == (want < m ? want : m - 1)) {
                *s_ans = (int)cols[tid];
            }
        }
    }
    __syncthreads();
    const int ans = *s_ans;
    __syncthreads();
    return ans;
}

// Header of a row.  It is put together one row ahead by thread 0, in stages spread over the row in front, so
// that none of the dependent loads behind it (ticket -> row number -> per-row arguments and generator state) is
// waited for.
struct FHdr {
    int    t;  // ticket; local_batch when no row is left
    int    r, mode, fin, end_id, k;
    float  top_p, u, inv_t, theta;
    __half inv_t_h;
    u64*   trace;  // the row's record of the diagnostic timeline, or null
};
// landing zone of the next row's arguments (32-bit words; the two generator states sit on 16-byte boundaries)
constexpr int kFPreWords = 48;
enum { kPreStateK = 0, kPreStateP = 12, kPreSkipK = 24, kPreSkipP, kPreFin, kPreEnd, kPreK, kPrePk, kPrePp, kPreTemp,
       kPreRep };


// Arguments of row nr on their way into pre[] (thread 0 only).
static __device__ void f_prefetch_header(const KParams& P, int nr, u32* pre)
{
    const u32 base = (u32)__cvta_generic_to_shared(pre);
    auto word = [&](int slot, const void* p) { cp_async4(base + 4u * (u32)slot, p); };
    if (P.topk_states != nullptr) {
        const char* st = (const char*)(P.topk_states + nr);
        cp_async16(base + 4u * kPreStateK, st);
        cp_async16(base + 4u * kPreStateK + 16u, st + 16);
        cp_async16(base + 4u * kPreStateK + 32u, st + 32);
        word(kPreK, P.topk_ks + nr);
        word(kPrePk, P.topk_ps + nr);
    }
    if (P.topp_states != nullptr) {
        const char* st = (const char*)(P.topp_states + nr);
        cp_async16(base + 4u * kPreStateP, st);
        cp_async16(base + 4u * kPreStateP + 16u, st + 16);
        cp_async16(base + 4u * kPreStateP + 32u, st + 32);
        word(kPrePp, P.topp_ps + nr);
    }
    // The flags are bytes: the words around them where those may be read whole, else the bytes, loaded together and put in
    // their places.  (A copy of a word's part inside its array, worked out here, where this is inlined at every stage of a
    // header, cost the mixed batch of 1024 x 128256 1 %: 204.4 us a step, this form 202.5.)
    const uint8_t *fk = P.topk_states != nullptr ? P.topk_skip : nullptr, *fp = P.topp_states != nullptr ? P.topp_skip : nullptr;
    if (P.whole_words) {
        auto around = [&](int slot, const uint8_t* p) {
            if (p != nullptr) {
                word(slot, (const void*)((size_t)(p + nr) & ~(size_t)3));
            }
        };
        around(kPreSkipK, fk);
        around(kPreSkipP, fp);
        around(kPreFin, P.finished);
    }
    else {
        const u32 a = fk != nullptr ? fk[nr] : 0u, b = fp != nullptr ? fp[nr] : 0u, c = P.finished != nullptr ? P.finished[nr] : 0u;
        pre[kPreSkipK] = a << (8 * ((size_t)(fk + nr) & 3));
        pre[kPreSkipP] = b << (8 * ((size_t)(fp + nr) & 3));
        pre[kPreFin]   = c << (8 * ((size_t)(P.finished + nr) & 3));
    }
    word(kPreEnd, P.end_ids + nr);
    if (P.apply_temp) {
        word(kPreTemp, P.temperature + nr);
    }
    if (P.apply_rep) {
        word(kPreRep, P.rep_penalty + nr);
    }
    cp_async_commit();
}

// Header of ticket nt / row nr from what f_prefetch_header brought in (thread 0 only, after its copies landed).
static __device__ void f_compose_header(const KParams& P, int nt, int rows, int nr, const u32* pre, FHdr& H)
{
    H.t = nt < rows ? nt : P.local_batch;
    if (nt >= rows) {
        return;
    }
    auto byte_at = [&](int slot, const void* p) { return (pre[slot] >> (8 * ((size_t)p & 3))) & 0xffu; };
    int  mode = 0;
    if (P.topk_states != nullptr && !(P.topk_skip != nullptr && byte_at(kPreSkipK, P.topk_skip + nr) != 0)) {
        mode = 1;
    }
    else if (P.topp_states != nullptr && !(P.topp_skip != nullptr && byte_at(kPreSkipP, P.topp_skip + nr) != 0)) {
        mode = 2;
    }
    H.r      = nr;
    H.mode   = mode;
    H.fin    = P.finished != nullptr ? (int)(byte_at(kPreFin, P.finished + nr) != 0) : 0;
    H.end_id = (int)pre[kPreEnd];
    int k    = (int)pre[kPreK];
    H.k      = k < 1 ? 1 : (k > kMaxTopK ? kMaxTopK : k);
    H.top_p  = __uint_as_float(mode == 1 ? pre[kPrePk] : pre[kPrePp]);
    float inv_t = 1.0f;
    if (P.apply_temp) {
        inv_t = 1.0f / (__uint_as_float(pre[kPreTemp]) + 1e-6f);
    }
    H.inv_t   = inv_t;
    H.inv_t_h = __float2half_rn(inv_t);
    H.theta   = P.apply_rep ? __uint_as_float(pre[kPreRep]) : 1.0f;
    H.u       = 0.0f;
    if (mode != 0) {
        // drawn from a copy: the state in memory moves on only when this kernel finishes the row
        curandState_t st = *(const curandState_t*)(pre + (mode == 1 ? kPreStateK : kPreStateP));
        H.u              = curand_uniform(&st);
    }
}

// Geometry of a row.
struct FGeo {
    const char* rowp;
    int         head, nfull;
};
__device__ __forceinline__ FGeo f_geometry(const KParams& P, int r)
{
    FGeo G;
    G.rowp          = (const char*)P.logits + (size_t)r * P.vocab_padded * 2;
    const size_t ad = (size_t)G.rowp;
    const int    hd = (int)(((16 - (ad & 15)) & 15) / 2);
    G.head          = hd < P.vocab_padded ? hd : P.vocab_padded;
    const int vend  = P.vocab < P.vocab_padded ? P.vocab : P.vocab_padded;
    G.nfull         = vend - G.head > 0 ? (vend - G.head) / 8 : 0;
    return G;
}


// ---- top-p rows ------------------------------------------------------------------------------------------
// After the pass a top-p row knows every column at or above the threshold (candidates, class counts, listed
// columns) and with them the row maximum.  What the reference does next, on probabilities
// (kernels/sampling_topp_kernels.cu:1294-1345 soft-max, :801-860 arg-max shortcut, :877-1004 sorted scan):
//   pass 2 (the row again, mostly from L2): the soft-max denominator in the reference's order - thread t owns
//     the "virtual threads" 4t..4t+3 (column mod 1024) and adds four exponentials per 1024-column chunk, strictly
//     in chunk order; special columns take their final value from records filed beforehand, by warp and pair of
//     chunks.  The same pass counts the bit patterns between a provisional cut and the threshold (the special
//     columns' have been taken off, and those of them that fall there are listed from the table), so that the
//     sorted probability sequence is known as (probability, count) runs down to the cut;
//   the block scan of topp_sampling is replayed over the runs (cub::BlockScan<float,256> raking order: 32
//     segments of 8, Kogge-Stone over the segment totals, running prefix chunk by chunk);
//   the class (bit patterns of equal probability) that holds the crossing gives the id: its J-th column in
//     column order, from the candidate list or - below the threshold - from one filtered pass over the row.
// Whatever does not fit (crossing below the cut, tables too small) sends the row to the general kernel.

constexpr int kFMassBins = 128;  // sample mass per 16 bit patterns below the threshold

struct FTopp {
    u32   thr_key, relmax;
    int   n_ord, n_sp;
    float thr_y, neg_max, maxv;
};

template<int DT>
__device__ __forceinline__ float f_round_T(float x)
{
    return DT == FTB200_F16 ? __half2float(__float2half_rn(x)) : x;
}

static __device__ float f_block_sum(float v, float* s_w)
{
    for (int m = 16; m > 0; m >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, m);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        s_w[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    float t = 0.0f;
    for (int i = 0; i < kWarps; ++i) {
        t += s_w[i];
    }
    return t;
}

// Exclusive prefix of one value per thread over the CTA; *total, where given, receives the sum.
static __device__ u32 f_block_excl(u32 v, u32* s_w, u32* total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    u32       incl = v;
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
    if (total != nullptr) {
        *total = tot;
    }
    return base + incl - v;
}

// ---- shared memory by 32-bit address (the hot loop of pass 2 keeps no generic pointer) ----
// Counter i of those at `base`, one more when i < n: the predicate is inside the instruction (no branch around it: a run of these
// stays one basic block).
__device__ __forceinline__ void reds_inc_below(u32 base, u32 i, u32 n)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.u32 p, %1, %2;\n\t@p red.shared.add.u32 [%0], 1;\n\t}" ::"r"(base + 4u * i), "r"(i), "r"(n));
}
__device__ __forceinline__ void sts_f32(u32 addr, float v)
{
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ uint2 lds_v2(u32 addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts_f4(u32 addr, float a, float b, float c, float d)
{
    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void lds_f4(u32 addr, float& a, float& b, float& c, float& d)
{
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "r"(addr) : "memory");
}
// slot of column `id` in the hash at shared address `hash`, -1 when it has none
__device__ __forceinline__ int f_hash_find_saddr(u32 hash, int shift, int mask, int id)
{
    u32 h = hash_slot(id, shift);
    for (int probe = 0; probe <= mask; ++probe) {
        const u32 v = lds_u32(hash + 4u * h);
        if (v == kHashEmpty) {
            return -1;
        }
        if ((v >> 2) == (u32)id) {
            return (int)h;
        }
        h = (h + 1) & mask;
    }
    return -1;
}

// Scalars of pass 2 (one argument block, by value: it travels in the parameter space of the call).
struct FPass2 {
    const char* rowp;
    int         nch, vocab, shift, mask;
    float       maxv, inv_t;
    u32         thr_key, lo_n;
    u32         hash, value, list, ends, ring, hlo, buf, out;  // shared-memory addresses
    __half      inv_t_h;
};

// Special columns of a top-p row, filed for pass 2: a bucket per warp and pair of 1024-column chunks (the columns that the
// warp holds in registers at a time), a record per column: its slot in the hash, whose value word is the column's final
// value, and its place among the warp's 2 x 128 columns.
__device__ __forceinline__ u32 f_bucket(int v, int npair)
{
    return (u32)(((v & 1023) >> 7) * npair + (v >> 11));
}
__device__ __forceinline__ u32 f_record(int slot, int v)
{
    return ((u32)slot << 8) | (u32)((v >> 10) & 1) << 7 | (u32)(v & 127);
}

// Pass 2 of a top-p row over the whole 1024-column chunks [0, nch) and the ragged rest up to `vocab`: thread t
// adds the exponentials of its four "virtual threads" chunk by chunk; with COUNT the columns whose bit
// pattern lies in the lo_n patterns below the threshold are counted (what the special ones among them add has been taken off
// beforehand).  The four sums go to out[4t .. 4t+3].
//
// Special columns: rare for a thread, but some lane of a warp has one in nearly every pair of chunks.  The warp's exponentials go
// through 1 KB of shared memory then, and lanes with a record each put the special ones in their places: 2 + 2 wide accesses
// instead of a divergent table walk that picks one of sixteen registers and puts it back with selects (a third of the
// instructions of the pass).  Rows of 116848
// bf16 with 640 special columns, two on an SM: 32.9 us with the walk, 18.6 so; 51200 half, 150 special columns: 19.7 and 7.9.
enum { kCountNone, kCountPositive, kCountAny };  // (positive: threshold and cut both at or above +0)
template<int DT, int COUNT>
__device__ __noinline__ void f_pass2(const FPass2 A)
{
    const int    tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const float  maxv = A.maxv, inv_t = A.inv_t;
    const __half inv_t_h = A.inv_t_h;
    const u32    thr_key = A.thr_key, lo_n = A.lo_n, hlo = A.hlo;
    float        a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
    const char*  base = A.rowp + (size_t)tid * 8;
    const int    nch = A.nch, npair = (nch + 1) >> 1;
    // (kCountPositive: the index below the threshold is a plain difference of the raw patterns; a negative value, or one at or
    // above the threshold, wraps to a huge index)
    const u32 below = COUNT == kCountPositive ? (thr_key & 0x7fffu) - 1u : thr_key - 1u;
    const u32  buf = A.buf + 1024u * (u32)wid, own = buf + 16u * (u32)lane;
    const u32  ends = A.ends + 4u * (u32)(wid * npair);
    u32        at   = wid > 0 ? lds_u32(ends - 4u) : 0u;
    // A thread's columns of three pairs of chunks are on their way while it works on a pair: eight bytes each into a place of its own,
    // so that nobody waits for anybody; a place is filled again a pair after it was read.
    const u32 ring = A.ring + 8u * (u32)tid;
    auto      send = [&](int m) {
        const u32 to = ring + (u32)(m & 6) * (kFRow2Ring / 8);
        if (m < nch) {
            cp_async8(to, base + (size_t)m * 2048);
        }
        if (m + 1 < nch) {
            cp_async8(to + kFRow2Ring / 8, base + (size_t)(m + 1) * 2048);
        }
        cp_async_commit();
    };
    auto       count = [&](const uint2& q) {
        const u32 w[4] = {q.x & 0xffffu, q.x >> 16, q.y & 0xffffu, q.y >> 16};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            reds_inc_below(hlo, below - (COUNT == kCountPositive ? w[e] : key16(w[e])), lo_n);
        }
    };
    send(0);
    send(2);
    send(4);
    // (one copy of the loop body: with two pairs in it, their loads in registers, it took 25 us for a row of 128256 without counts, with
    // four 49, waiting for its instructions)
#pragma unroll 1
    for (int m = 0; m < nch; m += 2) {
        cp_async_wait<2>();
        const u32   from = ring + (u32)(m & 6) * (kFRow2Ring / 8);
        const uint2 ca = lds_v2(from), cb = lds_v2(from + kFRow2Ring / 8);
        const u32   end = lds_u32(ends + 4u * (u32)(m >> 1));
        send(m + 6);
        float x[8];
        const u32 w[4] = {ca.x, ca.y, cb.x, cb.y};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            // a column at or below -MAX adds exactly zero, as in the reference's loop
            const float y = f_value<DT>((e & 1) ? w[e >> 1] >> 16 : w[e >> 1] & 0xffffu, true, inv_t, inv_t_h);
            x[e]          = f_round_T<DT>(__expf(y - maxv));
        }
        if (end != at) {
            sts_f4(own, x[0], x[1], x[2], x[3]);
            sts_f4(own + 512u, x[4], x[5], x[6], x[7]);
            __syncwarp();
            for (u32 i = at + (u32)lane; i < end; i += 32) {
                const u32 r = lds_u32(A.list + 4u * i);
                sts_f32(buf + 4u * (r & 255u), f_round_T<DT>(__expf(__uint_as_float(lds_u32(A.value + 4u * (r >> 8))) - maxv)));
            }
            __syncwarp();
            lds_f4(own, x[0], x[1], x[2], x[3]);
            lds_f4(own + 512u, x[4], x[5], x[6], x[7]);
            at = end;
        }
        a0 += x[0], a1 += x[1], a2 += x[2], a3 += x[3];
        if (COUNT) {
            count(ca);
        }
        if (m + 1 < nch) {
            a0 += x[4], a1 += x[5], a2 += x[6], a3 += x[7];
            if (COUNT) {
                count(cb);
            }
        }
    }
    // the ragged rest of the row: columns nch * 1024 .. vocab - 1 (padding columns add nothing)
    {
        const int v0 = nch * 1024 + 4 * tid;
        if (v0 < A.vocab) {
            const unsigned short* row16 = (const unsigned short*)A.rowp;
            for (int e = 0; e < 4 && v0 + e < A.vocab; ++e) {
                const u32 r    = (u32)__ldg(row16 + v0 + e);
                const int slot = f_hash_find_saddr(A.hash, A.shift, A.mask, v0 + e);
                const float yy = slot >= 0 ? __uint_as_float(lds_u32(A.value + 4u * (u32)slot)) : f_value<DT>(r, true, inv_t, inv_t_h);
                const float ex = f_round_T<DT>(__expf(yy - maxv));
                a0 += e == 0 ? ex : 0.0f, a1 += e == 1 ? ex : 0.0f, a2 += e == 2 ? ex : 0.0f, a3 += e == 3 ? ex : 0.0f;
                if (COUNT) {
                    reds_inc_below(hlo, thr_key - 1u - key16(r), lo_n);
                }
            }
        }
    }
    __syncthreads();  // (the sums lie over the warps' exponentials)
    sts_f4(A.out + 16u * (u32)tid, a0, a1, a2, a3);
}

// The runs of a nucleus for the replay of the reference's scan (shared-memory addresses): probability and first position of each,
// run at the first position of every 256-entry chunk, aggregate of every chunk.
struct FRuns {
    u32 pr, st, at, agg;
    u32 N;
    int M, nch;
};
// The 8 consecutive probabilities of this lane in chunks c, c + 8, .. (U of them, worked on together: a chunk alone is a search
// of dependent loads, a walk and two serial chains).
template<int U>
__device__ __forceinline__ void f_load8(const FRuns& R, int c, float (*x)[8])
{
    const u32 p0 = (u32)c * 256u + (threadIdx.x & 31u) * 8u;
    int       at[U], hi[U], span = 0;
#pragma unroll
    for (int q = 0; q < U; ++q) {
        const bool in = c + q * kWarps < R.nch;
        at[q]         = in ? (int)lds_u32(R.at + 4u * (u32)(c + q * kWarps)) : R.M - 1;
        hi[q]         = in ? (int)lds_u32(R.at + 4u * (u32)(c + q * kWarps) + 4u) : R.M - 1;
        span |= hi[q] - at[q];
    }
    for (int s = span > 0 ? 1 << (31 - __clz(span)) : 0; s > 0; s >>= 1) {
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int t = at[q] + s;
            if (t <= hi[q] && lds_u32(R.st + 4u * (u32)t) <= p0 + (u32)(q * kWarps) * 256u) {
                at[q] = t;
            }
        }
    }
    // Three runs from the first on, looked up ahead (a walk from run to run is a dependent load and a branch per step, which some
    // lane of the warp takes nearly every time); a lane that needs more walks.
    float pr[U][3];
    u32   nx[U][3];
#pragma unroll
    for (int q = 0; q < U; ++q) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int t = at[q] + i < R.M ? at[q] + i : R.M - 1;
            pr[q][i]    = __uint_as_float(lds_u32(R.pr + 4u * (u32)t));
            nx[q][i]    = lds_u32(R.st + 4u * (u32)t + 4u);  // (behind the last run stands N)
        }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
        const u32 p = p0 + (u32)(q * kWarps) * 256u;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const u32 pe = p + (u32)e;
            x[q][e]      = pe < nx[q][0] ? pr[q][0] : (pe < nx[q][1] ? pr[q][1] : pr[q][2]);
            x[q][e]      = pe < R.N ? x[q][e] : 0.0f;
        }
        if (p + 7u >= nx[q][2] && nx[q][2] < R.N) {
            int   i = at[q] + 2;
            float v = pr[q][2];
            u32   n = nx[q][2];
#pragma unroll
            for (int e = 3; e < 8; ++e) {
                const u32 pe = p + (u32)e;
                if (pe >= n && i + 1 < R.M) {
                    ++i;
                    v = __uint_as_float(lds_u32(R.pr + 4u * (u32)i));
                    n = lds_u32(R.st + 4u * (u32)i + 4u);
                }
                x[q][e] = pe >= nx[q][2] && pe < R.N ? v : x[q][e];
            }
        }
    }
}
// Aggregate of every 256-value chunk in cub::BlockScan's raking order (32 segments of 8, Kogge-Stone across the segment totals);
// the chunks are independent of the running prefix.  Four chunks a warp at a time.
static __device__ __forceinline__ void f_chunk_aggregates(const FRuns R)
{
    constexpr int U = 4;
    const int     lane = threadIdx.x & 31;
#pragma unroll 1
    for (int c = threadIdx.x >> 5; c < R.nch; c += kWarps * U) {
        float x[U][8], inc[U];
        f_load8<U>(R, c, x);
#pragma unroll
        for (int q = 0; q < U; ++q) {
            inc[q] = x[q][0];
#pragma unroll
            for (int i = 1; i < 8; ++i) {
                inc[q] = inc[q] + x[q][i];
            }
        }
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const float t = __shfl_up_sync(0xffffffffu, inc[q], off);
                if (lane >= off) {
                    inc[q] = inc[q] + t;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            if (lane == 31 && c + q * kWarps < R.nch) {
                sts_f32(R.agg + 4u * (u32)(c + q * kWarps), inc[q]);
            }
        }
    }
}

// The listed columns of a top-p row, (~key(probability) << 32) | column, into ascending order.  `bins` [kWarps * kFRing * 4] and `by` [n_sp]
// are scratch (the ring of the pass and the records of the second one); `first`: no entry's leading word is below it.
static __device__ __noinline__ void f_sort_listed(u64* spec, int n_sp, u32* bins, u64* by, u32* s_wsum, u32 first)
{
    const int tid = threadIdx.x;
    FTB_ASSUME_SHARED(spec);
    FTB_ASSUME_SHARED(bins);
    FTB_ASSUME_SHARED(by);
    FTB_ASSUME_SHARED(s_wsum);
    if (n_sp <= kThreads) {
        // (distinct words: the place of each is the number of smaller ones; no network and none of its barriers)
        const u64 mine = tid < n_sp ? spec[tid] : ~0ull;
        int       at   = 0;
        if ((tid & ~31) < n_sp) {
#pragma unroll 4
            for (int b = 0; b < n_sp; ++b) {
                at += spec[b] < mine ? 1 : 0;
            }
        }
        __syncthreads();
        if (tid < n_sp) {
            spec[at] = mine;
        }
    }
    else {
        // Many of them (a long history): by bins of the probability's leading bits, 128 an octave, then by counting inside a bin, which
        // holds a few.  (Rows with 550 listed columns, runs and
    // order together: 14.2 us with a sorting network over them, 13.1 so.)
        constexpr int kBins = kWarps * kFRing * 4;
        auto bin_of = [&](u64 e) {
            const u32 k = (u32)(e >> 32), b = (k > first ? k - first : 0u) >> 16;
            return b < (u32)kBins ? b : (u32)kBins - 1u;
        };
        for (int i = tid; i < kBins; i += kThreads) {
            bins[i] = 0;
        }
        __syncthreads();
        for (int i = tid; i < n_sp; i += kThreads) {
            smem_add(&bins[bin_of(spec[i])], 1u);
        }
        __syncthreads();
        {
            constexpr int PER = kBins / kThreads;
            u32           c[PER], mine = 0;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                c[i] = bins[tid * PER + i];
                mine += c[i];
            }
            u32 run = f_block_excl(mine, s_wsum, nullptr);
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                bins[tid * PER + i] = run;
                run += c[i];
            }
        }
        __syncthreads();
        for (int i = tid; i < n_sp; i += kThreads) {
            const u64 e = spec[i];
            by[atomicAdd(&bins[bin_of(e)], 1u)] = e;
        }
        __syncthreads();
        // (a bin's counter now holds where it ends, the one in front of it where it starts)
        for (int i = tid; i < n_sp; i += kThreads) {
            const u64 e  = by[i];
            const u32 b  = bin_of(e);
            const int lo = b > 0 ? (int)bins[b - 1] : 0, hi = (int)bins[b];
            int       at = lo;
#pragma unroll 1
            for (int j = lo; j < hi; ++j) {
                at += by[j] < e ? 1 : 0;
            }
            spec[at] = e;
        }
    }
}

// Everything of a top-p row after the pass and the listed columns.  Returns true when the row is done.
template<int DT>
__device__ __forceinline__ bool fast_topp_tail(const KParams& P, const FMap& S, const FHdr& H, const FGeo& G, const FTopp& T, u64* spec,
                               u32* s_nspec, const u32* s_mass, float mass_tail, u32 smax_key)
{
    __shared__ float s_w[kWarps], s_den;
    __shared__ u32   s_cut, s_wsum[kWarps], s_ncls, s_fail;
    __shared__ int   s_sel, s_imin, s_imax, s_first, s_after;
    const int        tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool       temp = P.apply_temp != 0;
    u32* const       hist = S.hist;
    u32* const       hlo  = S.lo;
    u32* const       cand = S.cand;
    FTB_ASSUME_SHARED(hist);
    FTB_ASSUME_SHARED(hlo);
    FTB_ASSUME_SHARED(cand);
    FTB_ASSUME_SHARED(spec);
    const u32   thr_key = T.thr_key;
    const float maxv = T.maxv, neg_max = T.neg_max;
    const int   nfull = G.nfull;
    auto value_of = [&](u32 key) { return f_value<DT>(key16_inv(key), temp, H.inv_t, H.inv_t_h); };

    // ---- provisional cut: how far below the threshold the bit patterns have to be counted ----
    // Mass (sum of exp(value - maximum)) at or above the threshold is known exactly; below it the sampled columns
    // give an estimate per 16 bit patterns.  The cut is placed where the estimated cumulative share passes
    // 1.02 u p + 0.05: the part above the threshold is exact and the sampled part (3 % of the row, values under the
    // threshold only, so without the heavy tail of the exponentials) is within about 1.5 % of the total; a cut
    // that proves too high costs the row a trip through the general kernel, a low one more counting.
    float mhi = 0.0f;
    for (int b = tid; b <= (int)T.relmax; b += kThreads) {
        const u32 c = hist[b];
        if (c != 0) {
            mhi += (float)c * __expf(value_of(thr_key + (u32)b) - maxv);
        }
    }
    for (int i = tid; i < T.n_sp; i += kThreads) {
        mhi += __expf(fkey_inv(~(u32)(spec[i] >> 32)) - maxv);
    }
    mhi = f_block_sum(mhi, s_w);
    // records of the special columns: their buckets' first places, then (below) every one to its place
    const int  nwhole = P.vocab >> 10, npair = (nwhole + 1) >> 1, nbucket = kWarps * npair;
    u32* const ends    = S.emask + kFRow2Ring / 4;
    u32* const records = ends + nbucket;
    FTB_ASSUME_SHARED(records);
    FTB_ASSUME_SHARED(ends);
    if (wid == 1) {
        const int per = (nbucket + 31) / 32, b0 = lane * per, b1 = b0 + per < nbucket ? b0 + per : nbucket;
        u32       mine = 0;
#pragma unroll 4
        for (int b = b0; b < b1; ++b) {
            mine += ends[b];
        }
        u32 incl = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, incl, off);
            incl += lane >= off ? t : 0u;
        }
        u32 run = incl - mine;
#pragma unroll 4
        for (int b = b0; b < b1; ++b) {
            const u32 c = ends[b];
            ends[b]     = run;
            run += c;
        }
    }
    if (wid == 0) {
        // (warp 0: four mass bins per lane, a scan over the lanes; the sums are estimates, their order is free)
        static_assert(kFMassBins == 128, "four bins per lane");
        const float scale = __expf(value_of(smax_key) - maxv) * ((float)(nfull * 8) / (float)(kThreads * 8));
        float       mb[4], mine = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            mb[i] = (float)s_mass[lane * 4 + i] * (1.0f / 1048576.0f);
            mine += mb[i];
        }
        float incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, incl, o);
            incl += lane >= o ? t : 0.0f;
        }
        const float lo_all = mass_tail + __shfl_sync(0xffffffffu, incl, 31);
        const float d_est  = mhi + scale * lo_all;
        const float share  = 1.02f * H.u * H.top_p + 0.05f;
        const float target = share * d_est;
        // first bin at which the running mass reaches the target (128: none)
        float acc   = mhi + scale * (incl - mine);
        int   first = kFMassBins;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc += scale * mb[i];
            if (acc >= target && first == kFMassBins) {
                first = lane * 4 + i;
            }
        }
        const u32 hit = __ballot_sync(0xffffffffu, first < kFMassBins);
        const int b   = hit != 0 ? __shfl_sync(0xffffffffu, first, __ffs(hit) - 1) : kFMassBins;
        if (lane == 0) {
            u32 cut = thr_key;
            if (mhi < target) {
                const u32 down = 16u * (u32)(b + 2);
                cut            = thr_key > down ? thr_key - down : 1u;
                if (thr_key - cut > (u32)kFBins) {
                    cut = thr_key - (u32)kFBins;
                }
            }
            s_cut  = cut;
            s_fail = 0;
        }
    }
    __syncthreads();
    const u32   cut_key = s_cut;
    const float cut_y   = cut_key < thr_key ? value_of(cut_key) : T.thr_y;
    for (int i = tid; i < P.hash_slots; i += kThreads) {
        const u32 w  = S.hash[i];
        const int id = (int)(w >> 2);
        if (w == kHashEmpty || id >= P.vocab) {
            continue;
        }
        if (id < nwhole * 1024) {
            records[atomicAdd(&ends[f_bucket(id, npair)], 1u)] = f_record(i, id);
        }
        const float y = __uint_as_float(S.sval[i]);
        if (y >= cut_y && !(y >= T.thr_y) && y > neg_max) {  // (those at or above the threshold are listed already)
            const u32 pos = atomicAdd(s_nspec, 1u);
            if (pos < (u32)kFPSpecCap) {
                spec[pos] = ((u64)(~fkey(y)) << 32) | (u32)id;
            }
        }
    }
    __syncthreads();
    trace_mark(H.trace, 6);

    // ---- pass 2 ----
    float* const s_vt = (float*)S.wbuf;  // [1024] per-virtual-thread sums (the ring of the pass is idle)
    FTB_ASSUME_SHARED(s_vt);
    {
        FPass2 A;
        A.rowp = G.rowp, A.nch = nwhole, A.vocab = P.vocab, A.shift = P.hash_shift, A.mask = P.hash_slots - 1;
        A.maxv = maxv, A.inv_t = H.inv_t, A.thr_key = thr_key, A.lo_n = thr_key - cut_key, A.inv_t_h = H.inv_t_h;
        A.hash = (u32)__cvta_generic_to_shared(S.hash), A.value = (u32)__cvta_generic_to_shared(S.sval);
        A.list = (u32)__cvta_generic_to_shared(records), A.ends = (u32)__cvta_generic_to_shared(ends), A.ring = (u32)__cvta_generic_to_shared(S.emask);
        A.hlo = (u32)__cvta_generic_to_shared(hlo), A.out = (u32)__cvta_generic_to_shared(s_vt), A.buf = A.out;
        const bool positive = cut_key >= 0x8000u && thr_key > 0x8000u;
        // (without a temperature the factor is one, and one multiplication a column: two more copies of the pass cost more)
        if (cut_key >= thr_key) {
            f_pass2<DT, kCountNone>(A);
        }
        else if (positive) {
            f_pass2<DT, kCountPositive>(A);
        }
        else {
            f_pass2<DT, kCountAny>(A);
        }
    }
    __syncthreads();
    trace_mark(H.trace, 7);
    {
        // the reference's blockReduceSum (utils/reduce_kernel_utils.cuh:73-103) over the 1024 partial sums: a
        // butterfly inside every group of 32, then one over the 32 group results
        float* const s_vw = s_vt + 1024;  // [32] (the ring area holds 8 KB)
        for (int w = wid; w < 32; w += kWarps) {
            float v = s_vt[w * 32 + lane];
            for (int m = 16; m > 0; m >>= 1) {
                v = v + __shfl_xor_sync(0xffffffffu, v, m);
            }
            if (lane == 0) {
                s_vw[w] = v;
            }
        }
        __syncthreads();
        if (wid == 0) {
            float v = s_vw[lane];
            for (int m = 16; m > 0; m >>= 1) {
                v = v + __shfl_xor_sync(0xffffffffu, v, m);
            }
            if (lane == 0) {
                s_den = v;
            }
        }
    }
    __syncthreads();
    const float denom = s_den + 1e-6f;
    if (!(denom > 0.0f && denom < 3.0e38f)) {
        return false;  // (not a number, or out of range: nothing below may index with what would follow from it)
    }
    auto prob_of = [&](float y) { return f_round_T<DT>(f_round_T<DT>(__expf(y - maxv)) / denom); };
    const size_t col = (size_t)P.ite * P.local_batch + H.r;
    int* const   id_out = P.output_ids + (size_t)P.step * P.batch_size + col;
    const int    n_sp   = (int)*s_nspec;
    if (n_sp > kFPSpecCap) {
        return false;
    }

    // ---- arg-max shortcut of topp_beam_topk_kernel: the largest probability alone reaches p ----
    const float p_max = f_round_T<DT>(f_round_T<DT>(1.0f) / denom);
    if (p_max >= H.top_p) {
        // first column holding the maximum (larger value, then smaller column)
        if (tid == 0) {
            s_sel = 0x7fffffff;
        }
        __syncthreads();
        const u32 kmaxv = fkey(maxv);
        if (DT == FTB200_F16 && temp && kmaxv == fkey(T.thr_y)) {
            return false;  // (a temperature rounds neighbouring half values to one: it may hold columns below the threshold)
        }
        for (int i = tid; i < T.n_ord; i += kThreads) {
            const u32 e = cand[i];
            if (fkey(value_of(thr_key + (e >> 20))) == kmaxv) {
                atomicMin(&s_sel, (int)(e & 0xfffffu));
            }
        }
        for (int i = tid; i < n_sp; i += kThreads) {
            if (~(u32)(spec[i] >> 32) == kmaxv) {
                atomicMin(&s_sel, (int)(spec[i] & 0xffffffffu));
            }
        }
        __syncthreads();
        const int id = s_sel;
        if (id == 0x7fffffff) {
            return false;
        }
        if (tid == 0) {
            *id_out = id;
            if (P.seq_len != nullptr && P.finished != nullptr) {
                atomicAdd(P.seq_len + H.r, 1);
                P.finished[H.r] = id == H.end_id ? 1 : 0;
            }
        }
        return true;
    }
    const float rand_num = H.u * H.top_p;

    // ---- runs: the counted bit patterns in descending value with the listed columns merged in by probability ----
    // pattern u of the window: key ktop - u, counted in hist (at or above the threshold) or hlo (below it)
    const u32 ktop = thr_key + T.relmax;
    const int npat = (int)(ktop - cut_key) + 1;
    if (npat > 16 * kThreads) {
        return false;
    }
    auto count_of = [&](int u) {
        const u32 key = ktop - (u32)u;
        return u >= npat ? 0u : (key >= thr_key ? hist[key - thr_key] : hlo[thr_key - 1u - key]);
    };
    // listed columns: value keys -> probability keys, sorted (probability descending, column ascending)
    for (int i = tid; i < n_sp; i += kThreads) {
        const u64 e = spec[i];
        spec[i]     = ((u64)(~fkey(prob_of(fkey_inv(~(u32)(e >> 32))))) << 32) | (e & 0xffffffffu);
    }
    __syncthreads();
    f_sort_listed(spec, n_sp, (u32*)S.wbuf, (u64*)S.emask, s_wsum, ~fkey(p_max));
    __syncthreads();
    u32* const run_pr = S.emask;            // [kFPRuns] probability of the run (float bits), descending
    u32* const run_st = run_pr + kFPRuns;   // [kFPRuns] length, then first position of the run
    FTB_ASSUME_SHARED(run_pr);
    FTB_ASSUME_SHARED(run_st);
    for (int i = tid; i < kFPRuns; i += kThreads) {
        run_st[i] = 0u;  // a position no pattern takes keeps length 0 and goes to a listed column
    }
    __syncthreads();
    // A thread takes `per` neighbouring patterns: what the window needs, not the most it can need, so that all threads
    // work.  1500 patterns are 6 to a thread; with 16 to a thread only 94 threads had any.  Counts are read again where
    // they are used (one small loop body instead of 16 copies of it).  Row of 51200, phase: 8.6 -> 5 us.
    const int per = (npat + kThreads - 1) / kThreads;
    int       nA;
    {
        u32 mine = 0;
#pragma unroll 4
        for (int i = 0; i < per; ++i) {
            mine += count_of(tid * per + i) != 0 ? 1u : 0u;
        }
        u32 incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) {
                incl += t;
            }
        }
        if (lane == 31) {
            s_wsum[wid] = incl;
        }
        __syncthreads();
        u32 base = 0, tot = 0;
        for (int i = 0; i < kWarps; ++i) {
            if (i < wid) {
                base += s_wsum[i];
            }
            tot += s_wsum[i];
        }
        nA = (int)tot;
        if (nA + n_sp > kFPRuns) {
            return false;
        }
        u32 at = base + incl - mine;
        int lo = -1;  // listed columns with a strictly larger probability (of neighbours in order: it only grows)
#pragma unroll 1
        for (int i = 0; i < per; ++i) {
            const u32 c = count_of(tid * per + i);
            if (c != 0) {
                const float pr = prob_of(value_of(ktop - (u32)(tid * per + i)));
                const u32   kp = ~fkey(pr);  // ascending in this key = descending probability
                if (lo < 0) {
                    int hi = n_sp;
                    lo     = 0;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if ((u32)(spec[mid] >> 32) < kp) {
                            lo = mid + 1;
                        }
                        else {
                            hi = mid;
                        }
                    }
                }
                while (lo < n_sp && (u32)(spec[lo] >> 32) < kp) {
                    ++lo;
                }
                run_pr[at + lo] = __float_as_uint(pr);
                run_st[at + lo] = c;
                ++at;
            }
        }
    }
    __syncthreads();
    // both lists keep their order in the merged sequence: the listed columns fill the positions the patterns left
    // free, in order
    const int M = nA + n_sp, rpt = (M + kThreads - 1) / kThreads;  // (<= kFPRuns / kThreads = 14)
    {
        u32 freem = 0, mine = 0;
#pragma unroll 4
        for (int i = 0; i < rpt; ++i) {
            const int q = tid * rpt + i;
            if (q < M && run_st[q] == 0u) {
                freem |= 1u << i;
                ++mine;
            }
        }
        u32 incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) {
                incl += t;
            }
        }
        __syncthreads();
        if (lane == 31) {
            s_wsum[wid] = incl;
        }
        __syncthreads();
        u32 j = incl - mine;
        for (int i = 0; i < wid; ++i) {
            j += s_wsum[i];
        }
        while (freem != 0) {
            const int q = tid * rpt + __ffs(freem) - 1;
            freem &= freem - 1;
            if (j >= (u32)n_sp) {
                s_fail = 1;  // two patterns took one position, which only an exponential out of order could bring about
                break;
            }
            run_pr[q] = __float_as_uint(fkey_inv(~(u32)(spec[j] >> 32)));
            run_st[q] = 1u;
            ++j;
        }
    }
    __syncthreads();
    // the exponential has to be monotone over the patterns for the order of the runs to be the sorted order
    for (int i = tid; i + 1 < M; i += kThreads) {
        if (__uint_as_float(run_pr[i]) < __uint_as_float(run_pr[i + 1])) {
            s_fail = 1;
        }
    }
    __syncthreads();
    if (s_fail) {
        return false;
    }
    // exclusive scan of the run lengths -> first position of each run
    u32 N;
    {
        u32 mine = 0;
#pragma unroll 4
        for (int i = 0; i < rpt; ++i) {
            const int q = tid * rpt + i;
            mine += q < M ? run_st[q] : 0u;
        }
        u32 incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) {
                incl += t;
            }
        }
        __syncthreads();
        if (lane == 31) {
            s_wsum[wid] = incl;
        }
        __syncthreads();
        u32 base = 0, tot = 0;
        for (int i = 0; i < kWarps; ++i) {
            if (i < wid) {
                base += s_wsum[i];
            }
            tot += s_wsum[i];
        }
        N      = tot;
        u32 at = base + incl - mine;
        for (int i = 0; i < rpt; ++i) {
            const int q = tid * rpt + i;
            if (q < M) {
                const u32 c = run_st[q];
                run_st[q]   = at;
                at += c;
            }
        }
        if (tid == 0) {
            run_st[M] = N;
        }
    }
    __syncthreads();
    trace_mark(H.trace, 8);
    if (H.trace != nullptr && tid == 0) {
        H.trace[4 + 20] = (u64)(thr_key - cut_key);
        H.trace[4 + 21] = (u64)N;
        H.trace[4 + 22] = (u64)T.n_ord;
    }
    const int nch = (int)((N + 255u) / 256u);
    if (nch > 1000 || N == 0) {
        return false;
    }
    auto run_of = [&](u32 p) {  // run that holds position p
        int lo = 0, hi = M - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (run_st[mid] <= p) {
                lo = mid;
            }
            else {
                hi = mid - 1;
            }
        }
        return lo;
    };
    FRuns R;
    R.pr = (u32)__cvta_generic_to_shared(run_pr), R.st = (u32)__cvta_generic_to_shared(run_st), R.at = (u32)__cvta_generic_to_shared(hlo), R.agg = (u32)__cvta_generic_to_shared(hlo + 1008), R.M = M, R.N = N, R.nch = nch;
    // run at the first position of every 256-entry chunk, and the chunk aggregates (the pattern counts below the
    // threshold are done with: both live where they were)
    int* const   run_at = (int*)hlo;              // [nch + 1]
    float* const agg    = (float*)(hlo + 1008);   // [nch]
    FTB_ASSUME_SHARED(run_at);
    FTB_ASSUME_SHARED(agg);
    for (int c = tid; c <= nch; c += kThreads) {
        run_at[c] = c < nch ? run_of((u32)c * 256u) : M - 1;
    }
    __syncthreads();
    f_chunk_aggregates(R);
    __syncthreads();
    // running prefix chunk by chunk, as the reference's prefix functor accumulates it; stopped a little early
    // (partial sums inside a chunk differ from prefix + aggregate only in the last bits)
    if (wid == 0) {
        float pre = 0.0f;
        int   sel = -2;
        int   c   = running_prefix(agg, nch, rand_num * (1.0f - 1e-4f), pre);  // (nch: the draw lies beyond the counted range)
        for (; c < nch; ++c) {
            float x1[1][8];
            f_load8<1>(R, c, x1);
            const float* x  = x1[0];
            float        up = x[0];
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
            const float ag  = __shfl_sync(0xffffffffu, inc, 31);
            const float ex  = __shfl_up_sync(0xffffffffu, inc, 1);
            float       o   = lane == 0 ? pre : pre + ex;
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
                if ((u32)(c * 256 + g * 32 + 31) >= N) {
                    sel = -2;  // the 32 probabilities of that warp are not all known
                }
                else {
                    sel = c * 256 + g * 32 + (32 - (int)pc);
                }
                break;
            }
            pre = pre + ag;
        }
        if (lane == 0) {
            s_sel = sel;
        }
    }
    __syncthreads();
    const int sel = s_sel;
    trace_mark(H.trace, 9);
    if (sel < 0 || (u32)sel >= N) {
        return false;
    }
    // ---- the class of the crossing: every column whose probability equals that of position sel ----
    const int   i_at  = run_of((u32)sel);
    const float p_sel = __uint_as_float(run_pr[i_at]);
    const u32   k_sel = fkey(p_sel);
    if (tid == 0) {
        s_ncls = 0;
        s_imin = 0x7fffffff;
        s_imax = -1;
        int lo = 0, hi = i_at;  // first run with probability == p_sel (runs are descending)
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (fkey(__uint_as_float(run_pr[mid])) > k_sel) {
                lo = mid + 1;
            }
            else {
                hi = mid;
            }
        }
        s_first = (int)run_st[lo];
        int hj = M;  // first run behind them
        lo     = i_at;
        while (lo < hj) {
            const int mid = (lo + hj) >> 1;
            if (fkey(__uint_as_float(run_pr[mid])) >= k_sel) {
                lo = mid + 1;
            }
            else {
                hj = mid;
            }
        }
        s_after = (int)run_st[lo];
    }
    __syncthreads();
    // bit patterns that map to this probability (one pattern past the counted range is looked at too: a class
    // that reaches down to the cut may go on below it)
#pragma unroll 2
    for (int u = tid; u <= npat && u <= (int)ktop; u += kThreads) {
        if (fkey(prob_of(value_of(ktop - (u32)u))) == k_sel) {
            atomicMin(&s_imin, u);
            atomicMax(&s_imax, u);
        }
    }
    __syncthreads();
    const int J = sel - s_first, n_all = s_after - s_first;  // place in the class, and its columns
    if (s_imax >= npat) {
        return false;
    }
    u32* const cls = S.emask;  // [kFPClsCap] columns of the class (the runs are done with)
    FTB_ASSUME_SHARED(cls);
    const int imin = s_imin, imax = s_imax;
    __syncthreads();
    // listed columns of the class
    for (int j = tid; j < n_sp; j += kThreads) {
        if ((u32)(spec[j] >> 32) == ~k_sel) {
            const u32 pos = atomicAdd(&s_ncls, 1u);
            if (pos < (u32)kFPClsCap) {
                cls[pos] = (u32)(spec[j] & 0xffffffffu);
            }
        }
    }
    int J_far = J;  // its place among the columns that are listed
    if (imax >= 0) {
        const u32 k_hi = ktop - (u32)imin, k_lo = ktop - (u32)imax;
        if (k_lo >= thr_key) {
            // the class lies at or above the threshold: its ordinary columns are candidates
            for (int i = tid; i < T.n_ord; i += kThreads) {
                const u32 e = cand[i], key = thr_key + (e >> 20);
                if (key >= k_lo && key <= k_hi) {
                    const u32 pos = atomicAdd(&s_ncls, 1u);
                    if (pos < (u32)kFPClsCap) {
                        cls[pos] = e & 0xfffffu;
                    }
                }
            }
        }
        else {
            // below the threshold: the ordinary columns of the band come from the row once more, and only as far as the J-th of
            // the class - from whichever end it is nearer to, so a quarter of the row on average.  First the row's last columns (those
            // at or above the threshold are listed columns).
            const int tail0 = nfull * 8;
            if (tail0 + tid < P.vocab && tid < 8 && hash_lookup_raw(S.hash, P.hash_shift, P.hash_slots - 1, tail0 + tid) == 0) {
                const u32 key = key16((u32)__ldg((const unsigned short*)G.rowp + tail0 + tid));
                if (key >= k_lo && key <= k_hi && key < thr_key) {
                    const u32 pos = atomicAdd(&s_ncls, 1u);
                    if (pos < (u32)kFPClsCap) {
                        cls[pos] = (u32)(tail0 + tid);
                    }
                }
            }
            __shared__ FSink s_band;
            if (tid == 0) {
                FSink& K = s_band;
                K.cand = cls, K.hist = S.hist, K.sval = S.sval, K.hash = S.hash, K.emask = (const unsigned char*)S.cand;
                K.ncand = &s_ncls, K.bad = &s_fail, K.shift = P.hash_shift, K.mask = P.hash_slots - 1, K.cap = kFPClsCap;
                K.wbuf = S.wbuf, K.wj = S.wj;
            }
            __syncthreads();
            const int  known = (int)s_ncls;  // columns from anywhere in the row, in front of the band's
            __syncthreads();
            const bool back  = n_all - 1 - J < J, whole = known > kThreads;
            const u32  kcol  = tid < known && !whole ? cls[tid] : 0u;
            const int  need  = back ? n_all - 1 - J : J;
            constexpr int kPart = kThreads * kFUnroll;
            const int  parts = (nfull + kPart - 1) / kPart;
            for (int i = 0; i < parts; ++i) {
                const int part = back ? parts - 1 - i : i, j0 = part * kPart, nv = nfull - j0 < kPart ? nfull - j0 : kPart;
                f_stream<DT, true, kFUnroll>((const uint4*)G.rowp + j0, nv, j0 * 8, k_lo, k_hi, s_band, &s_fail);
                // the class's columns on the near side of what has been read: listed ones and the band's
                const int edge = back ? j0 * 8 : (j0 + nv) * 8;
                const int near = __syncthreads_count(tid < known && (back ? (int)kcol >= edge : (int)kcol < edge));
                const int found = (int)s_ncls - known + near;
                __syncthreads();  // (the count has been read before it goes on)
                if (!whole && found > need) {
                    break;
                }
            }
            if (back) {
                // (counted from the end: the columns left out all lie in front)
                J_far = (int)s_ncls - 1 - need;
            }
        }
    }
    __syncthreads();
    trace_mark(H.trace, 10);
    const int ncls = (int)s_ncls;
    if (ncls > kFPClsCap || J_far < 0 || J_far >= ncls) {
        return false;
    }
    // J-th smallest column of the class (the reference's stable sort leaves equal probabilities in column order)
    if (tid == 0) {
        s_sel = -1;
    }
    __syncthreads();
    for (int a = tid; a < ncls; a += kThreads) {
        const u32    ca   = cls[a];
        int          rk   = 0;
        const uint4* four = (const uint4*)cls;
#pragma unroll 2
        for (int b = 0; b < ncls >> 2; ++b) {
            const uint4 o = four[b];
            rk += (o.x < ca ? 1 : 0) + (o.y < ca ? 1 : 0) + (o.z < ca ? 1 : 0) + (o.w < ca ? 1 : 0);
        }
        for (int b = ncls & ~3; b < ncls; ++b) {
            rk += cls[b] < ca ? 1 : 0;
        }
        if (rk == J_far) {
            s_sel = (int)ca;
        }
    }
    __syncthreads();
    const int id = s_sel;
    if (id < 0) {
        return false;
    }
    if (tid == 0) {
        *id_out = id;
        if (P.seq_len != nullptr && P.finished != nullptr) {
            atomicAdd(P.seq_len + H.r, 1);
            P.finished[H.r] = id == H.end_id ? 1 : 0;
        }
    }
    return true;
}

// One row of the top-k layer (TOPP: of the top-p layer, up to the point where the two part).  Returns true when
// the row is done, false when it has to go to the list
// (nothing of the row's state has been touched then).  CTA-collective.  `stage1` / `stage2` are the hooks
// of the next row's header (run by thread 0 at points where the loads of the previous stage have had time
// to land).
// VP: the row of a vocabulary-parallel local pass (top-k rows only).  The logits are one column shard of the
// vocabulary: token ids become columns by subtracting P.vocab_offset, and instead of drawing the row hands every
// column whose value reaches the shard's k-th value (whole tie class) to the exchange record, as topk_tail does.
template<int DT, bool TOPP, int VP, class S1, class S2>
__device__ __forceinline__ bool fast_row(const KParams& P, const FMap& S, const FHdr& H, S1&& stage1, S2&& stage2)
{
    static_assert(!(TOPP && VP), "the record form serves top-k rows");
    const int id_shift = VP ? P.vocab_offset : 0;
    __shared__ u32   s_mass[kFMassBins];  // sample mass per bin, in units of 2^-20 (integer adds are native)
    __shared__ float s_mtail[kWarps];
    __shared__ u32   s_smaxkey, s_vmaxkey;
    __shared__ FSink s_sink;
    __shared__ u32            s_ncand, s_nspec, s_bad, s_ncls, s_lane_base[8], s_thr, s_relmax;
    __shared__ unsigned short s_smax[kThreads];
    __shared__ int            s_pick_idx, s_ans, s_nruns;
    __shared__ float          s_vsel;
    const int                 tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool                temp = P.apply_temp != 0;
    u32* const                hash = S.hash;
    u32* const                sval = S.sval;
    u32* const                hist = S.hist;
    u32* const                cand = S.cand;
    FTB_ASSUME_SHARED(hash);
    FTB_ASSUME_SHARED(sval);
    FTB_ASSUME_SHARED(hist);
    FTB_ASSUME_SHARED(cand);
    const int    r     = H.r;
    const FGeo   G     = f_geometry(P, r);
    const uint4* vp    = (const uint4*)(G.rowp + (size_t)G.head * 2);
    const int    nfull = G.nfull;
    const size_t col   = (size_t)P.ite * P.local_batch + r;

    // ---- everything the row's set-up needs is sent for at once: the sampled columns into registers, the
    //      token history, the word list and the last three tokens into shared memory (asynchronous copies) ----
    // sample: 16 blocks of 512 contiguous bytes spread over the row (one per warp and round), 4096 columns
    uint4 smp[kFSampleV];
#pragma unroll
    for (int v = 0; v < kFSampleV; ++v) {
        const int blk   = v * kWarps + wid;
        const int start = (int)(((long long)blk * (nfull - 32)) / (kFSampleV * kWarps - 1)) & ~31;
        smp[v]          = ld_nc_v4(vp + start + lane);
    }
    int* const stage_ids   = (int*)S.stage;                 // [kFMaxHist] history ids (-1: position not counted)
    int* const stage_words = stage_ids + kFMaxHist;         // [2 * kFMaxWords] the row's word list
    int* const stage_last  = stage_words + 2 * kFMaxWords;  // [3] tokens of steps step-3 .. step-1
    FTB_ASSUME_SHARED(stage_ids);
    FTB_ASSUME_SHARED(stage_words);
    FTB_ASSUME_SHARED(stage_last);
    const int  L     = P.bad_words != nullptr ? P.bad_words_len : 0;
    const int* wbase = L > 0 ? (P.bad_words_shared ? P.bad_words : P.bad_words + (size_t)r * 2 * L) : nullptr;
    const int  nhist = P.apply_rep ? P.step : 0;
    {
        // (input_lengths is read here, one dependent load: it is the same few cache lines for every row)
        const int input_len = P.apply_rep ? (P.input_lengths != nullptr ? P.input_lengths[r] : P.max_input_len) : 0;
        for (int t = tid; t < nhist && t < kFMaxHist; t += kThreads) {
            if (t >= input_len && t < P.max_input_len) {
                stage_ids[t] = -1;
            }
            else {
                cp_async4((u32)__cvta_generic_to_shared(&stage_ids[t]), P.output_ids + (size_t)t * P.batch_size + col);
            }
        }
        for (int i = tid; i < 2 * L; i += kThreads) {
            cp_async4((u32)__cvta_generic_to_shared(&stage_words[i]), wbase + i);
        }
        if (tid < 3 && P.step - 3 + tid >= 0) {
            cp_async4((u32)__cvta_generic_to_shared(&stage_last[tid]),
                      P.output_ids + (size_t)(P.step - 3 + tid) * P.batch_size + col);
        }
        cp_async_commit();
    }
    u32* const emask32 = S.emask;
    FTB_ASSUME_SHARED(emask32);
    {
        // (four words a store: every array starts on a 16-byte boundary and has a multiple of four words)
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u), ones = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
        static_assert(kHashEmpty == 0xffffffffu && kFBins % (4 * kThreads) == 0, "clearing by four words");
        for (int i = tid; i < P.hash_slots / 4; i += kThreads) {
            ((uint4*)hash)[i] = ones;
            ((uint4*)sval)[i] = ones;  // no raw value seen: the column lies below the threshold
        }
#pragma unroll
        for (int i = 0; i < kFBins / 4; i += kThreads) {
            ((uint4*)hist)[i + tid] = zero;
            if (TOPP) {
                ((uint4*)S.lo)[i + tid] = zero;
            }
        }
        for (int i = tid; i < (nfull + 15) / 16; i += kThreads) {
            ((uint4*)emask32)[i] = zero;
        }
    }
    if (tid < 8) {
        s_lane_base[tid] = 0;
    }
    if (tid == 0) {
        s_ncand = 0, s_nspec = 0, s_bad = 0, s_ncls = 0, s_relmax = 0, s_vmaxkey = 0;
        FSink& K = s_sink;
        K.cand = cand, K.hist = hist, K.sval = sval, K.hash = hash, K.emask = (const unsigned char*)S.emask;
        K.ncand = &s_ncand, K.bad = &s_bad, K.shift = P.hash_shift, K.mask = P.hash_slots - 1, K.cap = kFCap;
        K.wbuf = S.wbuf, K.wj = S.wj;
    }
    if (TOPP && tid < kFMassBins) {
        s_mass[tid] = 0u;
    }
    {
        // largest sampled column of this thread, as an ordered key
        u32 m2 = max2<DT>(max2<DT>(smp[0].x, smp[0].y), max2<DT>(smp[0].z, smp[0].w));
#pragma unroll
        for (int v = 1; v < kFSampleV; ++v) {
            m2 = max2<DT>(m2, max2<DT>(max2<DT>(smp[v].x, smp[v].y), max2<DT>(smp[v].z, smp[v].w)));
        }
        const u32 ka = key16(m2 & 0xffffu), kb = key16(m2 >> 16);
        s_smax[tid]  = (unsigned short)(ka > kb ? ka : kb);
    }
    cp_async_wait_all();  // history, word list and last tokens have landed
    __syncthreads();
    stage1();
    trace_mark(H.trace, 0);

    // ---- threshold from the sample (warp 0) while the other warps file the special columns: token history,
    //      banned words, min-length mask (the rules of build_row; kernels/sampling_penalty_kernels.cu:385-410,
    //      :493-499, kernels/ban_bad_words.cu:35-85) ----
    const int k      = H.k;
    const int ncols  = nfull * 8;
    // columns the threshold should let through: 2k, at least k + 256 (the estimate from a few sampled maxima
    // scatters widely); for k = 1 a handful is enough
    // (a top-p row of a smaller vocabulary aims lower: the estimate needs the wanted rank well inside the 256
    //  per-thread maxima of the sample, want_s <= 96 below)
    const int tp_cap = (int)(((long long)ncols * kFMaxRank) / (kFSampleV * kThreads * 8));
    const u32 want_s = fast_sample_rank(TOPP ? (tp_cap < 2048 ? tp_cap : 2048) : fast_topk_target(k), ncols);
    bool words_ok    = true;
    if (wid == 0) {
        u32       kmx = 0;
        const u32 t   = f_select_from_maxima(s_smax, want_s, &kmx);
        if (lane == 0) {
            s_thr     = t;
            s_smaxkey = kmx;
        }
    }
    else {
        const int wt = tid - 32, wn = kThreads - 32;
        for (int t = wt; t < nhist && t < kFMaxHist; t += wn) {
            const int id = stage_ids[t];
            if (id >= 0) {
                f_hash_insert(hash, P.hash_slots, P.hash_shift, id - id_shift, kFlagHist, P.vocab_padded);
            }
        }
        for (int i = wt; i < L; i += wn) {
            const int e1 = stage_words[L + i];
            if (e1 < 0) {
                continue;
            }
            const int s1 = i > 0 ? stage_words[L + i - 1] : 0, size = e1 - s1;
            if (size > 4) {
                words_ok = false;  // longer words: the general kernel's loop
                continue;
            }
            bool b = size == 1;
            if (size > 1 && P.step >= size - 1) {
                b = true;
                for (int j = 0; j < size - 1; ++j) {
                    // generated token of step (step - (size - 1) + j)
                    b = b && stage_last[3 - (size - 1) + j] == stage_words[s1 + j];
                }
            }
            if (b) {
                const int tok = stage_words[e1 - 1];
                if (0 < tok && (VP || tok < P.vocab_padded)) {
                    f_hash_insert(hash, P.hash_slots, P.hash_shift, tok - id_shift, kFlagDead, P.vocab_padded);
                }
            }
        }
        if (P.apply_minlen && wt == 0) {
            if (P.seq_len[r] + 1 - P.max_input_len < P.min_lengths[r]) {
                f_hash_insert(hash, P.hash_slots, P.hash_shift, H.end_id - id_shift, kFlagDead, P.vocab_padded);
            }
        }
    }
    const bool long_words = __syncthreads_or(!words_ok);
    // a history of more than kFMaxHist ids comes through the staging area a tile at a time
    for (int base = kFMaxHist; base < nhist; base += kFMaxHist) {
        const int input_len = P.input_lengths != nullptr ? P.input_lengths[r] : P.max_input_len;
        for (int t = base + tid; t < nhist && t < base + kFMaxHist; t += kThreads) {
            if (t >= input_len && t < P.max_input_len) {
                stage_ids[t - base] = -1;
            }
            else {
                cp_async4((u32)__cvta_generic_to_shared(&stage_ids[t - base]), P.output_ids + (size_t)t * P.batch_size + col);
            }
        }
        cp_async_commit();
        cp_async_wait_all();
        __syncthreads();
        for (int t = base + tid; t < nhist && t < base + kFMaxHist; t += kThreads) {
            const int id = stage_ids[t - base];
            if (id >= 0) {
                f_hash_insert(hash, P.hash_slots, P.hash_shift, id - id_shift, kFlagHist, P.vocab_padded);
            }
        }
        __syncthreads();
    }
    stage2();
    // per-vector byte: which columns of the vector are special
    for (int i = tid; i < P.hash_slots; i += kThreads) {
        const u32 w = hash[i];
        if (w != kHashEmpty) {
            const int rel = (int)(w >> 2) - G.head;
            if (rel >= 0 && (rel >> 3) < nfull) {
                smem_or(&emask32[rel >> 5], (1u << (rel & 7)) << (8 * ((rel >> 3) & 3)));
            }
        }
    }
    const u32   thr_key = s_thr;
    const u32   thr_raw = key16_inv(thr_key);
    const float thr_y   = f_value<DT>(thr_raw, temp, H.inv_t, H.inv_t_h);
    const float neg_max = DT == FTB200_F16 ? -65504.0f : -FLT_MAX;
    if (TOPP) {
        // mass of the sampled columns below the threshold, per 16 bit patterns, relative to the largest sampled value
        // (the provisional cut of the second pass is placed with it)
        const float v_ref = f_value<DT>(key16_inv(s_smaxkey), temp, H.inv_t, H.inv_t_h);
        float       far   = 0.0f;
        {
            constexpr int v = 0;  // (half the sample is plenty here; the scale below accounts for it)
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const u32 raw = raw_bits<DT>(smp[v], e);
                const u32 kk  = key16(raw);
                if (kk < thr_key && (raw & 0x7fffu) <= (DT == FTB200_F16 ? 0x7c00u : 0x7f80u)) {
                    const float w = __expf(f_value<DT>(raw, temp, H.inv_t, H.inv_t_h) - v_ref);
                    const u32   b = (thr_key - 1u - kk) >> 4;
                    if (b < (u32)kFMassBins) {
                        smem_add(&s_mass[b], (u32)(w * 1048576.0f));
                    }
                    else {
                        far += w;
                    }
                }
            }
        }
        for (int m = 16; m > 0; m >>= 1) {
            far += __shfl_xor_sync(0xffffffffu, far, m);
        }
        if (lane == 0) {
            s_mtail[wid] = far;
        }
    }
    __syncthreads();
    trace_mark(H.trace, 1);
    if (long_words || want_s > (u32)kFMaxRank || !(thr_y > neg_max) || thr_key == 0u) {
        return false;  // (uniform for the CTA)
    }

    // ---- the pass ----
    f_stream<DT, false, kFUnroll>(vp, nfull, G.head, thr_key, 0u, s_sink, &s_relmax);
    __syncthreads();
    trace_mark(H.trace, 2);
    trace_mark(H.trace, 3);
    trace_mark(H.trace, 4);
    // ---- listed columns: special ones with their final value, and the row's edges ----
    // (~key(value) << 32) | column.  Top-k rows: [kFSpecCap] where the per-vector bytes were (they are done with);
    // top-p rows: [kFPSpecCap] where the row's set-up data was (the bytes make room for the records of the second pass)
    u64* const    spec     = TOPP ? (u64*)S.stage : (u64*)S.emask;
    constexpr int spec_cap = TOPP ? kFPSpecCap : kFSpecCap;
    FTB_ASSUME_SHARED(spec);
    const int  nwhole = P.vocab >> 10, npair = (nwhole + 1) >> 1, nbucket = kWarps * npair;
    u32* const ends   = S.emask + kFRow2Ring / 4;  // top-p rows: records per bucket, then where the buckets end
    if (TOPP) {
        FTB_ASSUME_SHARED(ends);
        for (int i = tid; i < nbucket; i += kThreads) {
            ends[i] = 0;
        }
        __syncthreads();
    }
    {
        Xf X;
        X.bias = nullptr, X.inv_t = H.inv_t, X.theta = H.theta, X.neg_max = neg_max, X.inv_t_h = H.inv_t_h;
        X.apply_temp = P.apply_temp, X.apply_rep = P.apply_rep, X.penalty_type = P.penalty_type, X.vocab = P.vocab;
        X.hash_shift = P.hash_shift, X.hash_mask = P.hash_slots - 1, X.hash = hash;
        auto push = [&](int c, float y) {
            if (y >= thr_y && y > neg_max) {
                const u32 pos = atomicAdd(&s_nspec, 1u);
                if (pos < (u32)spec_cap) {
                    spec[pos] = ((u64)(~fkey(y)) << 32) | (u32)c;
                }
                if (TOPP) {
                    atomicMax(&s_vmaxkey, fkey(y));
                }
            }
        };
        if (TOPP) {
            // Every special column's final value goes where its raw value was, the pass that sums the exponentials reads it
            // there.  That pass counts columns by raw value, the special ones with them, so they are taken off here.  Raw values
            // below the threshold come from the row (it has just been read), four on their way per thread.
            u32* const lo = S.lo;
            FTB_ASSUME_SHARED(lo);
            for (int i0 = tid; i0 < P.hash_slots; i0 += 4 * kThreads) {
                u32 w[4], raw[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int i = i0 + q * kThreads;
                    w[q]        = i < P.hash_slots ? hash[i] : kHashEmpty;
                    w[q]        = w[q] != kHashEmpty && (int)(w[q] >> 2) < P.vocab ? w[q] : kHashEmpty;
                    raw[q]      = w[q] != kHashEmpty ? sval[i] : 0u;
                    if (raw[q] == 0xffffffffu) {
                        raw[q] = (u32)__ldg((const unsigned short*)G.rowp + (w[q] >> 2));
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (w[q] == kHashEmpty) {
                        continue;
                    }
                    const int   id = (int)(w[q] >> 2);
                    const float y  = special_value<DT>(X, temp_value<DT>(X, raw[q], id), w[q] & 3u);
                    sval[i0 + q * kThreads] = __float_as_uint(y);
                    push(id, y);
                    const u32 down = thr_key - 1u - key16(raw[q]);
                    if (down < (u32)kFBins) {
                        smem_add(&lo[down], 0xffffffffu);
                    }
                    if (id < nwhole * 1024) {
                        smem_add(&ends[f_bucket(id, npair)], 1u);
                    }
                }
            }
        }
        for (int i = tid; !TOPP && i < P.hash_slots; i += kThreads) {
            const u32 w = hash[i];
            if (w == kHashEmpty) {
                continue;
            }
            const int id = (int)(w >> 2);
            if (id >= P.vocab) {
                continue;
            }
            const int rel = id - G.head;
            const u32 raw = (rel >= 0 && (rel >> 3) < nfull) ? sval[i] : (u32)__ldg((const unsigned short*)G.rowp + id);
            if (raw == 0xffffffffu) {
                continue;  // below the threshold before its penalty, and a penalty only lowers a value here
            }
            push(id, special_value<DT>(X, temp_value<DT>(X, raw, id), w & 3u));
        }
        const int tail0 = G.head + nfull * 8;
        const int nedge = G.head + (P.vocab - tail0 > 0 ? P.vocab - tail0 : 0);
        for (int i = tid; i < nedge; i += kThreads) {
            const int v = i < G.head ? i : tail0 + (i - G.head);
            if (v < P.vocab && hash_lookup_raw(hash, X.hash_shift, X.hash_mask, v) == 0) {
                // (top-p rows: on this side of the threshold by its raw value, as every column that is not special; the second pass counts
                // the others, half values that a temperature rounds to the threshold's among them)
                const u32 raw = (u32)__ldg((const unsigned short*)G.rowp + v);
                if (!TOPP || key16(raw) >= thr_key) {
                    push(v, temp_value<DT>(X, raw, v));
                }
            }
        }
    }
    __syncthreads();
    trace_mark(H.trace, 5);
    const int n_ord = (int)s_ncand, n_sp = (int)s_nspec;
    if (s_bad || n_ord > kFCap || n_sp > spec_cap || n_ord + n_sp < (TOPP ? 1 : k)) {
        return false;
    }
    if constexpr (VP != 0) {
        // ---- vocabulary-parallel local pass: the record of this row (see topk_tail) ----
        const int n = n_ord + n_sp;
        if (n > kFCap / 2) {
            return false;  // (the entries are sorted as 64-bit words in the candidate area)
        }
        __shared__ int s_m;
        u64* const     big = (u64*)cand;
        FTB_ASSUME_SHARED(big);
        {
            constexpr int PER = (kFCap / 2 + kThreads - 1) / kThreads;
            u64           mine[PER];
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int a = tid + i * kThreads;
                mine[i]     = ~0ull;
                if (a < n_ord) {
                    const u32 e = cand[a];
                    const u32 kv = fkey(f_value<DT>(key16_inv(thr_key + (e >> 20)), temp, H.inv_t, H.inv_t_h));
                    mine[i]      = ((u64)(~kv) << 32) | (u64)(e & 0xfffffu);
                }
                else if (a < n) {
                    mine[i] = spec[a - n_ord];
                }
            }
            __syncthreads();  // every 32-bit entry has been read before the 64-bit ones take its place
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int a = tid + i * kThreads;
                if (a < n) {
                    big[a] = mine[i];
                }
            }
        }
        __syncthreads();
        group_sort_u64(big, n, tid, kThreads, CtaSync());
        __syncthreads();
        const int k_eff = k < n ? k : n;
        if (tid == 0) {
            s_m = k_eff;
        }
        __syncthreads();
        const u32 kv = (u32)(big[k_eff - 1] >> 32);
        if (DT == FTB200_F16 && temp && ~kv == fkey(thr_y)) {
            return false;  // half products round: patterns below the threshold may share the lowest class's value
        }
        for (int i = k_eff + tid; i < n; i += kThreads) {
            if ((u32)(big[i] >> 32) == kv) {
                atomicMax(&s_m, i + 1);
            }
        }
        __syncthreads();
        const int m   = s_m;
        u64*      out = P.vp_out + (size_t)r * (P.vp_cap + 2);
        if (tid == 0) {
            out[0] = m > P.vp_cap ? ~0ull : (u64)m;  // ~0: more ties than the exchange record holds
        }
        for (int i = tid; i < m && i < P.vp_cap; i += kThreads) {
            const u64 e = big[i];
            out[1 + i]  = (e & 0xffffffff00000000ull) | (u64)((u32)(e & 0xffffffffu) + (u32)P.vocab_offset);
        }
        return true;
    }
    if constexpr (TOPP) {
        if (n_ord < 1) {
            return false;
        }
        __shared__ FTopp s_T;  // (read where they are used: every register is taken)
        __shared__ FGeo  s_G;
        const float top_ord = f_value<DT>(key16_inv(thr_key + s_relmax), temp, H.inv_t, H.inv_t_h);
        const float top_sp  = s_vmaxkey != 0 ? fkey_inv(s_vmaxkey) : -INFINITY;
        if (tid == 0) {
            s_T.thr_key = thr_key, s_T.relmax = s_relmax, s_T.n_ord = n_ord, s_T.n_sp = n_sp;
            s_T.thr_y = thr_y, s_T.neg_max = neg_max, s_T.maxv = fmaxf(top_ord, top_sp);
            s_G       = G;
        }
        float mass_tail     = 0.0f;
        for (int i = 0; i < kWarps; ++i) {
            mass_tail += s_mtail[i];
        }
        __syncthreads();
        return fast_topp_tail<DT>(P, S, H, s_G, s_T, spec, &s_nspec, s_mass, mass_tail, s_smaxkey);
    }

    // ---- the draw (warp 0): runs of equal values from the top, then the reference's sequential sum and walk ----
    float* const          fe    = (float*)(spec + kFSpecCap);      // [kFRuns] value of the run
    unsigned short* const fc    = (unsigned short*)(fe + kFRuns);  // [kFRuns] columns of the run
    unsigned short* const crank = fc + kFRuns;                     // [kFBins] relative key of the a-th class from the top
    float* const          flat  = (float*)hist;                    // [k] exponentials of the first k entries (the counts are
                                                                   //     done with once the runs stand)
    FTB_ASSUME_SHARED(fe);
    FTB_ASSUME_SHARED(fc);
    FTB_ASSUME_SHARED(crank);
    FTB_ASSUME_SHARED(flat);
    if (wid == 0) {
        group_sort_u64<WarpSync, true>(spec, n_sp, lane, 32, WarpSync());
        __syncwarp();
        auto spec_above = [&](float v) {  // listed columns with a value strictly above v
            int       lo = 0, hi = n_sp;
            const u32 kc = ~fkey(v);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if ((u32)(spec[mid] >> 32) < kc) {
                    lo = mid + 1;
                }
                else {
                    hi = mid;
                }
            }
            return lo;
        };
        // classes from the top bin down, 32 bins per trip, until they alone cover k columns (the listed columns
        // can only add to that); a class sits at (its rank among the classes) + (listed columns above it)
        int  nA = 0, covered = 0;
        bool over = false;
        for (int b0 = (int)s_relmax; b0 >= 0 && covered < k; b0 -= 32) {
            const int b   = b0 - lane;
            const u32 c   = b >= 0 ? hist[b] : 0u;
            const u32 any = __ballot_sync(0xffffffffu, c != 0);
            if (any == 0) {
                continue;
            }
            if (c != 0) {
                const float cv  = f_value<DT>(key16_inv(thr_key + (u32)b), temp, H.inv_t, H.inv_t_h);
                const int   a   = nA + __popc(any & ((1u << lane) - 1u));
                const int   pos = a + spec_above(cv);
                if (pos < kFRuns) {
                    fe[pos]  = cv;
                    fc[pos]  = (unsigned short)c;
                    crank[a] = (unsigned short)b;
                }
                else {
                    over = true;
                }
            }
            covered += (int)__reduce_add_sync(0xffffffffu, c);
            nA += __popc(any);
        }
        over = __any_sync(0xffffffffu, over);
        __syncwarp();
        // a listed column sits at (its rank among the listed columns) + (classes at or above its value); below
        // the last class taken the order no longer matters (k columns are covered before that)
        if (!over) {
            for (int i = lane; i < n_sp; i += 32) {
                const float sv = fkey_inv(~(u32)(spec[i] >> 32));
                int         lo = 0, hi = nA;  // classes (descending values) with value >= sv
                while (lo < hi) {
                    const int   mid = (lo + hi) >> 1;
                    const float cv  = f_value<DT>(key16_inv(thr_key + (u32)crank[mid]), temp, H.inv_t, H.inv_t_h);
                    if (cv >= sv) {
                        lo = mid + 1;
                    }
                    else {
                        hi = mid;
                    }
                }
                const int pos = i + lo;
                if (pos < kFRuns) {
                    fe[pos] = sv;
                    fc[pos] = 1;
                }
                else {
                    over = true;
                }
            }
            over = __any_sync(0xffffffffu, over);
        }
        const int nruns = nA + n_sp;
        __syncwarp();
        trace_mark(H.trace, 7);
        if (!over) {
            // the first k entries of the sorted sequence, as exponentials against the largest value: every run
            // writes its copies (the sequence the reference's thread 0 walks, sampling_topk_kernels.cu:276-287)
            const float vmax = fe[0];
            int         at   = 0;  // entries in front of the current batch of runs
            for (int p0 = 0; p0 < nruns && at < k; p0 += 32) {
                const int p    = p0 + lane;
                const int c    = p < nruns ? (int)fc[p] : 0;
                int       incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    incl += lane >= o ? t : 0;
                }
                if (c != 0) {
                    const float e   = __expf(fe[p] - vmax);
                    const int   beg = at + incl - c;
                    const int   end = beg + c < k ? beg + c : k;
                    for (int i = beg; i < end; ++i) {
                        flat[i] = e;
                    }
                }
                at += __shfl_sync(0xffffffffu, incl, 31);
            }
            const int k16 = (k + 15) & ~15;  // (zeros behind the last term change neither the sum nor the walk)
            if (k + lane < k16) {
                flat[k + lane] = 0.0f;
            }
            __syncwarp();
            trace_mark(H.trace, 8);
            // Dependent adds in the reference's order, by one lane: sixteen terms a round, eight on their way while eight are added.
            // The walk leaves its running values where the terms were; they only fall, so the first one that ends the
            // reference's loop lies in the last round and is found by the warp, as is the run that it belongs to (1024 x
            // 128256 bf16 with both kinds of rows: 182 us a step, 200 with a walk tested term by term and a search run by run).
            int walked = 0;
            if (lane == 0) {
                float  sum = 0.0f;
                float4 v0 = *(const float4*)flat, v1 = *(const float4*)(flat + 4);
#pragma unroll 1
                for (int i = 0; i < k16; i += 16) {
                    const float4 w0 = *(const float4*)(flat + i + 8), w1 = *(const float4*)(flat + i + 12);
                    sum += v0.x, sum += v0.y, sum += v0.z, sum += v0.w;
                    sum += v1.x, sum += v1.y, sum += v1.z, sum += v1.w;
                    const int nx = i + 16 < k16 ? i + 16 : 0;
                    v0 = *(const float4*)(flat + nx), v1 = *(const float4*)(flat + nx + 4);
                    sum += w0.x, sum += w0.y, sum += w0.z, sum += w0.w;
                    sum += w1.x, sum += w1.y, sum += w1.z, sum += w1.w;
                }
                float rand_num = H.u * H.top_p * sum;
                auto  walk4    = [&](const float4& x, int i) {
                    float4 r;
                    r.x                  = rand_num - x.x;
                    r.y                  = r.x - x.y;
                    r.z                  = r.y - x.z;
                    r.w                  = r.z - x.w;
                    rand_num             = r.w;
                    *(float4*)(flat + i) = r;
                };
#pragma unroll 1
                do {
                    const float4 w0 = *(const float4*)(flat + walked + 8), w1 = *(const float4*)(flat + walked + 12);
                    walk4(v0, walked);
                    walk4(v1, walked + 4);
                    const int nx = walked + 16 < k16 ? walked + 16 : 0;
                    v0 = *(const float4*)(flat + nx), v1 = *(const float4*)(flat + nx + 4);
                    walk4(w0, walked + 8);
                    walk4(w1, walked + 12);
                    walked += 16;
                } while (walked < k16 && !(rand_num <= 0.0f));
            }
            walked = __shfl_sync(0xffffffffu, walked, 0);
            __syncwarp();
            const int  i0   = walked - 16 + lane;
            const bool ends = lane < 16 && i0 < k && flat[i0] <= 0.0f;
            const u32  hit  = __ballot_sync(0xffffffffu, ends);
            const int  pick = hit != 0 ? walked - 16 + __ffs(hit) - 1 : k - 1;
            // value of the picked entry: the run that holds position `pick`
            int acc = 0, prun = 0;
            for (int p0 = 0; p0 < nruns; p0 += 32) {
                const int p    = p0 + lane;
                int       incl = p < nruns ? (int)fc[p] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    incl += lane >= o ? t : 0;
                }
                const u32 beyond = __ballot_sync(0xffffffffu, acc + incl > pick);
                if (beyond != 0) {
                    prun = p0 + __ffs(beyond) - 1;
                    break;
                }
                acc += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) {
                s_pick_idx = pick;
                s_vsel     = fe[prun];
            }
        }
        if (lane == 0) {
            s_nruns = over ? -1 : nruns;
        }
    }
    __syncthreads();
    trace_mark(H.trace, 9);
    if (s_nruns < 0) {
        return false;
    }
    // ---- the class the draw landed in: its members (all of them, also beyond the first k) and, per lane of
    //      the reference's first stage, the number of larger candidates ----
    const float vsel = s_vsel;
    const u32   ksel = fkey(vsel);
    if (DT == FTB200_F16 && temp && ksel == fkey(thr_y)) {
        return false;  // half products round: patterns below the threshold may share the lowest class's value
    }
    // (the run arrays are not needed any more: the class members take their place)
    u32* const cls  = (u32*)(spec + kFSpecCap);  // [kFClsCap]
    u32* const key2 = cls + kFClsCap;   // [kThreads] scratch of the small resolve
    FTB_ASSUME_SHARED(cls);
    const u32 bs1 = P.max_top_k <= 16 ? 128 : 256;
    const u32 bs2 = P.max_top_k <= 32 ? 128 : 256;
    const int sh1 = bs1 == 128 ? 7 : 8;
    {
        u32 packd_lo = 0, packd_hi = 0;  // 8 x 8-bit counters (a thread sees at most kFCap / kThreads entries)
        auto visit = [&](u32 kv, u32 c) {
            if (kv == ksel) {
                const u32 pos = atomicAdd(&s_ncls, 1u);
                if (pos < (u32)kFClsCap) {
                    cls[pos] = c;
                }
            }
            else if (kv > ksel) {
                const u32 l = (c >> sh1) & 7u;
                if (l < 4) {
                    packd_lo += 1u << (8 * l);
                }
                else {
                    packd_hi += 1u << (8 * (l - 4));
                }
            }
        };
        for (int i = tid; i < n_ord; i += kThreads) {
            const u32 e = cand[i];
            visit(fkey(f_value<DT>(key16_inv(thr_key + (e >> 20)), temp, H.inv_t, H.inv_t_h)), e & 0xfffffu);
        }
        for (int i = tid; i < n_sp; i += kThreads) {
            visit(~(u32)(spec[i] >> 32), (u32)(spec[i] & 0xffffffffu));
        }
        for (int l = 0; l < 8; ++l) {
            u32 cnt = ((l < 4 ? packd_lo : packd_hi) >> (8 * (l & 3))) & 0xffu;
            cnt     = __reduce_add_sync(0xffffffffu, cnt);
            if (lane == 0 && cnt != 0) {
                atomicAdd(&s_lane_base[l], cnt);
            }
        }
    }
    __syncthreads();
    trace_mark(H.trace, 10);
    const int m = (int)s_ncls;
    // number of candidates above the class = position of its first member in the sorted sequence
    int lo_cnt = 0;
    for (int l = 0; l < 8; ++l) {
        lo_cnt += (int)s_lane_base[l];
    }
    const int want = s_pick_idx - lo_cnt;
    if (m > kFClsCap || m < 1 || want < 0 || want >= m) {
        return false;  // (cannot happen for a consistent walk; the list takes the row if it does)
    }
    int idc;
    if (m == 1) {
        idc = (int)cls[0];
    }
    else if (m <= kThreads) {
        idc = f_resolve_small(cls, m, want, k, (int)bs1, (int)bs2, s_lane_base, key2, &s_ans);
    }
    else {
        // large classes: the sorting form, on 64-bit entries in the candidate area (its contents are done with)
        u64* big = (u64*)cand;
        for (int i = tid; i < m; i += kThreads) {
            big[i] = (u64)cls[i];
        }
        __syncthreads();
        idc = resolve_topk_class(big, m, want, k, (int)bs1, (int)bs2, s_lane_base);
    }
    if (tid == 0) {
        if (idc < 0) {
            idc = 0;
        }
        P.output_ids[(size_t)P.step * P.batch_size + col] = idc;
        if (P.seq_len != nullptr && P.finished != nullptr) {
            atomicAdd(P.seq_len + r, 1);
            P.finished[r] = idc == H.end_id ? 1 : 0;
        }
    }
    return true;
}

// The step's end for a host that waits for it, by every CTA of the two kernels (stop words are seen to row by row): the last one
// does the length limit and the count of finished rows, or tells the host that rows are on the list.  A step of 1024 x 128256
// then ends with its last row, where the join of two streams, the general kernel over an empty list and the criteria's kernel followed
// one another.  CTAs without a row arrive too (those of the top-k rows' kernel may come up last, where the top-p rows' one held their
// SMs), and nothing is queued behind: when the host hears of the end, nothing of the step is left that could read the workspace or
// take its tickets.
static __device__ __noinline__ void f_step_end(const KParams& P, const StopArgs& T)
{
    if (arrived_last(T.arrived, T.ctas)) {
        count_finished(P, T, nullptr, __ldcg(P.redo_count) != 0);
    }
}

// In front of the single-pass kernels: the header of the workspace (tickets, counters) to zero, and, where a call has rows of both
// layers, either kernel's rows in the given order.  (Idle CTAs of the top-p rows' kernel that took 860 of 1024 rows off the tickets only
// to see that they are the other kernel's held their SMs for 9 us.)  The layers' skip flags alone decide; the flags of finished
// rows change while the kernels run.
constexpr int kFListThreads = 1024;
enum { kFHeadRowsK = 5, kFHeadRowsP = 6 };  // words of the header: rows of the two lists
static __global__ void __launch_bounds__(kFListThreads) fast_rows_kernel(const __grid_constant__ KParams P, int* list_k, int* list_p)
{
    __shared__ u32 s_k[kFListThreads / 32], s_p[kFListThreads / 32];
    let_next_come_up();
    wait_for_previous();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    int       n_k = 0, n_p = 0;
    for (int base = 0; list_k != nullptr && base < P.local_batch; base += kFListThreads) {
        const int  t  = base + tid;
        const bool in = t < P.local_batch;
        const int  r  = in ? (P.row_order != nullptr ? P.row_order[t] : t) : 0;
        const bool topp = in && P.topk_skip != nullptr && P.topk_skip[r] != 0 && !(P.topp_skip != nullptr && P.topp_skip[r] != 0);
        const u32  bk = __ballot_sync(0xffffffffu, in && !topp), bp = __ballot_sync(0xffffffffu, topp), below = (1u << lane) - 1u;
        __syncthreads();
        if (lane == 0) {
            s_k[wid] = __popc(bk), s_p[wid] = __popc(bp);
        }
        __syncthreads();
        int at_k = n_k, at_p = n_p;
        for (int w = 0; w < kFListThreads / 32; ++w) {
            const int ck = (int)s_k[w], cp = (int)s_p[w];
            at_k += w < wid ? ck : 0, at_p += w < wid ? cp : 0;
            n_k += ck, n_p += cp;
        }
        if (topp) {
            list_p[at_p + __popc(bp & below)] = r;
        }
        else if (in) {
            list_k[at_k + __popc(bk & below)] = r;
        }
    }
    if (tid < 64 && tid != kFHeadRowsK) {
        P.ticket[tid] = tid == kFHeadRowsP ? (u32)n_p : 0u;
    }
    __syncthreads();
    if (tid == 0) {
        store_release(P.ticket + kFHeadRowsK, (u32)n_k);  // (what the top-k rows' kernel acquires: see there)
    }
}

// The two kernels of a step with both kinds of rows follow each other in one stream and run side by side: the top-p rows' kernel lets
// the other one come up at once, and that one waits for it at its end, so that what follows in the stream finds both done.  (A second
// stream, forked and joined with events, cost four calls of the host in front of the kernels and a wait behind them.)
// Spilled registers cost the top-p rows' kernel more than anything else: two CTAs with 100 KB of shared memory each leave L1 too little for
// 200 bytes a thread, and every access goes to L2.  With its scalars in shared memory and three copies of the second pass it spills
// 12 to 20 bytes (196 before): 256 x 51200 half 61.0 -> 52.8 us a step, 1024 x 128256 bf16 of both kinds 174.9 -> 163.0.
template<int DT, bool TOPP, int VP = 0>
__global__ void __launch_bounds__(kThreads, TOPP ? 2 : 3) fast_sampling_kernel(const __grid_constant__ KParams P, const __grid_constant__ StopArgs T)
{
    // With both kinds of rows the top-k rows' kernel comes up beside the top-p rows' one, whose CTAs have all seen the end of the list
    // kernel by then, and that one the end of what is in front of it: everything read here has been written before this grid
    // starts.  That it is seen follows from the list kernel's release of the number of rows, its last store, which thread 0 acquires
    // below before any thread reads memory.
    const bool beside = !TOPP && VP == 0 && P.row_count_dev != nullptr;
    if (!beside) {
        wait_for_previous();
    }
    let_next_come_up();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ FHdr                               s_hdr[2];
    __shared__ __align__(16) u32                  s_pre[kFPreWords];
    __shared__ uint4                              s_wbuf[kWarps * 64];
    __shared__ unsigned short                     s_wj[kWarps * 64];
    FMap S;
    {
    S.wbuf = s_wbuf;
    S.wj   = s_wj;
    S.cand = (u32*)smem_raw;
    S.emask = S.cand + kFCap;
    S.hash  = S.emask + fast_mask_bytes(P.hash_slots, P.vocab_padded, TOPP) / 4;
    S.sval  = S.hash + P.hash_slots;
    S.hist  = S.sval + (TOPP || P.hash_slots > kFBins ? P.hash_slots : kFBins);
    S.stage = S.hist + kFBins;
    S.lo    = S.stage + 2 * kFPSpecCap;  // (top-p rows' kernel alone)
    }
    const int tid = threadIdx.x;
    // thread 0 keeps the next row's ticket and number between the stages
    __shared__ int s_rows;  // rows of this kernel
    int            nt = 0, nr = 0;
    if (tid == 0) {
        s_rows = P.row_count_dev != nullptr ? (int)load_acquire(P.row_count_dev) : P.local_batch;
        nt     = (int)atomicAdd(P.ticket + (TOPP ? 3 : 0), 1u);
        if (nt < s_rows) {
            nr = P.row_order != nullptr ? __ldcg(P.row_order + nt) : nt;
            f_prefetch_header(P, nr, s_pre);
            cp_async_wait_all();
        }
        f_compose_header(P, nt, s_rows, nr, s_pre, s_hdr[0]);
    }
    for (int cur = 0;; cur ^= 1) {
        __syncthreads();
        const FHdr& H = s_hdr[cur];
        if (H.t >= P.local_batch) {
            break;
        }
        const int  r   = H.r;
        if (tid == 0) {
            u64* const rec = P.trace != nullptr ? P.trace + ((size_t)H.t + (TOPP ? 2 * (size_t)P.local_batch : 0)) * kTraceWords : nullptr;
            s_hdr[cur].trace = rec;
            if (rec != nullptr) {
                rec[0] = (u64)r, rec[1] = (u64)blockIdx.x, rec[2] = global_timer_ns();
                rec[4 + 25] = (u64)clock64();
            }
            nt = (int)atomicAdd(P.ticket + (TOPP ? 3 : 0), 1u);  // stage 0 of the next row's header
        }
        auto stage1 = [&]() {
            if (tid == 0 && nt < s_rows) {
                nr = P.row_order != nullptr ? __ldcg(P.row_order + nt) : nt;
            }
        };
        auto stage2 = [&]() {
            if (tid == 0 && nt < s_rows) {
                f_prefetch_header(P, nr, s_pre);
            }
        };
        bool       done   = false;
        int* const id_out = P.output_ids + (size_t)P.step * P.batch_size + (size_t)P.ite * P.local_batch + r;
        const bool topp_row = H.mode == 2;
        if (VP != 0 && !(H.mode == 1 && !H.fin)) {
            // vocabulary-parallel local pass: a top-p row is left to the general kernel (its statistics form), any
            // other row has nothing to send
            stage1();
            stage2();
            if (!topp_row || H.fin) {
                if (tid == 0) {
                    P.vp_out[(size_t)r * (P.vp_cap + 2)] = 0;
                }
                done = true;
            }
        }
        else if (H.mode != 0 && !H.fin) {
            const FGeo G  = f_geometry(P, r);
            // (a penalty that can raise a value - repetition below 1, presence below 0 - would make columns
            //  under the threshold candidates: those rows go to the general kernel)
            const bool lowers = !P.apply_rep || (P.penalty_type == FTB200_PENALTY_MULTIPLICATIVE ? H.theta >= 1.0f :
                                                 P.penalty_type == FTB200_PENALTY_ADDITIVE ? H.theta >= 0.0f : true);
            // (the second pass of a top-p row wants it on a 16-byte boundary)
            const bool ok = lowers && (!TOPP || G.head == 0) && G.nfull >= 2048 && G.nfull <= 65535 && H.inv_t > 0.0f && H.inv_t < 3.0e38f
                            && (P.apply_rep ? P.step : 0) <= kFMaxHistAll
                            && (P.bad_words != nullptr ? P.bad_words_len : 0) <= kFMaxWords;
            if (ok) {
                done = fast_row<DT, TOPP, VP>(P, S, H, stage1, stage2);
                if (VP == 0 && done && tid == 0) {
                    curandState_t* states = H.mode == 1 ? P.topk_states : P.topp_states;
                    curandState_t  st     = states[r];
                    (void)curand_uniform(&st);
                    states[r] = st;
                }
            }
            else {
                stage1();
                stage2();
            }
        }
        else {
            stage1();
            stage2();
            if (H.mode == 0) {
                done = true;
            }
            else if (H.mode == 1) {
                // kernels/sampling_topk_kernels.cu:249-252: end id, no draw, length unchanged
                if (tid == 0) {
                    *id_out = H.end_id;
                }
                done = true;
            }
            else {
                // a finished row of the top-p layer: one-hot on the end id with probability 1 / (1 + 1e-6)
                // (kernels/sampling_topp_kernels.cu:1309-1341); the layer still draws
                if (tid == 0) {
                    const float p0 = DT == FTB200_F16 ? __half2float(__float2half_rn(1.0f / (1.0f + 1e-6f))) :
                                                        1.0f / (1.0f + 1e-6f);
                    *id_out        = H.end_id;
                    if ((p0 >= H.top_p || H.u * H.top_p <= p0) && P.seq_len != nullptr && P.finished != nullptr) {
                        P.finished[r] = 1;
                    }
                    curandState_t st = P.topp_states[r];
                    (void)curand_uniform(&st);
                    P.topp_states[r] = st;
                }
                done = true;
            }
        }
        __syncthreads();
        if (tid == 0) {
            if (H.trace != nullptr) {
                H.trace[3] = global_timer_ns();
                H.trace[4 + 26] = (u64)clock64();
                H.trace[4 + 27] = done ? 1 : 0;
            }
            if (!done) {
                P.redo_rows[atomicAdd(P.redo_count, 1u)] = r;
            }
            else if (VP == 0 && P.topp_states != nullptr && P.topp_decay != nullptr) {
                // top-p decay / reset (kernels/sampling_topp_kernels.cu:1381-1408), applied to every row of the call
                const int id = *id_out;
                float     p  = P.topp_ps[r];
                if (id == P.topp_reset[r]) {
                    p = P.topp_initial[r];
                }
                else {
                    p = fmaxf(p * P.topp_decay[r], P.topp_min[r]);
                }
                P.topp_ps[r] = p;
            }
            // the next row's header: its arguments were sent for before this row's pass
            cp_async_wait_all();
            f_compose_header(P, nt, s_rows, nr, s_pre, s_hdr[cur ^ 1]);
        }
        if (VP == 0 && T.limit != nullptr && T.stop_words != nullptr && done) {
            row_stop_words(P, T.stop_words, T.stop_words_len, T.finished, r);
        }
    }
    if (VP == 0 && T.limit != nullptr && T.ctas != 0) {
        f_step_end(P, T);
    }
    if (beside) {
        wait_for_previous();
    }
}

template<int DT, bool TOPP, int VP = 0>
int fast_sampling_occupancy(size_t smem, int* per_sm)
{
    // per device: the opt-in to the shared-memory size (a per-device attribute of the kernel) and the answer
    static std::mutex mu;
    static size_t     highest[kDevicesKnown], asked[kDevicesKnown];
    static int        val[kDevicesKnown];
    int               dev = 0;
    FTB_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kDevicesKnown) {
        set_error("ftb200_decode_step_sampling: device ordinal out of range");
        return FTB200_UNSUPPORTED;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (asked[dev] != smem) {
        FTB_CUDA_CHECK(raise_smem(fast_sampling_kernel<DT, TOPP, VP>, smem, highest[dev]));
        FTB_CUDA_CHECK(
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&val[dev], fast_sampling_kernel<DT, TOPP, VP>, kThreads, smem));
        asked[dev] = smem;
    }
    *per_sm = val[dev];
    return FTB200_OK;
}

inline int fast_rows_launch(const KParams& K, int* list_k, int* list_p, cudaStream_t st)
{
    FTB_CUDA_CHECK(launch_early(fast_rows_kernel, dim3(1), dim3(kFListThreads), 0, st, K, list_k, list_p));
    return FTB200_OK;
}

template<int DT, bool TOPP, int VP = 0>
int fast_sampling_launch(const KParams& K, const StopArgs& T, int grid, size_t smem, bool beside, cudaStream_t st)
{
    if (beside) {
        FTB_CUDA_CHECK(launch_early(fast_sampling_kernel<DT, TOPP, VP>, dim3((unsigned)grid), dim3(kThreads), smem, st, K, T));
        return FTB200_OK;
    }
    fast_sampling_kernel<DT, TOPP, VP><<<grid, kThreads, smem, st>>>(K, T);
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

}  // namespace ftb200
