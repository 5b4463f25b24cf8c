// Launch arguments of the split decode-sampling kernel (split_sampling.cuh), shared with the entry point.
#pragma once
#include "sampling_params.cuh"

namespace ftb200 {

constexpr int kSpBins     = 2048;
constexpr int kSpAreaMin  = 5120;                   // fp32 keys a CTA can receive of a nucleus: least,
constexpr int kSpAreaMid  = 6144;                   // most where the kernel keeps to 80 registers,
constexpr int kSpAreaMax  = 10240;                  // and most where it has 128 and two CTAs are on an SM (multiples of 1024; the launch chooses)
constexpr int kSpAreaWide = 16384;                  // with one CTA on an SM, the second launch over flagged rows too: all of 128000 columns
constexpr int kSpCandCap  = kSpAreaMin / 2;         // 64-bit candidates the leader can receive
constexpr int kSpMaxN     = 8;                       // portable cluster size
constexpr size_t kSpMaxSmem = 216 * 1024;
constexpr int kSpMinSlice = (kNB * 4 + 1024 * 4) / 4;  // the draw's histogram and values lie over the slice

// What a launch that leaves rows stores in place of its result.  No result: its high word is not the step's sequence number, so
// that a caller who waits for that number goes on waiting.
__host__ __device__ inline u64 rows_left(u32 sequence) { return ((u64)~sequence << 32) | 0xffffffffu; }

// Stop criteria of the step, for the launch forms that finish everything themselves.
struct StopArgs {
    const int*      stop_words;      // [local_batch, 2, stop_words_len] or null
    int             stop_words_len;
    const uint32_t* limit;           // [batch_size] or null: then nothing is counted
    uint8_t*        finished;        // [batch_size], the whole batch
    u32*            arrived;         // one word, zero between calls
    u64*            result;          // page-locked host word: sequence << 32 | finished rows
    u32             sequence;
    u32             ctas;            // single-pass kernels: CTAs that arrive, all of them; 0: the general kernel behind ends the step
};

struct SplitArgs {
    int  lgn;         // log2 of the CTAs per row
    int  slice;       // floats of the slice area
    int  area;        // keys of the collection area
    int  roomy;       // the form with 128 registers
    int  criteria;    // whether the launch may do the step's stop criteria (roomy form)
    int  at_once;     // all clusters are resident together: the rows' order does not matter
    int* redo_flags;  // [local_batch]: 1 when the row is left to another launch
    StopArgs stop;    // (roomy form; without a limit the rows' stop words alone)
    int  clusters;    // 0: one per row; else so many, which look for rows with redo_flags set and serve those (roomy form)
};

__host__ __device__ inline size_t split_smem_bytes(int slice, int area)
{
    return (size_t)slice * 4 + (size_t)area * 5 + (size_t)kSpBins * 8;  // (five: a key, and two 16-bit sub-buckets for four)
}

}  // namespace ftb200
