// Chains of beam parents followed in parallel, shared by the gather tree, the archive and the beam step's penalties.
#pragma once
#include "common.cuh"
#include "device_once.cuh"
#include "ftb200.h"

namespace ftb200 {

// ---- parent chains in parallel ----------------------------------------------------------------------------
// A level's parents map a beam to a beam, and maps compose: the levels are cut into segments, every segment finds
// where each of its K possible entries comes out (all segments at once), a short walk over the segments gives every
// beam its entry, and the segments are walked again, now writing.  Three walks of about sqrt(levels) dependent
// shared-memory reads instead of one of `levels` (2048 levels x 4 beams: 5 us, against 60).
// `par` [levels][K + 1]: byte offset (2 x beam) of each beam's parent within its row; the last entry of a row stands for
// "no parent" and leads to itself, so that a step of a walk is one add and one shared-memory read.  `sel` [levels][K]
// receives the beam that beam j's chain passes at each level below its start (K: none); `start` / `from`: the level
// above which beam j's chain begins and its beam there (K: none).
struct Chains {
    u32 par, sel, comp, entry;  // 32-bit shared-memory addresses; comp, entry: [segments][K + 1], [segments][K]
    u32 start, from;            // [K] ints
    int K, levels, seglen, segments;
};
constexpr int kChainThreads  = 1024;
constexpr int kChainSegments = 64;

__device__ __forceinline__ u32 lds_u16(u32 a)
{
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ void walk_chains(const Chains& c)
{
    const int tid = threadIdx.x, K = c.K, W = K + 1;
    const u32 row = 2u * (u32)W;
    for (int e = tid; e < c.segments * W; e += kChainThreads) {
        const int seg = e / W, lo = seg * c.seglen, hi = min(lo + c.seglen, c.levels);
        u32       cur = 2u * (u32)(e % W), at = c.par + (u32)hi * row;
        for (int i = lo; i < hi; ++i) {
            at -= row;
            cur = lds_u16(at + cur);
        }
        sts_u16(c.comp + 2u * (u32)e, cur);
    }
    __syncthreads();
    for (int j = tid; j < K; j += kChainThreads) {
        const int top = (int)lds_u32(c.start + 4u * (u32)j);
        u32       cur = 2u * lds_u32(c.from + 4u * (u32)j);
        int       seg = top > 0 ? (top - 1) / c.seglen : -1;
        if (seg >= 0) {
            sts_u16(c.entry + 2u * (u32)(seg * K + j), cur);
            const int lo = seg * c.seglen;  // the chain starts inside this segment
            for (int level = top - 1; level >= lo; --level) {
                cur = lds_u16(c.par + (u32)level * row + cur);
            }
            for (--seg; seg >= 0; --seg) {
                sts_u16(c.entry + 2u * (u32)(seg * K + j), cur);
                cur = lds_u16(c.comp + (u32)seg * row + cur);
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < c.segments * K; e += kChainThreads) {
        const int seg = e / K, j = e % K, lo = seg * c.seglen, top = (int)lds_u32(c.start + 4u * (u32)j);
        const int hi  = min(min(lo + c.seglen, c.levels), top);
        if (lo < hi) {
            u32 cur = lds_u16(c.entry + 2u * (u32)e), at = c.par + (u32)hi * row, out = c.sel + 2u * (u32)(hi * K + j);
            for (int i = lo; i < hi; ++i) {
                at -= row;
                out -= 2u * (u32)K;
                sts_u16(out, cur >> 1);
                cur = lds_u16(at + cur);
            }
        }
    }
    __syncthreads();
}

__host__ __device__ inline int chain_segments(int levels, int K)
{
    int s = 1;
    while (s * s < levels && s < kChainSegments && (s + 1) * (K + 1) <= kChainThreads) {
        ++s;
    }
    return s;
}
inline size_t chain_smem_bytes(int levels, int K)
{
    return (size_t)levels * (2 * K + 1) * 2 + (size_t)chain_segments(levels, K) * (2 * K + 1) * 2 + 64;
}
// Tables of an entry behind each other in dynamic shared memory.
__device__ __forceinline__ Chains map_chains(void* smem, int levels, int K, const int* start, const int* from)
{
    Chains c;
    c.K = K, c.levels = levels;
    c.segments = chain_segments(levels, K);
    c.seglen   = levels > 0 ? (levels + c.segments - 1) / c.segments : 1;
    c.par      = (u32)__cvta_generic_to_shared(smem);
    c.sel      = c.par + 2u * (u32)(levels * (K + 1));
    c.comp     = c.sel + 2u * (u32)(levels * K);
    c.entry    = c.comp + 2u * (u32)(c.segments * (K + 1));
    c.start    = (u32)__cvta_generic_to_shared(start);
    c.from     = (u32)__cvta_generic_to_shared(from);
    return c;
}
constexpr size_t kChainMaxSmem = 200 * 1024;

}  // namespace ftb200
