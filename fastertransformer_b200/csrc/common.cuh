// Shared device helpers for the decode-sampling kernels (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <string>

namespace ftb200 {

typedef unsigned long long u64;
typedef unsigned int       u32;

// ---- error plumbing shared by the extern "C" entry points --------------------------------------
void        set_error(const std::string& msg);
const char* get_error();
void        note_launch(int n);
void        reset_launch_count();

#define FTB_CUDA_CHECK(expr)                                                                                           \
    do {                                                                                                               \
        cudaError_t e__ = (expr);                                                                                      \
        if (e__ != cudaSuccess) {                                                                                      \
            ftb200::set_error(std::string(#expr) + ": " + cudaGetErrorString(e__));                                    \
            return FTB200_CUDA_ERROR;                                                                                  \
        }                                                                                                              \
    } while (0)

// ---- order-preserving integer image of a float ---------------------------------------------------
// key(a) < key(b)  <=>  a < b   for all non-NaN a, b (with -0 < +0).
__device__ __forceinline__ u32 fkey(float x)
{
    u32 b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(u32 k)
{
    u32 b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(b);
}

// 16-byte read-only load that does not pollute L1.
__device__ __forceinline__ uint4 ld_nc_v4(const void* p)
{
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

// Add to a counter that is known to live in shared memory.  Through a plain pointer the compiler has to
// emit a generic-address atomic; this states the address space.
__device__ __forceinline__ void smem_add(u32* p, u32 v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"((u32)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

// The same on a 32-bit shared-memory address.
__device__ __forceinline__ void reds_add(u32 addr, u32 v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ u32 lds_u32(u32 addr)
{
    u32 v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void smem_or(u32* p, u32 v)
{
    asm volatile("red.shared.or.b32 [%0], %1;" ::"r"((u32)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
__device__ __forceinline__ u32 smem_cas(u32* p, u32 expect, u32 want)
{
    u32 old;
    asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;"
                 : "=r"(old)
                 : "r"((u32)__cvta_generic_to_shared(p)), "r"(expect), "r"(want)
                 : "memory");
    return old;
}

__device__ __forceinline__ uint2 ld_nc_v2(const void* p)
{
    uint2 r;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

// 16-byte asynchronous copy global -> shared (both 16-byte aligned), past L1.
__device__ __forceinline__ void cp_async16(u32 smem, const void* g)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template<int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void sts_u32(u32 a, u32 v)
{
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts_u16(u32 a, u32 v)
{
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((unsigned short)v) : "memory");
}

// A launch whose blocks may come up while the kernel in front of it in the stream drains; the kernel calls
// wait_for_previous() before it touches memory, which returns when that one has ended.  Hides the launch of a short kernel
// (steps follow each other in a stream: 1 to 2 us each).
template<class... P, class... A>
inline cudaError_t launch_early(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args)
{
    cudaLaunchConfig_t  cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim          = grid;
    cfg.blockDim         = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = st;
    cfg.attrs            = attr;
    cfg.numAttrs         = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
// The blocks of a launch behind this kernel that allows for it may come up from here on, where they would else come up when the last
// block of this one has gone.  (Not worth saying everywhere: beam rows and merge, 64 x 4 x 32000, took 23.9 us so and 19.9 without; the
// general kernel, the gather tree and the log-probabilities the same either way.)
__device__ __forceinline__ void let_next_come_up()
{
    asm volatile("griddepcontrol.launch_dependents;");
}
__device__ __forceinline__ void wait_for_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void store_release(u32* p, u32 v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ u32 load_acquire(const u32* p)
{
    u32 v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Tells the compiler that a pointer loaded from a structure points into shared memory, so that it emits
// ld.shared / st.shared instead of generic accesses (every pointer of the kernel's shared-memory map qualifies).
#define FTB_ASSUME_SHARED(p) __builtin_assume(__isShared(p))

// ---- word lists -----------------------------------------------------------------------------------
// A word list is [2, L]: row 0 the concatenated token ids, row 1 the exclusive end offset of each word,
// padded with -1.  Returns true when word `i` matches the tail of the sequence ending at position
// `last` (inclusive) of column `col`, following parent_ids for beams.
// kernels/ban_bad_words.cu:49-75 (n_match = size-1, last = step-1) and
// kernels/stop_criteria_kernels.cu:53-75 (n_match = size, last = step).
__device__ __forceinline__ bool tail_matches(const int* ids, const int* parents, const int* words, int item_start,
                                             int n_match, int first_pos, size_t row_stride, size_t col_base,
                                             int beam_idx, int beam_width)
{
    int parent = beam_idx;
    for (int t = n_match - 1; t >= 0; --t) {
        const size_t at = (size_t)(first_pos + t) * row_stride + col_base + parent;
        if (ids[at] != words[item_start + t]) {
            return false;
        }
        if (beam_width > 1) {
            parent = parents[at];
            if (parent < 0 || parent >= beam_width) {
                return false;
            }
        }
    }
    return true;
}

// ---- in-place ascending sort of u64 keys by a cooperating thread group ---------------------------
// Bitonic network in its "all ascending" form (first sub-step of every merge compares mirrored
// positions), which tolerates any n: positions >= n behave as +infinity and are never touched.
// `sync` is __syncthreads for a whole CTA or __syncwarp for one warp.
template<class Sync, bool SMEM = false>
__device__ __forceinline__ void group_sort_u64(u64* a, int n, int tid, int nthr, Sync sync)
{
    if (SMEM) {
        FTB_ASSUME_SHARED(a);
    }
    if (n < 2) {
        return;
    }
    int np = 1;
    while (np < n) {
        np <<= 1;
    }
    const int half = np >> 1;
    for (int k = 2; k <= np; k <<= 1) {
        const int hk = k >> 1;
        for (int i = tid; i < half; i += nthr) {
            int l = (i / hk) * k + (i % hk);
            int h = l ^ (k - 1);
            if (h < n) {
                u64 x = a[l], y = a[h];
                if (x > y) {
                    a[l] = y;
                    a[h] = x;
                }
            }
        }
        sync();
        for (int j = k >> 2; j > 0; j >>= 1) {
            for (int i = tid; i < half; i += nthr) {
                int l = 2 * i - (i & (j - 1));
                int h = l + j;
                if (h < n) {
                    u64 x = a[l], y = a[h];
                    if (x > y) {
                        a[l] = y;
                        a[h] = x;
                    }
                }
            }
            sync();
        }
    }
}

struct CtaSync {
    __device__ __forceinline__ void operator()() const
    {
        __syncthreads();
    }
};
struct WarpSync {
    __device__ __forceinline__ void operator()() const
    {
        __syncwarp();
    }
};

}  // namespace ftb200
