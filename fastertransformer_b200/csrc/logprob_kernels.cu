// Log-probabilities of given token ids under the soft-max of context logits, summed per sequence.
// Replaces invokeLogProbFromLogits (kernels/logprob_kernels.cu:142-183): log_probs_kernel (:36-103) and
// accumulate_log_probs (:105-140).
//
// The reference reads every row twice (maximum, then sum of exponentials) with one 1024-thread block per
// (step, sequence).  Here a row is read once with 16-byte loads, each thread keeping a running
// (maximum, scaled sum) pair that is merged across the block at the end, and a fixed grid of 8 CTAs per SM
// walks the rows.  Both kernels are bound by HBM: vocab * sizeof(T) bytes per counted (step, sequence).
#include "common.cuh"
#include "ftb200.h"

namespace ftb200 {

namespace {

// 16-bit rows want every warp that fits (the exponentials alone take 137 of 188 us): 4 CTAs of 256 threads 254 us, 6 CTAs 243,
// 8 CTAs 222; 8 loads in flight instead of 4 change nothing there.
constexpr int   kLpThreads = 256;
constexpr int   kLpCtas    = 8;   // per SM
constexpr int   kLpLoads   = 4;   // 16-byte loads in flight per thread
constexpr float kLog2e     = 1.4426950408889634f;

template<typename T>
struct LpType;
template<>
struct LpType<float> {
    static constexpr int   kPerVec = 4;
    __device__ static float maximum(const uint4&, const float* x)
    {
        return fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
    }
    static constexpr float kLowest = -FLT_MAX;
    __device__ static float get(const float* p) { return *p; }
    __device__ static void  unpack(const uint4& v, float* x)
    {
        x[0] = __uint_as_float(v.x);
        x[1] = __uint_as_float(v.y);
        x[2] = __uint_as_float(v.z);
        x[3] = __uint_as_float(v.w);
    }
};
template<>
struct LpType<__half> {
    static constexpr int   kPerVec = 8;
    __device__ static float maximum(const uint4& v, const float*)
    {
        const __half2* h = reinterpret_cast<const __half2*>(&v);
        const float2   m = __half22float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
        return fmaxf(m.x, m.y);
    }
    static constexpr float kLowest = -65504.0f;  // the reference starts the maximum at -HALF_FLT_MAX (:58-59)
    __device__ static float get(const __half* p) { return __half2float(*p); }
    __device__ static void  unpack(const uint4& v, float* x)
    {
        const u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
            x[2 * i]       = f.x;
            x[2 * i + 1]   = f.y;
        }
    }
};
template<>
struct LpType<__nv_bfloat16> {
    static constexpr int   kPerVec = 8;
    __device__ static float maximum(const uint4& v, const float*)
    {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
        const float2          m = __bfloat1622float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
        return fmaxf(m.x, m.y);
    }
    static constexpr float kLowest = -FLT_MAX;
    __device__ static float get(const __nv_bfloat16* p) { return __bfloat162float(*p); }
    __device__ static void  unpack(const uint4& v, float* x)
    {
        const u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[2 * i]     = __uint_as_float(w[i] << 16);
            x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

// (m, s) stands for s * exp(m): the sum of exp(x) over the elements seen so far, with m their maximum
// (or the type's lowest value when nothing larger was seen, as in the reference).
struct MaxSum {
    float m, s;
};

__device__ __forceinline__ float fast_exp(float d)
{
    return exp2f(d * kLog2e);  // __expf under the reference's fast-math build
}

__device__ __forceinline__ void add_plain(MaxSum& a, float x)
{
    if (x > a.m) {
        a.s = a.s * fast_exp(a.m - x) + 1.0f;
        a.m = x;
    }
    else {
        a.s += fast_exp(x - a.m);
    }
}

__device__ __forceinline__ MaxSum merge(const MaxSum& a, const MaxSum& b)
{
    const float m = fmaxf(a.m, b.m);
    return {m, a.s * fast_exp(a.m - m) + b.s * fast_exp(b.m - m)};
}

__device__ __forceinline__ void add_plain_vec(MaxSum& a, const uint4& v)
{
    constexpr int N = LpType<float>::kPerVec;
    float         x[N];
    LpType<float>::unpack(v, x);
    const float vm = LpType<float>::maximum(v, x);
    if (vm > a.m) {
        a.s *= fast_exp(a.m - vm);
        a.m = vm;
    }
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        t += fast_exp(x[i] - a.m);
    }
    a.s += t;
}

// ---- 16-bit rows ------------------------------------------------------------------------------------------------
// Two logits per instruction where that exists (packed fp32 fused multiply-add and add): the exponent of a term is one fused
// multiply-add, x * log2(e) - m2 with m2 = m * log2(e) as it was rounded, and what that rounding lost, m * log2(e) - m2, is the
// same for all terms and comes off the sum at the end.  Half of the instructions of a subtract, a multiply, an exponential
// and an add a logit: 512 x 32 x 50257 half 238 -> 232 us (256 -> 249 on a warmer card).  Every fourth exponential by a polynomial
// on the multiply-add pipes instead of the special-function unit was slower (242, half of them 278).
__device__ __forceinline__ u64 pack2(float a, float b)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
    u64 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
    u64 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The sum of the two halves of s, times 2^m2, is the sum of exp(x) so far.  That wants a small d = m * log2(e) - m2: the terms
// are 2^d times what they stand for, and total() takes that off with two terms of the series.  d is half a unit of m2's last
// place, up to 2^-8 for the largest half (of the third term 3e-9 is left); bf16 reaches further, and a thread whose columns are all
// masked with -1e10 so far has it for its maximum, with a d of hundreds.  From kBeyond on a bf16 maximum has no m2: s stands
// for s * exp(m), by exact differences.  Values of bf16 on both sides of the line are 32 and more apart, so that going from one
// form to the other scales the sum by e^-32 at most, and 2^d, within 2^-11 of 1, is no part of it.
template<typename T>
struct PairSum {
    float m, m2;
    u64   s;
    static constexpr bool  kWide   = sizeof(T) == 2 && LpType<T>::kLowest < -65504.0f;
    static constexpr float kBeyond = 8192.0f;
    __device__ static bool beyond(float m) { return kWide && !(fabsf(m) < kBeyond); }
    __device__ void        start()
    {
        m = LpType<T>::kLowest, m2 = m * kLog2e, s = 0;
    }
    // the sum with `to` >= m as its maximum
    __device__ void raise(float to)
    {
        const float to2 = to * kLog2e;
        const float f   = beyond(m) || beyond(to) ? fast_exp(m - to) : exp2f(m2 - to2);
        float       a, b;
        unpack2(s, a, b);
        s = pack2(a * f, b * f);
        m = to, m2 = to2;
    }
    __device__ void add_one(float x)
    {
        if (x > m) {
            raise(x);
        }
        s = add2(s, pack2(beyond(m) ? fast_exp(x - m) : exp2f(fmaf(x, kLog2e, -m2)), 0.0f));
    }
    __device__ void add_vec(const uint4& v)
    {
        float x[8];
        LpType<T>::unpack(v, x);
        const float vm = LpType<T>::maximum(v, x);
        if (vm > m) {
            raise(vm);
        }
        if (beyond(m)) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                s = add2(s, pack2(fast_exp(x[i] - m), 0.0f));
            }
            return;
        }
        const u64 l = pack2(kLog2e, kLog2e), o = pack2(-m2, -m2);
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            float a, b;
            unpack2(fma2(pack2(x[i], x[i + 1]), l, o), a, b);
            s = add2(s, pack2(exp2f(a), exp2f(b)));
        }
    }
    __device__ MaxSum total() const
    {
        float a, b;
        unpack2(s, a, b);
        const float d = fmaf(m, kLog2e, -m2);  // 2^-d = 1 - d ln 2 + (d ln 2)^2 / 2 - ...
        return {m, beyond(m) ? a + b : (a + b) * fmaf(d, fmaf(d, 0.24022651f, -0.69314718f), 1.0f)};
    }
};
// fp32 rows: at the copy rate with the plain form
struct PlainSum {
    MaxSum          a;
    __device__ void start() { a = {LpType<float>::kLowest, 0.0f}; }
    __device__ void add_one(float x) { add_plain(a, x); }
    __device__ void add_vec(const uint4& v) { add_plain_vec(a, v); }
    __device__ MaxSum total() const { return a; }
};
template<typename T>
struct RowSum {
    using type = PairSum<T>;
};
template<>
struct RowSum<float> {
    using type = PlainSum;
};

// One CTA per (step, sequence) row at a time.  Rows past a sequence's length are skipped without a read.
//
// The counted rows are dealt out evenly: every CTA adds up the sequences' counts and takes each gridDim-th of the counted
// rows.  With the rows of the whole [step, sequence] array dealt out instead, the skipped ones included, 1184 CTAs and 32
// sequences gave a CTA the same sequence every time (512 x 32 x 50257 half, lengths spread over 256 .. 512: 14 rows for
// some, 7 for others, and the 10.4 of the average took as long as 14: 254 us, now 222).  A batch of more sequences than the
// table holds keeps that deal; no sequence is a large part of it.
constexpr int kLpMaxSeq = 1024;
template<typename T>
__global__ void __launch_bounds__(kLpThreads, kLpCtas) context_log_probs_kernel(float* log_probs, const T* logits,
                                                                        const int* ids, const int* lengths,
                                                                        int max_len, int batch, int vocab,
                                                                        size_t vocab_padded, int batch_first,
                                                                        long long rows)
{
    wait_for_previous();
    constexpr int N = LpType<T>::kPerVec;
    __shared__ MaxSum s_part[kLpThreads / 32];
    const int         tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int         steps = max_len - 1;
    __shared__ int    s_end[kLpMaxSeq];  // counted rows of the sequences up to and with this one
    const bool        dealt = batch <= kLpMaxSeq && rows <= 0x7fffffff;
    if (dealt) {
        constexpr int  PER = kLpMaxSeq / kLpThreads;
        __shared__ int s_warp[kLpThreads / 32];
        int            c[PER], sum = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int b = tid * PER + i;
            sum += b < batch ? max(0, min(lengths[b] - 1, steps)) : 0;
            c[i] = sum;
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, incl, o);
            incl += lane >= o ? x : 0;
        }
        if (lane == 31) {
            s_warp[wid] = incl;
        }
        __syncthreads();
        int before = incl - sum;
        for (int w = 0; w < wid; ++w) {
            before += s_warp[w];
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            s_end[tid * PER + i] = before + c[i];
        }
        __syncthreads();
        rows = s_end[kLpMaxSeq - 1];
    }

    for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
        int step, b;
        if (dealt) {
            int lo = 0, hi = batch - 1;  // the first sequence that ends after row r
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_end[mid] > r) {
                    hi = mid;
                }
                else {
                    lo = mid + 1;
                }
            }
            b    = lo;
            step = (int)(r - (lo > 0 ? s_end[lo - 1] : 0));
        }
        else if (batch_first) {
            b    = (int)(r / steps);
            step = (int)(r % steps);
        }
        else {
            step = (int)(r / batch);
            b    = (int)(r % batch);
        }
        if (step >= lengths[b] - 1) {
            continue;
        }
        const size_t row_idx = batch_first ? (size_t)b * max_len + step : (size_t)step * batch + b;
        const T*     row     = logits + row_idx * vocab_padded;

        typename RowSum<T>::type sum;
        sum.start();
        // Scalars up to the first 16-byte boundary, 16-byte vectors, scalars after the last full vector.
        const int mis  = (int)((reinterpret_cast<uintptr_t>(row) & 15) / sizeof(T));
        const int head = min(vocab, mis ? N - mis : 0);
        const int nvec = (vocab - head) / N;
        if (tid < head) {
            sum.add_one(LpType<T>::get(row + tid));
        }
        const uint4* vp = reinterpret_cast<const uint4*>(row + head);
        int          i  = tid;
        for (; i + (kLpLoads - 1) * kLpThreads < nvec; i += kLpLoads * kLpThreads) {
            uint4 v[kLpLoads];
#pragma unroll
            for (int u = 0; u < kLpLoads; ++u) {
                v[u] = ld_nc_v4(vp + i + u * kLpThreads);
            }
#pragma unroll
            for (int u = 0; u < kLpLoads; ++u) {
                sum.add_vec(v[u]);
            }
        }
        for (; i < nvec; i += kLpThreads) {
            sum.add_vec(ld_nc_v4(vp + i));
        }
        const int tail0 = head + nvec * N;
        if (tail0 + tid < vocab) {  // fewer than N <= 8 elements remain
            sum.add_one(LpType<T>::get(row + tail0 + tid));
        }
        MaxSum acc = sum.total();

#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            MaxSum other{__shfl_xor_sync(0xffffffffu, acc.m, o), __shfl_xor_sync(0xffffffffu, acc.s, o)};
            acc = merge(acc, other);
        }
        if (lane == 0) {
            s_part[wid] = acc;
        }
        __syncthreads();
        if (tid == 0) {
            MaxSum tot = s_part[0];
#pragma unroll
            for (int w = 1; w < kLpThreads / 32; ++w) {
                tot = merge(tot, s_part[w]);
            }
            const size_t out = batch_first ? (size_t)b * steps + step : (size_t)step * batch + b;
            const size_t tok = batch_first ? (size_t)b * max_len + step + 1 : (size_t)(step + 1) * batch + b;
            const int    id  = ids[tok];
            // The reference reads logits[id] unchecked; an id outside the padded row gives NaN here.
            const float x = (id >= 0 && (size_t)id < vocab_padded) ? LpType<T>::get(row + id) : NAN;
            log_probs[out] = x - tot.m - __logf(tot.s + 1e-9f);
        }
        __syncthreads();
    }
}

// cum_log_probs[b] = sum over step < lengths[b] - 1 of log_probs[step, b], in a fixed order.
__global__ void __launch_bounds__(kLpThreads) sum_log_probs_kernel(float* cum, const float* log_probs,
                                                                    const int* lengths, int max_len, int batch,
                                                                    int batch_first)
{
    wait_for_previous();
    __shared__ float s_part[kLpThreads / 32];
    const int        b = blockIdx.x, tid = threadIdx.x;
    const int        n = min(lengths[b], max_len) - 1;
    const float*     p = log_probs + (batch_first ? (size_t)b * (max_len - 1) : (size_t)b);
    const size_t     stride = batch_first ? 1 : (size_t)batch;
    float            acc = 0.0f;
    for (int step = tid; step < n; step += kLpThreads) {
        acc += p[(size_t)step * stride];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if ((tid & 31) == 0) {
        s_part[tid >> 5] = acc;
    }
    __syncthreads();
    if (tid == 0) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < kLpThreads / 32; ++w) {
            t += s_part[w];
        }
        cum[b] = t;
    }
}

template<typename T>
int launch_log_probs(float* cum, const void* logits, const int* ids, const int* lengths, size_t max_len,
                     size_t batch, size_t vocab, size_t vocab_padded, float* log_probs, cudaStream_t st,
                     int batch_first)
{
    // (asked per call: the attribute query is a host-side table look-up, and a process may drive several devices)
    int n_sm = 0, dev = 0;
    FTB_CUDA_CHECK(cudaGetDevice(&dev));
    FTB_CUDA_CHECK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    const long long rows = (long long)(max_len - 1) * (long long)batch;
    if (rows > 0) {
        const int grid = (int)std::min<long long>(rows, (long long)n_sm * kLpCtas);
        FTB_CUDA_CHECK(launch_early(context_log_probs_kernel<T>, dim3((unsigned)grid), dim3(kLpThreads), 0, st, log_probs,
                                    (const T*)logits, ids, lengths, (int)max_len, (int)batch, (int)vocab, vocab_padded, batch_first, rows));
        FTB_CUDA_CHECK(cudaGetLastError());
        note_launch(1);
    }
    FTB_CUDA_CHECK(launch_early(sum_log_probs_kernel, dim3((unsigned)batch), dim3(kLpThreads), 0, st, cum, log_probs, lengths, (int)max_len,
                                (int)batch, batch_first));
    FTB_CUDA_CHECK(cudaGetLastError());
    note_launch(1);
    return FTB200_OK;
}

}  // namespace
}  // namespace ftb200

using namespace ftb200;

extern "C" int ftb200_log_prob_from_logits(float* cum_log_probs, const void* logits, int dtype,
                                           const int* input_ids, const int* input_lengths,
                                           size_t max_input_length, size_t batch_size, size_t vocab_size,
                                           size_t vocab_size_padded, void* workspace, size_t workspace_size,
                                           void* stream, int batch_first)
{
    if (cum_log_probs == nullptr || logits == nullptr || input_ids == nullptr || input_lengths == nullptr
        || max_input_length == 0 || batch_size == 0 || vocab_size == 0 || vocab_size > vocab_size_padded
        || max_input_length > 0x7fffffffu || batch_size > 0x7fffffffu || vocab_size_padded > 0x7fffffffu) {
        set_error("ftb200_log_prob_from_logits: invalid argument");
        return FTB200_INVALID_ARG;
    }
    // The reference asserts this bound (logprob_kernels.cu:169); it holds one float per (step, sequence).
    if (workspace == nullptr || workspace_size < sizeof(float) * max_input_length * batch_size) {
        set_error("ftb200_log_prob_from_logits: workspace below sizeof(float) * max_input_length * batch_size");
        return FTB200_WORKSPACE_SMALL;
    }
    cudaStream_t st = (cudaStream_t)stream;
    float*       lp = (float*)workspace;
    switch (dtype) {
        case FTB200_F32:
            return launch_log_probs<float>(cum_log_probs, logits, input_ids, input_lengths, max_input_length,
                                           batch_size, vocab_size, vocab_size_padded, lp, st, batch_first);
        case FTB200_F16:
            return launch_log_probs<__half>(cum_log_probs, logits, input_ids, input_lengths, max_input_length,
                                            batch_size, vocab_size, vocab_size_padded, lp, st, batch_first);
        case FTB200_BF16:
            return launch_log_probs<__nv_bfloat16>(cum_log_probs, logits, input_ids, input_lengths,
                                                   max_input_length, batch_size, vocab_size, vocab_size_padded, lp,
                                                   st, batch_first);
        default:
            set_error("ftb200_log_prob_from_logits: unknown dtype");
            return FTB200_INVALID_ARG;
    }
}
