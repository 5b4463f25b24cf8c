// Error / version plumbing of the C ABI, curand state set-up and the runtime-argument
// normalisation kernels of the two sampling layers.
#include <curand_kernel.h>

#include "common.cuh"
#include "ftb200.h"

namespace ftb200 {

static thread_local std::string g_error;
static thread_local int         g_launches = 0;

void set_error(const std::string& msg)
{
    g_error = msg;
}
const char* get_error()
{
    return g_error.c_str();
}
void note_launch(int n)
{
    g_launches += n;
}
void reset_launch_count()
{
    g_launches = 0;
}

// curand_init(seed, 0, 0, &state[i]) per row, as kernels/sampling_topk_kernels.cu:32-55.
__global__ void curand_init_kernel(curandState_t* states, int n, unsigned long long seed,
                                   const unsigned long long* seeds)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        curand_init(seeds != nullptr ? seeds[i] : seed, 0, 0, &states[i]);
    }
}

__global__ void curand_peek_kernel(const curandState_t* states, int n, int n_draws, float* out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        curandState_t st = states[i];
        for (int d = 0; d < n_draws; ++d) {
            out[(size_t)d * n + i] = curand_uniform(&st);
        }
    }
}

// One row of the top-k layer's arguments, layers/sampling_layers/TopKSamplingLayer.cu:28-77
__device__ __forceinline__ void topk_args_row(int i, u32 top_k, u32* top_ks, int top_ks_size, float top_p, float* top_ps,
                                              int top_ps_size, uint8_t* skip_decode)
{
    u32   k = top_ks_size > 1 ? top_ks[i] : top_k;
    float p = top_ps_size > 1 ? top_ps[i] : top_p;
    if (k == 0 && p == 0.0f) {
        k = 1;
    }
    if (k > 0 && p == 0.0f) {
        p = 1.0f;
    }
    top_ks[i]      = k > 1024u ? 1024u : k;
    top_ps[i]      = p < 0.0f ? 0.0f : (p > 1.0f ? 1.0f : p);
    skip_decode[i] = k == 0 ? 1 : 0;
}
__global__ void setup_topk_args_kernel(int batch, u32 top_k, u32* top_ks, int top_ks_size, float top_p, float* top_ps,
                                       int top_ps_size, uint8_t* skip_decode)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < batch; i += gridDim.x * blockDim.x) {
        topk_args_row(i, top_k, top_ks, top_ks_size, top_p, top_ps, top_ps_size, skip_decode);
    }
}

// One row of the top-p layer's arguments, layers/sampling_layers/TopPSamplingLayer.cu:30-109
struct TopPArgs {
    u32             top_k;
    u32*            top_ks;
    int             top_ks_size;
    float           top_p;
    float*          top_ps;
    int             top_ps_size;
    uint8_t*        skip_decode;
    float*          initial_top_p;
    float*          top_p_decay_buf;
    const float*    top_p_decay;
    float*          top_p_min_buf;
    const float*    top_p_min;
    int32_t*        top_p_reset_ids_buf;
    const uint32_t* top_p_reset_ids;
};
__device__ __forceinline__ void topp_args_row(int i, const TopPArgs& A)
{
    u32   k = A.top_ks_size > 1 ? A.top_ks[i] : A.top_k;
    float p = A.top_ps_size > 1 ? A.top_ps[i] : A.top_p;
    if (k == 0 && p == 0.0f) {
        k = 1;
    }
    p                  = p < 0.0f ? 0.0f : (p > 1.0f ? 1.0f : p);
    A.top_ks[i]        = k;
    A.top_ps[i]        = p;
    A.skip_decode[i]   = k > 0 ? 1 : 0;
    A.initial_top_p[i] = p;
    float d            = A.top_p_decay == nullptr ? 1.0f : A.top_p_decay[i];
    if (d > 1.0f || d <= 0.0f) {
        d = 1.0f;
    }
    A.top_p_decay_buf[i] = d;
    float m              = A.top_p_min == nullptr ? 1e-6f : A.top_p_min[i];
    if (m > 1.0f || m <= 0.0f) {
        m = 0.5f;
    }
    A.top_p_min_buf[i]       = m;
    A.top_p_reset_ids_buf[i] = (int32_t)(A.top_p_reset_ids == nullptr ? -1 : A.top_p_reset_ids[i]);
}
__global__ void setup_topp_args_kernel(int batch, TopPArgs A)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < batch; i += gridDim.x * blockDim.x) {
        topp_args_row(i, A);
    }
}

// Everything a request's set-up does on the device, one thread per row: generators and arguments of both layers.
__global__ void setup_sampling_kernel(int batch, curandState_t* topk_states, curandState_t* topp_states, unsigned long long seed,
                                      const unsigned long long* seeds, u32 top_k, u32* top_ks, int top_ks_size, float top_p,
                                      float* top_ps, int top_ps_size, uint8_t* skip_decode, TopPArgs A)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < batch; i += gridDim.x * blockDim.x) {
        topk_args_row(i, top_k, top_ks, top_ks_size, top_p, top_ps, top_ps_size, skip_decode);
        if (A.top_ps != nullptr) {
            topp_args_row(i, A);
        }
        curandState_t st;
        curand_init(seeds != nullptr ? seeds[i] : seed, 0, 0, &st);
        // (the bytes a generator never reads are zero too: states can be compared whole)
        memset(&topk_states[i], 0, sizeof st);
        memset(&topp_states[i], 0, sizeof st);
        topk_states[i] = st;
        topp_states[i] = st;
    }
}

}  // namespace ftb200

using namespace ftb200;

extern "C" const char* ftb200_version(void)
{
    return "ftb200 0.1 (sm_100a)";
}

extern "C" const char* ftb200_last_error_string(void)
{
    return get_error();
}

extern "C" int ftb200_last_launch_count(void)
{
    return g_launches;
}

extern "C" int ftb200_curand_init(void* states, int n, unsigned long long seed, const unsigned long long* seeds,
                                  void* stream)
{
    if (states == nullptr || n < 0) {
        set_error("ftb200_curand_init: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (n == 0) {
        return FTB200_OK;
    }
    curand_init_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>((curandState_t*)states, n, seed, seeds);
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

extern "C" int ftb200_curand_peek_uniforms(const void* states, int n, int n_draws, float* out, void* stream)
{
    if (states == nullptr || out == nullptr || n < 0 || n_draws < 0) {
        set_error("ftb200_curand_peek_uniforms: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (n == 0 || n_draws == 0) {
        return FTB200_OK;
    }
    curand_peek_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
        (const curandState_t*)states, n, n_draws, out);
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

extern "C" int ftb200_setup_topk_runtime_args(int batch, uint32_t top_k, uint32_t* top_ks, int top_ks_size,
                                              float top_p, float* top_ps, int top_ps_size, uint8_t* skip_decode,
                                              void* stream)
{
    if (batch < 0 || top_ks == nullptr || top_ps == nullptr || skip_decode == nullptr) {
        set_error("ftb200_setup_topk_runtime_args: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (batch == 0) {
        return FTB200_OK;
    }
    int block = batch < 256 ? batch : 256;
    setup_topk_args_kernel<<<(batch + block - 1) / block, block, 0, (cudaStream_t)stream>>>(
        batch, top_k, top_ks, top_ks_size, top_p, top_ps, top_ps_size, skip_decode);
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

extern "C" int ftb200_setup_topp_runtime_args(int batch, uint32_t top_k, uint32_t* top_ks, int top_ks_size,
                                              float top_p, float* top_ps, int top_ps_size, uint8_t* skip_decode,
                                              float* initial_top_p, float* top_p_decay_buf, const float* top_p_decay,
                                              float* top_p_min_buf, const float* top_p_min,
                                              int32_t* top_p_reset_ids_buf, const uint32_t* top_p_reset_ids,
                                              void* stream)
{
    if (batch < 0 || top_ks == nullptr || top_ps == nullptr || skip_decode == nullptr || initial_top_p == nullptr
        || top_p_decay_buf == nullptr || top_p_min_buf == nullptr || top_p_reset_ids_buf == nullptr) {
        set_error("ftb200_setup_topp_runtime_args: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (batch == 0) {
        return FTB200_OK;
    }
    int block = batch < 256 ? batch : 256;
    const TopPArgs A{top_k,         top_ks,          top_ks_size, top_p,         top_ps,    top_ps_size,        skip_decode,
                     initial_top_p, top_p_decay_buf, top_p_decay, top_p_min_buf, top_p_min, top_p_reset_ids_buf, top_p_reset_ids};
    setup_topp_args_kernel<<<(batch + block - 1) / block, block, 0, (cudaStream_t)stream>>>(batch, A);
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}

extern "C" int ftb200_setup_sampling(const ftb200_setup_params* p)
{
    if (p == nullptr || p->batch < 0 || p->topk_states == nullptr || p->topp_states == nullptr || p->topk_ks == nullptr
        || p->topk_ps == nullptr || p->topk_skip == nullptr
        || (p->topp_ps != nullptr
            && (p->topp_ks == nullptr || p->topp_skip == nullptr || p->topp_initial == nullptr || p->topp_decay == nullptr
                || p->topp_min == nullptr || p->topp_reset_ids == nullptr))) {
        set_error("ftb200_setup_sampling: invalid argument");
        return FTB200_INVALID_ARG;
    }
    if (p->batch == 0) {
        return FTB200_OK;
    }
    const TopPArgs A{p->topp_top_k,   p->topp_ks,    p->top_ks_size, p->top_p,    p->topp_ps,   p->top_ps_size,    p->topp_skip,
                     p->topp_initial, p->topp_decay, p->top_p_decay, p->topp_min, p->top_p_min, p->topp_reset_ids, p->top_p_reset_ids};
    setup_sampling_kernel<<<(p->batch + 63) / 64, 64, 0, (cudaStream_t)p->stream>>>(
        p->batch, (curandState_t*)p->topk_states, (curandState_t*)p->topp_states, p->seed, p->seeds, p->topk_top_k, p->topk_ks,
        p->top_ks_size, p->top_p, p->topk_ps, p->top_ps_size, p->topk_skip, A);
    FTB_CUDA_CHECK(cudaGetLastError());
    return FTB200_OK;
}
