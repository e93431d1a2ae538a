// The scalars of an optimizer step: target count and loss scale, gradient norm, clip factor and hyper-parameter vector, and the record that
// the host reads back.  Each replaces a chain of one-element tensor operations; a small training step is bound by its launches (about
// 5 us of host time each), and these chains were a third of them.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "step_kernels.h"

namespace sg {

constexpr int STEP_THREADS = 1024;

template <typename T> __device__ __forceinline__ T block_sum(T v) {
    __shared__ T sh[STEP_THREADS / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = sh[threadIdx.x & 31];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// out[0] = number of targets that are not `ignore`, out[1] = 1 / max(out[0], 1).  One block: 16 K targets take a few us.
__global__ void __launch_bounds__(STEP_THREADS) count_targets_kernel(const int* __restrict__ targets, long long n, int ignore, float* __restrict__ out) {
    long long c = 0;
    for (long long i = threadIdx.x; i < n; i += STEP_THREADS) c += targets[i] != ignore;
    c = block_sum(c);
    if (threadIdx.x == 0) {
        const float f = static_cast<float>(c);
        out[0] = f;
        out[1] = 1.f / fmaxf(f, 1.f);
    }
}

// out[0] = sum of partial[0, split), out[1] = sum of partial[split, n)
__global__ void __launch_bounds__(STEP_THREADS) sum_partials_kernel(const float* __restrict__ partial, int split, int n, float* __restrict__ out) {
    const int lo = blockIdx.x == 0 ? 0 : split, hi = blockIdx.x == 0 ? split : n;
    float s = 0.f;
    for (int i = lo + threadIdx.x; i < hi; i += STEP_THREADS) s += partial[i];
    s = block_sum(s);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// hp = [lr, beta1, beta2, eps, weight decay, bias correction 1, 2, clip factor]; norm = sqrt(total).  The clip factor is
// min(max_norm / (norm + 1e-6), 1), 1 without a limit, and 0 (the update is skipped) when the norm is not finite.
__global__ void step_hyper_kernel(const float* __restrict__ total, StepHyper h, float* __restrict__ hp, float* __restrict__ norm_out) {
    const float norm = sqrtf(*total);
    float clip = 1.f;
    if (h.max_norm > 0.f) clip = fminf(h.max_norm / (norm + 1e-6f), 1.f);
    if (!(fabsf(norm) < CUDART_INF_F)) clip = 0.f;
    for (int i = 0; i < 7; ++i) hp[i] = h.v[i];
    hp[7] = clip;
    *norm_out = norm;
}

// out = [loss_sum / max(n_valid, 1) + aux, norm, aux, error flag]
__global__ void step_report_kernel(const float* __restrict__ loss_sum, const float* __restrict__ n_valid, const float* __restrict__ aux, const float* __restrict__ norm,
                                   const int* __restrict__ error_flag, float* __restrict__ out) {
    out[0] = *loss_sum / fmaxf(*n_valid, 1.f) + *aux;
    out[1] = *norm;
    out[2] = *aux;
    out[3] = static_cast<float>(*error_flag);
}

void count_targets(const int* targets, long long n, int ignore, float* out, cudaStream_t s) { count_targets_kernel<<<1, STEP_THREADS, 0, s>>>(targets, n, ignore, out); }
void sum_partials(const float* partial, int split, int n, float* out, cudaStream_t s) { sum_partials_kernel<<<2, STEP_THREADS, 0, s>>>(partial, split, n, out); }
void step_hyper(const float* total, const StepHyper& h, float* hp, float* norm_out, cudaStream_t s) { step_hyper_kernel<<<1, 1, 0, s>>>(total, h, hp, norm_out); }
void step_report(const float* loss_sum, const float* n_valid, const float* aux, const float* norm, const int* error_flag, float* out, cudaStream_t s) {
    step_report_kernel<<<1, 1, 0, s>>>(loss_sum, n_valid, aux, norm, error_flag, out);
}

}  // namespace sg
