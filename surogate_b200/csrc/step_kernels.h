// Launch API of the optimizer step's scalar kernels (step_kernels.cu).
#pragma once
#include <cuda_runtime.h>

namespace sg {

struct StepHyper {
    float v[7];       // lr, beta1, beta2, eps, weight decay, bias corrections
    float max_norm;   // <= 0: no clipping
};
void count_targets(const int* targets, long long n, int ignore, float* out, cudaStream_t s);
void sum_partials(const float* partial, int split, int n, float* out, cudaStream_t s);   // out[0] = [0, split), out[1] = [split, n)
void step_hyper(const float* total, const StepHyper& h, float* hp, float* norm_out, cudaStream_t s);
void step_report(const float* loss_sum, const float* n_valid, const float* aux, const float* norm, const int* error_flag, float* out, cudaStream_t s);

}  // namespace sg
