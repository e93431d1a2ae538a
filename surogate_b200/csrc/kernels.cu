// Memory-bound training kernels for sm_100a: RMSNorm (+residual, +FP8 output) fwd/bwd, QK-norm + RoPE
// fwd/bwd on packed QKV, SwiGLU fwd/bwd (+FP8 output), embedding fwd/bwd, softmax cross-entropy fwd+bwd in
// place, FP8 quantise / abs-max, sum of squares, AdamW (fp32 state and 8-bit state).
// All loads/stores are 16-byte vectors; reductions are warp shuffles + one shared-memory hop.
//
// Replaces csrc/src/kernels/{rmsnorm,qk_norm,rope,swiglu,encoder,fused_classifier,global_norm}.cu,
// recipes/fp8_hybrid/kernels/quant.cu and runtime/optimizers/{adamw,flash_adamw_8bit}.cu of the reference.
#include <cstdlib>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "launch_limits.h"
#include "sm100_ptx.cuh"

namespace sg {

using bf16 = __nv_bfloat16;
using bf162 = __nv_bfloat162;

struct alignas(16) Vec8 { bf162 v[4]; };

__device__ __forceinline__ void load8(const bf16* p, float (&f)[8]) {
    const Vec8 t = *reinterpret_cast<const Vec8*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 x = __bfloat1622float2(t.v[i]); f[2 * i] = x.x; f[2 * i + 1] = x.y; }
}
__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
    const bf162* t = reinterpret_cast<const bf162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 x = __bfloat1622float2(t[i]); f[2 * i] = x.x; f[2 * i + 1] = x.y; }
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
    Vec8 t;
#pragma unroll
    for (int i = 0; i < 4; ++i) t.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *reinterpret_cast<Vec8*>(p) = t;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <bool IS_MAX> __device__ __forceinline__ float block_reduce(float v, float* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = IS_MAX ? warp_max(v) : warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    v = (lane < nw) ? sh[lane] : (IS_MAX ? -INFINITY : 0.f);
    v = IS_MAX ? warp_max(v) : warp_sum(v);
    return v;
}
__device__ __forceinline__ void atomic_max_pos(float* addr, float v) {
    if (v > 0.f) atomicMax(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}

// eight values times `s` as FP8, two to a conversion instruction
template <bool E5M2> __device__ __forceinline__ uint2 to_fp8x8(const float (&a)[8], float s) {
    uint2 o;
    __nv_fp8x2_storage_t* ob = reinterpret_cast<__nv_fp8x2_storage_t*>(&o);
#pragma unroll
    for (int i = 0; i < 4; ++i) ob[i] = __nv_cvt_float2_to_fp8x2(make_float2(a[2 * i] * s, a[2 * i + 1] * s), __NV_SATFINITE, E5M2 ? __NV_E5M2 : __NV_E4M3);
    return o;
}

// ------------------------------------------------------------------------------------------ RMSNorm forward
// One CTA per row.  res_out = residual + x (optional) ; y = res_out * rstd * w ; optionally y also as FP8.
// ITERS > 0: the row (C <= blockDim * 8 * ITERS) stays in registers as packed bf16 between the sum and the scaling, with all its loads and
// those of w in flight together; ITERS = 0 (wider rows) reads it again.
// With the residual on B200: 16384 x 1024 37 -> 27 us, 8192 x 4096 64 -> 48 us (FP8 output 60 -> 44), 8192 x 5120 78 -> 64 us.
template <int ITERS>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ residual, const bf16* __restrict__ w,
                                                          bf16* __restrict__ res_out, bf16* __restrict__ y, float* __restrict__ rstd_out,
                                                          uint8_t* __restrict__ y_fp8, const float* __restrict__ fp8_scale, float* __restrict__ amax_out,
                                                          int C, float eps) {
    __shared__ float sh[32];
    constexpr int N = ITERS > 0 ? ITERS : 1;
    const size_t row = blockIdx.x;
    const bf16* xr = x + row * C;
    const bf16* rr = residual ? residual + row * C : nullptr;
    bf16* ro = res_out ? res_out + row * C : nullptr;
    const int step = blockDim.x * 8;
    float ss = 0.f;
    uint4 xk[N], rk[N], wk[N];
    auto add_residual = [&](uint4 xv, uint4 rv) {   // rounded to the stored precision, so that forward and backward see the same residual stream
        float a[8], b[8];
        unpack8(xv, a);
        unpack8(rv, b);
        uint4 o;
        bf162* po = reinterpret_cast<bf162*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) po[i] = __floats2bfloat162_rn(a[2 * i] + b[2 * i], a[2 * i + 1] + b[2 * i + 1]);
        return o;
    };
    auto square = [&](const uint4& v) {
        float a[8];
        unpack8(v, a);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += a[i] * a[i];
    };
    if (ITERS > 0) {
#pragma unroll
        for (int it = 0; it < N; ++it) {
            const int c = threadIdx.x * 8 + it * step;
            if (c < C) {
                xk[it] = *reinterpret_cast<const uint4*>(xr + c);
                if (rr) rk[it] = *reinterpret_cast<const uint4*>(rr + c);
                wk[it] = *reinterpret_cast<const uint4*>(w + c);
            }
        }
#pragma unroll
        for (int it = 0; it < N; ++it) {
            const int c = threadIdx.x * 8 + it * step;
            if (c < C) {
                if (rr) {
                    xk[it] = add_residual(xk[it], rk[it]);
                    *reinterpret_cast<uint4*>(ro + c) = xk[it];
                }
                square(xk[it]);
            }
        }
    } else {
        for (int c = threadIdx.x * 8; c < C; c += step) {
            uint4 v = *reinterpret_cast<const uint4*>(xr + c);
            if (rr) {
                v = add_residual(v, *reinterpret_cast<const uint4*>(rr + c));
                *reinterpret_cast<uint4*>(ro + c) = v;
            }
            square(v);
        }
    }
    ss = block_reduce<false>(ss, sh);
    const float rstd = rsqrtf(ss / C + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
    const float qs = fp8_scale ? __ldg(fp8_scale) : 1.f;
    float amax = 0.f;
    auto scale_out = [&](int c, const uint4& v, const uint4& wv) {
        float a[8], g[8];
        unpack8(v, a);
        unpack8(wv, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) { a[i] = a[i] * rstd * g[i]; amax = fmaxf(amax, fabsf(a[i])); }
        if (y) store8(y + row * C + c, a);
        if (y_fp8) *reinterpret_cast<uint2*>(y_fp8 + row * C + c) = to_fp8x8<false>(a, qs);
    };
    if (ITERS > 0) {
#pragma unroll
        for (int it = 0; it < N; ++it) {
            const int c = threadIdx.x * 8 + it * step;
            if (c < C) scale_out(c, xk[it], wk[it]);
        }
    } else {
        const bf16* src = rr ? ro : xr;
        for (int c = threadIdx.x * 8; c < C; c += step) scale_out(c, *reinterpret_cast<const uint4*>(src + c), *reinterpret_cast<const uint4*>(w + c));
    }
    if (amax_out) {
        amax = block_reduce<true>(amax, sh);
        if (threadIdx.x == 0) atomic_max_pos(amax_out, amax);
    }
}

// ------------------------------------------------------------------------------------------ RMSNorm backward
// Persistent CTAs stride over rows; each thread owns fixed columns and keeps dw partial sums in registers.
// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ d_res) ; dw_partial[block, C] reduced by a second kernel.
// ITERS = 8-element vectors per thread (C <= blockDim * 8 * ITERS).  The block size follows C (128 threads up to C = 1024, else
// 256) so that no thread idles on narrow rows, and the number of CTAs follows the register budget: narrow rows run many small
// CTAs per SM, which is what hides the two dependent passes (dot product, then dx) of each row.  With ITERS <= 2 the row stays in
// registers between the passes instead of being read again.
constexpr int RB_THREADS = 256;
template <int ITERS>
__global__ void __launch_bounds__(RB_THREADS) rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                                 const float* __restrict__ rstd, const bf16* __restrict__ d_res,
                                                                 bf16* __restrict__ dx, float* __restrict__ dw_partial, int rows, int C) {
    constexpr bool KEEP = ITERS <= 2;
    __shared__ float sh[32];
    float dw[ITERS][8];
    float ww[ITERS][8];
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int c = (it * blockDim.x + threadIdx.x) * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) { dw[it][i] = 0.f; ww[it][i] = 0.f; }
        if (c < C) load8(w + c, ww[it]);
    }
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const size_t base = static_cast<size_t>(row) * C;
        const float rs = rstd[row];
        float dot = 0.f;
        // the row stays in registers as packed bf16 between the two passes (KEEP), and the incoming residual gradient is requested
        // together with dy and x, so that its latency hides behind the block reduction instead of following it
        uint4 gk[KEEP ? ITERS : 1], ak[KEEP ? ITERS : 1], rk[KEEP ? ITERS : 1];
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            const int c = (it * blockDim.x + threadIdx.x) * 8;
            if (c < C) {
                const uint4 graw = *reinterpret_cast<const uint4*>(dy + base + c);
                const uint4 araw = *reinterpret_cast<const uint4*>(x + base + c);
                if (KEEP) {
                    gk[it] = graw;
                    ak[it] = araw;
                    if (d_res) rk[it] = *reinterpret_cast<const uint4*>(d_res + base + c);
                }
                float g[8], a[8];
                unpack8(graw, g);
                unpack8(araw, a);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float xhat = a[i] * rs;
                    dot += g[i] * ww[it][i] * xhat;
                    dw[it][i] += g[i] * xhat;
                }
            }
        }
        dot = block_reduce<false>(dot, sh) / C;
#pragma unroll
        for (int it = 0; it < ITERS; ++it) {
            const int c = (it * blockDim.x + threadIdx.x) * 8;
            if (c < C) {
                float g[8], a[8], o[8];
                if (KEEP) {
                    unpack8(gk[it], g);
                    unpack8(ak[it], a);
                } else {
                    load8(dy + base + c, g);
                    load8(x + base + c, a);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = rs * (g[i] * ww[it][i] - a[i] * rs * dot);
                if (d_res) {
                    float r[8];
                    if (KEEP) unpack8(rk[it], r);
                    else load8(d_res + base + c, r);
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[i] += r[i];
                }
                store8(dx + base + c, o);
            }
        }
    }
#pragma unroll
    for (int it = 0; it < ITERS; ++it) {
        const int c = (it * blockDim.x + threadIdx.x) * 8;
        if (c < C) {
            float* o = dw_partial + static_cast<size_t>(blockIdx.x) * C + c;
            *reinterpret_cast<float4*>(o) = make_float4(dw[it][0], dw[it][1], dw[it][2], dw[it][3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(dw[it][4], dw[it][5], dw[it][6], dw[it][7]);
        }
    }
}
// out[c] = sum of the partial rows.  One CTA per 16 columns: four lanes x 16 bytes span the columns, 256 rows are read side by side, so
// that a thread has its few loads in flight together, and the sums meet by shuffle and in shared memory (fixed order, no atomics, no
// cleared output).  Latency-bound: a few us, where 32 CTAs whose threads walked 148 rows each, with an
// atomic per slice and a memset before it, took 43 us for [1184, 1024].  RMSNorm backward on B200 in all, L2 flushed: 8192 x 4096 81 -> 65 us,
// 3000 x 1024 53 -> 17 us, 1024 x 512 42 -> 11 us.
constexpr int CS_COLS = 16, CS_THREADS = 1024;
__global__ void __launch_bounds__(CS_THREADS) column_sum_kernel(const float* __restrict__ partial, float* __restrict__ out, int nblocks, int C) {
    __shared__ float sh[CS_THREADS / 32][CS_COLS];
    const int c = blockIdx.x * CS_COLS + (threadIdx.x & 3) * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < C) {
#pragma unroll 4
        for (int b = threadIdx.x >> 2; b < nblocks; b += CS_THREADS / 4) {
            const float4 v = *reinterpret_cast<const float4*>(partial + static_cast<size_t>(b) * C + c);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o); s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        s.z += __shfl_xor_sync(0xffffffffu, s.z, o); s.w += __shfl_xor_sync(0xffffffffu, s.w, o);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane < 4) *reinterpret_cast<float4*>(&sh[warp][lane * 4]) = s;
    __syncthreads();
    if (threadIdx.x < CS_COLS && blockIdx.x * CS_COLS + threadIdx.x < C) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < CS_THREADS / 32; ++w) t += sh[w][threadIdx.x];
        out[blockIdx.x * CS_COLS + threadIdx.x] = t;
    }
}

// ------------------------------------------------------------------------------------------ SwiGLU
// x = [up | gate] per row (2M); y = silu(gate) * up.  Optional FP8 copy of y with scale + abs-max.
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, uint8_t* __restrict__ y_fp8,
                                                         const float* __restrict__ fp8_scale, float* __restrict__ amax_out, size_t rows, int M,
                                                         const int* __restrict__ rows_limit) {
    __shared__ float sh[32];
    // rows_limit (device): only the first *rows_limit rows are in use (expert buffers sized for the worst case); cost follows the use
    if (rows_limit) rows = min(rows, static_cast<size_t>(max(0, __ldg(rows_limit))));
    const float qs = fp8_scale ? __ldg(fp8_scale) : 1.f;
    float amax = 0.f;
    // grid.x x block covers the M / 8 column vectors, grid.y strides over the rows: no index division, and a thread's consecutive
    // trips touch consecutive rows of the same columns
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c < M) {
        for (size_t row = blockIdx.y; row < rows; row += gridDim.y) {
            float up[8], gate[8], o[8];
            load8(x + row * 2 * M + c, up);
            load8(x + row * 2 * M + M + c, gate);
#pragma unroll
            for (int i = 0; i < 8; ++i) { o[i] = gate[i] / (1.f + __expf(-gate[i])) * up[i]; amax = fmaxf(amax, fabsf(o[i])); }
            if (y) store8(y + row * M + c, o);
            if (y_fp8) *reinterpret_cast<uint2*>(y_fp8 + row * M + c) = to_fp8x8<false>(o, qs);
        }
    }
    if (amax_out) {
        amax = block_reduce<true>(amax, sh);
        if (threadIdx.x == 0) atomic_max_pos(amax_out, amax);
    }
}
// dx (bf16) and / or dx_fp8 (E5M2 with the given scale, recording the abs-max of the unscaled values): when the only reader of the
// gradient is an FP8 GEMM, the bf16 tensor is never written and no separate quantise pass reads it back.
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, bf16* __restrict__ dx, size_t rows, int M,
                                                         const int* __restrict__ rows_limit, uint8_t* __restrict__ dx_fp8, const float* __restrict__ fp8_scale,
                                                         float* __restrict__ amax_out) {
    __shared__ float sh[32];
    if (rows_limit) rows = min(rows, static_cast<size_t>(max(0, __ldg(rows_limit))));
    const float qs = fp8_scale ? __ldg(fp8_scale) : 1.f;
    float amax = 0.f;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    for (size_t row = blockIdx.y; c < M && row < rows; row += gridDim.y) {
        float up[8], gate[8], g[8], du[8], dg[8];
        load8(x + row * 2 * M + c, up);
        load8(x + row * 2 * M + M + c, gate);
        load8(dy + row * M + c, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float s = 1.f / (1.f + __expf(-gate[i]));
            du[i] = g[i] * gate[i] * s;
            dg[i] = g[i] * up[i] * s * (1.f + gate[i] * (1.f - s));
        }
        if (dx) {
            store8(dx + row * 2 * M + c, du);
            store8(dx + row * 2 * M + M + c, dg);
        }
        if (dx_fp8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fmaxf(fabsf(du[i]), fabsf(dg[i])));
            *reinterpret_cast<uint2*>(dx_fp8 + row * 2 * M + c) = to_fp8x8<true>(du, qs);
            *reinterpret_cast<uint2*>(dx_fp8 + row * 2 * M + M + c) = to_fp8x8<true>(dg, qs);
        }
    }
    if (amax_out) {
        amax = block_reduce<true>(amax, sh);
        if (threadIdx.x == 0) atomic_max_pos(amax_out, amax);
    }
}

// ------------------------------------------------------------------------------------------ QK-norm + RoPE
// Half a warp per (token, head); head_dim 128: lane s = lane & 15 of the half holds elements [8s, 8s+8) (one 16-byte access), the
// rotary partner (i +/- 64) lives in lane s ^ 8 of the same half.  A warp works on one token at a time and walks all of its heads,
// two at a time (one per half-warp).  A block takes TOK tokens at a time; its threads evaluate the sines and cosines of all of them
// together, each angle once, into shared memory (two tables in turn, so one barrier per group of tokens).  Evaluated in every lane that
// uses them they cost four times the work and the registers of a third resident block.  TOK is eight (a warp to a token), or four (two) in the
// forward from 17 heads on, where eight left a second wave of few blocks at 4096 tokens; up to 16 heads the second warp would have half a
// batch of loads or none (1 x 333 x 32 heads 8.6 -> 5.6 us with four, 2 x 1024 x 7 heads 4.9 -> 8.0).  On B200, in L2, with angles per lane -> eight tokens -> four,
// 2 x 2048 x 48 heads 31.3 -> 33.1 -> 30.3 us,
// 2 x 4096 x 48 61.8 -> 53.7 -> 54.2, 1 x 1000 x 32 8.5 -> 8.6 -> 7.0; backward (eight) 95.3 -> 93.0 us at 2 x 4096 x 48.
// Layout per token: [Hq heads | Hkv heads (K) | Hkv heads (V)] x D.  V heads are copied (forward) / passed through (backward).
constexpr int ROPE_PAIRS_IN_FLIGHT = 4;      // head pairs whose loads are issued before the first is used
constexpr int ROPE_SPLIT_HEADS = 2 * 2 * ROPE_PAIRS_IN_FLIGHT;      // more heads than two batches of loads: two warps to a token
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <bool BACKWARD, int TOK>
__global__ void __launch_bounds__(256, BACKWARD ? 2 : 3) qk_norm_rope_kernel(const bf16* __restrict__ in, const bf16* __restrict__ qkv_pre, const bf16* __restrict__ qw,
                                                           const bf16* __restrict__ kw, const int* __restrict__ pos, bf16* __restrict__ out,
                                                           float* __restrict__ q_rstd, float* __restrict__ k_rstd, float* __restrict__ dqw,
                                                           float* __restrict__ dkw, size_t tokens, int Hq, int Hkv, float eps, float log2_theta,
                                                           int lim_h, int lim_w) {
    // Multi-axis rotary positions (vision-language models): when lim_h or lim_w is non-zero, ``pos`` holds three rows of
    // ``tokens`` entries (temporal, height, width) and frequency j uses the height row if j % 3 == 1 and j < lim_h, the width
    // row if j % 3 == 2 and j < lim_w, else the temporal row.
    constexpr int D = 128;
    constexpr int U = ROPE_PAIRS_IN_FLIGHT;
    __shared__ float sdw[2][D];
    constexpr int WPT = 8 / TOK;     // warps per token
    __shared__ alignas(16) float trig[2][TOK][2][D / 2];   // [table][token][cos | sin][frequency]
    const bool multi_axis = (lim_h | lim_w) != 0;
    if (BACKWARD) {
        for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) (&sdw[0][0])[i] = 0.f;
    }
    const int H = Hq + 2 * Hkv;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane & 15, hsel = lane >> 4;
    const bool use_norm = qw != nullptr;
    float dw_acc[2][8];      // this lane's 8 elements: [q|k] norm-weight grads
    uint4 wq_raw = make_uint4(0, 0, 0, 0), wk_raw = wq_raw;
    if (use_norm) {
        alignas(16) bf16 q8[8], k8[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) { q8[i] = qw[sub * 8 + i]; k8[i] = kw[sub * 8 + i]; }
        wq_raw = *reinterpret_cast<const uint4*>(q8);
        wk_raw = *reinterpret_cast<const uint4*>(k8);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        dw_acc[0][i] = 0.f;
        dw_acc[1][i] = 0.f;
    }
    // the frequency whose angles this thread evaluates, for tokens threadIdx.x / 64 (and + 4) of the block's
    const int freq = threadIdx.x & 63, m3 = freq % 3;
    const float inv = exp2f(-log2_theta * (2.f * freq) / D);
    const size_t axis_row = (m3 == 1 && freq < lim_h) ? tokens : ((m3 == 2 && freq < lim_w) ? 2 * tokens : 0);
    const float sign = (sub < 8) ? -1.f : 1.f;  // first half of the head: x1*c - x2*s ; second half: x2*c + x1*s
    int table = 0;
    for (size_t tok0 = static_cast<size_t>(blockIdx.x) * TOK; tok0 < tokens; tok0 += static_cast<size_t>(gridDim.x) * TOK, table ^= 1) {
#pragma unroll
        for (int k = 0; k < TOK / 4; ++k) {
            const int w = (threadIdx.x >> 6) + 4 * k;
            if (tok0 + w < tokens) {
                float sn, cs;
                sincosf(static_cast<float>(pos[(multi_axis ? axis_row : 0) + tok0 + w]) * inv, &sn, &cs);
                trig[table][w][0][freq] = cs;
                trig[table][w][1][freq] = sn;
            }
        }
        __syncthreads();
        const int slot = warp / WPT;
        const size_t tok = tok0 + slot;
        if (tok >= tokens) continue;
        float cs[8], sn[8];
        *reinterpret_cast<float4*>(cs) = *reinterpret_cast<const float4*>(&trig[table][slot][0][(sub & 7) * 8]);
        *reinterpret_cast<float4*>(cs + 4) = *reinterpret_cast<const float4*>(&trig[table][slot][0][(sub & 7) * 8 + 4]);
        *reinterpret_cast<float4*>(sn) = *reinterpret_cast<const float4*>(&trig[table][slot][1][(sub & 7) * 8]);
        *reinterpret_cast<float4*>(sn + 4) = *reinterpret_cast<const float4*>(&trig[table][slot][1][(sub & 7) * 8 + 4]);
        const size_t tbase = tok * static_cast<size_t>(H) * D + sub * 8;
        for (int hb = (warp % WPT) * 2 * U; hb < H; hb += 2 * U * WPT) {
            // all loads of this batch of head pairs are issued before any of them is used
            uint4 raws[U], pres[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int h = hb + 2 * u + hsel;
                if (h < H) {
                    const size_t off = tbase + static_cast<size_t>(h) * D;
                    raws[u] = *reinterpret_cast<const uint4*>(in + off);
                    if (BACKWARD && use_norm && h < Hq + Hkv) pres[u] = *reinterpret_cast<const uint4*>(qkv_pre + off);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int h = hb + 2 * u + hsel;
                // a half-warp whose head index ran past H still takes part in the shuffles of the other half's head
                const bool live = h < H;
                const bool is_v = h >= Hq + Hkv;
                const bool is_q = h < Hq;
                const size_t off = tbase + static_cast<size_t>(h) * D;
                if (hb + 2 * u >= H) break;           // both halves past the end (uniform over the warp)
                float v[8];
                if (live) unpack8(raws[u], v);
                else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = 0.f;
                }
                if (!BACKWARD) {
                    float rstd = 1.f;
                    if (use_norm) {
                        float ss = 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
                        ss = half_warp_sum(ss);
                        rstd = rsqrtf(ss / D + eps);
                        if (live && !is_v) {
                            float w8[8];
                            unpack8(is_q ? wq_raw : wk_raw, w8);
#pragma unroll
                            for (int i = 0; i < 8; ++i) v[i] = v[i] * rstd * w8[i];
                            if (sub == 0) {
                                if (is_q) q_rstd[tok * Hq + h] = rstd;
                                else k_rstd[tok * Hkv + (h - Hq)] = rstd;
                            }
                        }
                    }
                    float o[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float partner = __shfl_xor_sync(0xffffffffu, v[i], 8);
                        o[i] = v[i] * cs[i] + sign * partner * sn[i];
                    }
                    if (live) {
                        if (is_v) *reinterpret_cast<uint4*>(out + off) = raws[u];
                        else store8(out + off, o);
                    }
                } else {
                    // v = d(out).  Inverse rotation: g1 = d1*c + d2*s ; g2 = d2*c - d1*s
                    float g[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float partner = __shfl_xor_sync(0xffffffffu, v[i], 8);
                        g[i] = v[i] * cs[i] - sign * partner * sn[i];
                    }
                    if (use_norm) {
                        float xin[8];
                        const bool normed = live && !is_v;
                        if (normed) unpack8(pres[u], xin);
                        else {
#pragma unroll
                            for (int i = 0; i < 8; ++i) xin[i] = 0.f;
                        }
                        const float rstd = normed ? (is_q ? q_rstd[tok * Hq + h] : k_rstd[tok * Hkv + (h - Hq)]) : 0.f;
                        float dot = 0.f, dn[8], xhat[8], w8[8];
                        unpack8(is_q ? wq_raw : wk_raw, w8);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            xhat[i] = xin[i] * rstd;
                            dn[i] = g[i] * w8[i];
                            dot += dn[i] * xhat[i];
                        }
                        if (normed) {
#pragma unroll
                            for (int i = 0; i < 8; ++i) dw_acc[is_q ? 0 : 1][i] += g[i] * xhat[i];
                        }
                        dot = half_warp_sum(dot) / D;
#pragma unroll
                        for (int i = 0; i < 8; ++i) g[i] = rstd * (dn[i] - xhat[i] * dot);
                    }
                    if (live) {
                        if (is_v) *reinterpret_cast<uint4*>(out + off) = raws[u];
                        else store8(out + off, g);
                    }
                }
            }
        }
    }
    if (BACKWARD && use_norm) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            atomicAdd(&sdw[0][sub * 8 + i], dw_acc[0][i]);
            atomicAdd(&sdw[1][sub * 8 + i], dw_acc[1][i]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < D; i += blockDim.x) {
            atomicAdd(dqw + i, sdw[0][i]);
            atomicAdd(dkw + i, sdw[1][i]);
        }
    }
}

// ------------------------------------------------------------------------------------------ embedding
// A token id outside [0, V) writes zeros for that row and raises the error flag instead of reading outside the table.
__global__ void embedding_fwd_kernel(const int* __restrict__ tokens, const bf16* __restrict__ table, bf16* __restrict__ out, size_t n, int C, int V,
                                     int* __restrict__ error_flag) {
    const size_t nvec = n * (C / 8);
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < nvec; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t t = v / (C / 8);
        const int c = static_cast<int>(v % (C / 8)) * 8;
        const int tok = tokens[t];
        if (tok < 0 || tok >= V) {
            *reinterpret_cast<uint4*>(out + t * C + c) = make_uint4(0, 0, 0, 0);
            if (c == 0 && error_flag) atomicExch(error_flag, 2);
            continue;
        }
        *reinterpret_cast<uint4*>(out + t * C + c) = *reinterpret_cast<const uint4*>(table + static_cast<size_t>(tok) * C + c);
    }
}
template <typename G> __global__ void embedding_bwd_kernel(const int* __restrict__ tokens, const bf16* __restrict__ d_out, G* __restrict__ d_table, size_t n, int C) {
    const size_t npair = n * (C / 2);
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < npair; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t t = v / (C / 2);
        const int c = static_cast<int>(v % (C / 2)) * 2;
        const bf162 g = *reinterpret_cast<const bf162*>(d_out + t * C + c);
        G* dst = d_table + static_cast<size_t>(tokens[t]) * C + c;
        if constexpr (sizeof(G) == 2) {
            atomicAdd(reinterpret_cast<bf162*>(dst), g);
        } else {
            const float2 f = __bfloat1622float2(g);
            atomicAdd(dst, f.x);
            atomicAdd(dst + 1, f.y);
        }
    }
}

// Deterministic variant: positions are sorted by token id first; CTA (i, y) owns the run of equal ids that STARTS at sorted position i
// (other CTAs leave at once) and EMB_COLS columns, sums the run's rows in fp32 in sorted order and adds the sum to the table row once.  No
// atomics, so the result does not depend on scheduling.  Ids outside [0, V) are skipped.
// The longest run is the critical path (text repeats its frequent tokens hundreds of times per batch): EMB_AHEAD rows are requested before
// the first is added, and the columns are spread over CTAs.  8192 rows of 4096, longest run 160, on B200: 577 -> 166 us with the sort
// (about 100 us of it).
// VEC elements per thread and access: 8 where rows are whole 16-byte vectors, else 2, or 1 for bases off a 4-byte boundary.  On B200, 4096 x
// 1022 in vectors of 2 147 us (297 us in a kernel with one row in flight, 330 us through copies padded to 8).
constexpr int EMB_COLS = 512, EMB_AHEAD = 8;
template <int VEC> struct EmbWord { using T = uint4; };
template <> struct EmbWord<2> { using T = uint32_t; };
template <> struct EmbWord<1> { using T = unsigned short; };
__device__ __forceinline__ void emb_unpack(const uint4& w, float (&f)[8]) { unpack8(w, f); }
__device__ __forceinline__ void emb_unpack(const uint32_t& w, float (&f)[2]) { f[0] = __uint_as_float(w << 16); f[1] = __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ void emb_unpack(const unsigned short& w, float (&f)[1]) { f[0] = __uint_as_float(static_cast<uint32_t>(w) << 16); }
template <typename G, int VEC>
__global__ void __launch_bounds__(EMB_COLS / VEC) embedding_bwd_sorted_kernel(const int* __restrict__ sorted_ids, const long long* __restrict__ order,
                                                                              const bf16* __restrict__ d_out, G* __restrict__ d_table, int n, int C, int V) {
    const int i = blockIdx.x;
    const int id = sorted_ids[i];
    if (id < 0 || id >= V || (i > 0 && sorted_ids[i - 1] == id)) return;
    using Word = typename EmbWord<VEC>::T;
    for (int c = blockIdx.y * EMB_COLS + threadIdx.x * VEC; c < C; c += gridDim.y * EMB_COLS) {
        float acc[VEC];
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] = 0.f;
        if (i + 1 == n || sorted_ids[i + 1] != id) {      // most ids of a batch without frequent ones
            emb_unpack(*reinterpret_cast<const Word*>(d_out + static_cast<size_t>(order[i]) * C + c), acc);
        } else for (int j = i;; j += EMB_AHEAD) {
            bool mine[EMB_AHEAD];
            long long src[EMB_AHEAD];
#pragma unroll
            for (int u = 0; u < EMB_AHEAD; ++u) {
                mine[u] = j + u < n && sorted_ids[j + u] == id;       // sorted: once false, false from there on
                src[u] = mine[u] ? order[j + u] : 0;
            }
            Word raw[EMB_AHEAD];
#pragma unroll
            for (int u = 0; u < EMB_AHEAD; ++u)
                if (mine[u]) raw[u] = *reinterpret_cast<const Word*>(d_out + static_cast<size_t>(src[u]) * C + c);
#pragma unroll
            for (int u = 0; u < EMB_AHEAD; ++u)
                if (mine[u]) {
                    float f[VEC];
                    emb_unpack(raw[u], f);
#pragma unroll
                    for (int k = 0; k < VEC; ++k) acc[k] += f[k];
                }
            if (!mine[EMB_AHEAD - 1]) break;
        }
        G* dst = d_table + static_cast<size_t>(id) * C + c;
        if constexpr (sizeof(G) == 2) {
            float o[VEC];
            emb_unpack(*reinterpret_cast<const Word*>(dst), o);
            alignas(16) bf16 r[VEC];
#pragma unroll
            for (int k = 0; k < VEC; ++k) r[k] = __float2bfloat16_rn(o[k] + acc[k]);
            *reinterpret_cast<Word*>(dst) = *reinterpret_cast<const Word*>(r);
        } else if constexpr (VEC == 8) {
#pragma unroll
            for (int k = 0; k < VEC; k += 4) {
                float4 o = *reinterpret_cast<const float4*>(dst + k);
                o.x += acc[k]; o.y += acc[k + 1]; o.z += acc[k + 2]; o.w += acc[k + 3];
                *reinterpret_cast<float4*>(dst + k) = o;
            }
        } else {
#pragma unroll
            for (int k = 0; k < VEC; ++k) dst[k] += acc[k];
        }
    }
}

// whole 16-byte vectors of zeros, stored past the caches' working set: gradient tables are far larger than L2 (1.2 GB on B200: 320 -> 214 us)
__global__ void __launch_bounds__(256) zero_fill_kernel(uint4* __restrict__ p, size_t nvec) {
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < nvec; v += static_cast<size_t>(gridDim.x) * blockDim.x)
        __stcs(p + v, make_uint4(0, 0, 0, 0));
}

// ------------------------------------------------------------------------------------------ cross-entropy (fwd + bwd in place)
// One CTA per row of bf16 logits [rows, V].  loss[row] = lse - logit[target]; logits are overwritten with
// d_logits = (softmax - onehot) * scale * row_weight[row] (scale read from device memory), zero for ignored rows.
// row_weight is the hook for sequence-level objectives whose gradient is a per-token multiple of the log-likelihood gradient
// (DPO: +-beta*sigmoid(-margin) per sequence; GRPO: clipped ratio x advantage per token).
// Optional knowledge distillation on a teacher's top-K log-probabilities: kd_loss[row] = sum_k p_k (log p_k - log q_k) with
// q the student softmax, and d_logits += kd_weight * (S * q - scatter(p)), S = sum_k p_k.  A row with an ignored target
// contributes neither term.
// FP8 (without distillation): the gradient leaves as E5M2 of gradient * *q_scale in `d8` [rows, V] (rounded to bf16 first, as a separate
// quantise pass would have it) and the logits stay as they are: no bf16 gradient is written and read back.  Memory-bound: the logits are
// read twice; 4096 x 151936 on B200: 890 us with the quantise pass, 596 us without it.  Holding the row in registers across a cluster of
// eight CTAs reads it once but was slower (778 us against 590 in bf16): the exchange costs more than the second read.
template <bool FP8>
__global__ void __launch_bounds__(1024) cross_entropy_fwd_bwd_kernel(bf16* __restrict__ logits, uint8_t* __restrict__ d8, const float* __restrict__ q_scale,
                                                                     const int* __restrict__ targets, float* __restrict__ loss,
                                                                     const float* __restrict__ scale_ptr, float scale_host, int V, int ld,
                                                                     int write_grad, const float* __restrict__ row_weight,
                                                                     const int* __restrict__ kd_idx, const float* __restrict__ kd_logp, int kd_k,
                                                                     float kd_weight, float* __restrict__ kd_loss) {
    __shared__ float sh[32];
    __shared__ float kd_sum_p;
    const size_t row = blockIdx.x;
    bf16* lr = logits + row * ld;
    const int tgt = targets[row];
    if (tgt < 0) {
        if (threadIdx.x == 0) {
            loss[row] = 0.f;
            if (kd_loss) kd_loss[row] = 0.f;
        }
        if (write_grad) {
            for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
                if (FP8) *reinterpret_cast<uint2*>(d8 + row * V + c) = make_uint2(0, 0);
                else *reinterpret_cast<uint4*>(lr + c) = make_uint4(0, 0, 0, 0);
            }
        }
        return;
    }
    float mx = -INFINITY, sum = 0.f;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
        float a[8];
        load8(lr + c, a);
        float m = a[0];
#pragma unroll
        for (int i = 1; i < 8; ++i) m = fmaxf(m, a[i]);
        if (m > mx) { sum *= __expf(mx - m); mx = m; }
        const float base = mx == -INFINITY ? 0.f : mx;      // nothing but masked logits so far
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += __expf(a[i] - base);
    }
    const float gmax = block_reduce<true>(mx, sh);
    sum *= __expf(mx - gmax);
    const float gsum = block_reduce<false>(sum, sh);
    const float lse = gmax + __logf(gsum);
    if (threadIdx.x == 0) loss[row] = lse - __bfloat162float(lr[tgt]);
    float S = 0.f;
    if (kd_k > 0) {  // the first warp walks the teacher's top-K entries of this row
        if (threadIdx.x < 32) {
            float kl = 0.f, sp = 0.f;
            for (int k = threadIdx.x; k < kd_k; k += 32) {
                const int j = kd_idx[row * kd_k + k];
                if (j < 0 || j >= V) continue;
                const float lp = kd_logp[row * kd_k + k];
                const float pk = __expf(lp);
                kl += pk * (lp - (__bfloat162float(lr[j]) - lse));
                sp += pk;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) { kl += __shfl_xor_sync(0xffffffffu, kl, o); sp += __shfl_xor_sync(0xffffffffu, sp, o); }
            if (threadIdx.x == 0) { kd_sum_p = sp; if (kd_loss) kd_loss[row] = kl; }
        }
        __syncthreads();
        S = kd_sum_p;
    }
    if (!write_grad) return;
    __syncthreads();
    const float scale = scale_host * (scale_ptr ? __ldg(scale_ptr) : 1.f);
    const float w_ce = scale * (row_weight ? row_weight[row] : 1.f);
    const float w_kd = kd_k > 0 ? scale * kd_weight : 0.f;
    const float w_soft = w_ce + w_kd * S;
    const float qs = FP8 ? __ldg(q_scale) : 1.f;
    for (int c = threadIdx.x * 8; c < V; c += blockDim.x * 8) {
        float a[8];
        load8(lr + c, a);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float g = __expf(a[i] - lse) * w_soft;
            if (c + i == tgt) g -= w_ce;
            a[i] = g;
        }
        if (FP8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = __bfloat162float(__float2bfloat16_rn(a[i]));
            *reinterpret_cast<uint2*>(d8 + row * V + c) = to_fp8x8<true>(a, qs);
        } else {
            store8(lr + c, a);
        }
    }
    if (!FP8 && kd_k > 0) {
        __syncthreads();  // every gradient of the row is written; now subtract the teacher mass at its K positions
        for (int k = threadIdx.x; k < kd_k; k += blockDim.x) {
            const int j = kd_idx[row * kd_k + k];
            if (j < 0 || j >= V) continue;
            bool first = true;  // a repeated index is applied once per occurrence by the lowest k only (sequentially below)
            for (int q = 0; q < k; ++q) first = first && kd_idx[row * kd_k + q] != j;
            if (!first) continue;
            float pm = 0.f;
            for (int q = k; q < kd_k; ++q)
                if (kd_idx[row * kd_k + q] == j) pm += __expf(kd_logp[row * kd_k + q]);
            lr[j] = __float2bfloat16(__bfloat162float(lr[j]) - w_kd * pm);
        }
    }
}

// ------------------------------------------------------------------------------------------ FP8 quantise / abs-max / sum of squares
template <bool E5M2>
__global__ void __launch_bounds__(256) quantize_fp8_kernel(const bf16* __restrict__ x, uint8_t* __restrict__ q, const float* __restrict__ scale,
                                                           float* __restrict__ amax_out, size_t n, const int* __restrict__ rows_limit, int row_len) {
    __shared__ float sh[32];
    const float s = scale ? __ldg(scale) : 1.f;
    float amax = 0.f;
    if (rows_limit) n = min(n, static_cast<size_t>(max(0, __ldg(rows_limit))) * row_len);   // only the leading rows are in use
    const size_t nvec = n / 8;
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < nvec; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float a[8];
        load8(x + v * 8, a);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(a[i]));
        *reinterpret_cast<uint2*>(q + v * 8) = to_fp8x8<E5M2>(a, s);
    }
    if (amax_out) {
        amax = block_reduce<true>(amax, sh);
        if (threadIdx.x == 0) atomic_max_pos(amax_out, amax);
    }
}
// FP8 -> bf16 with the per-tensor de-scale: q * *scale in fp32, rounded once.  16 values per thread and trip; bound by the 3 bytes per value
// that it moves.  4096 x 12288: three ATen passes through fp32 took 160 us on B200; the packed-documents LoRA step 32.3 -> 26.8 ms.
template <bool E5M2>
__global__ void __launch_bounds__(256) dequantize_fp8_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scale, bf16* __restrict__ out, size_t n) {
    const float s = __ldg(scale);
    const size_t nvec = n / 16, tid = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x, stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    auto value = [](uint8_t b) { return __half2float(__half(__nv_cvt_fp8_to_halfraw(b, E5M2 ? __NV_E5M2 : __NV_E4M3))); };
    for (size_t v = tid; v < nvec; v += stride) {
        const uint4 raw = *reinterpret_cast<const uint4*>(q + v * 16);
        const __nv_fp8x2_storage_t* b = reinterpret_cast<const __nv_fp8x2_storage_t*>(&raw);
        uint4 o[2];
        bf162* ob = reinterpret_cast<bf162*>(o);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 f = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(b[i], E5M2 ? __NV_E5M2 : __NV_E4M3)));
            ob[i] = __floats2bfloat162_rn(f.x * s, f.y * s);
        }
        *reinterpret_cast<uint4*>(out + v * 16) = o[0];
        *reinterpret_cast<uint4*>(out + v * 16 + 8) = o[1];
    }
    for (size_t i = nvec * 16 + tid; i < n; i += stride) out[i] = __float2bfloat16_rn(value(q[i]) * s);
}

__global__ void __launch_bounds__(256) amax_kernel(const bf16* __restrict__ x, float* __restrict__ amax_out, size_t n, const int* __restrict__ rows_limit,
                                                   int row_len) {
    __shared__ float sh[32];
    float amax = 0.f;
    if (rows_limit) n = min(n, static_cast<size_t>(max(0, __ldg(rows_limit))) * row_len);
    const size_t nvec = n / 8;
    for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < nvec; v += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float a[8];
        load8(x + v * 8, a);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(a[i]));
    }
    amax = block_reduce<true>(amax, sh);
    if (threadIdx.x == 0) atomic_max_pos(amax_out, amax);
}
// vectorised sum of squares: 16-byte loads, tail handled by the first threads
template <typename T> __global__ void __launch_bounds__(512) sumsq_kernel(const T* __restrict__ x, float* __restrict__ partial, size_t n) {
    __shared__ float sh[32];
    constexpr int VEC = 16 / sizeof(T);
    float s = 0.f;
    const size_t nvec = n / VEC;
    const size_t tid = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x, stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t v = tid; v < nvec; v += stride) {
        if constexpr (sizeof(T) == 2) {
            float a[8];
            load8(reinterpret_cast<const bf16*>(x) + v * 8, a);
#pragma unroll
            for (int i = 0; i < 8; ++i) s += a[i] * a[i];
        } else {
            const float4 a = *reinterpret_cast<const float4*>(x + v * 4);
            s += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
        }
    }
    for (size_t i = nvec * VEC + tid; i < n; i += stride) {
        float v;
        if constexpr (sizeof(T) == 2) v = __bfloat162float(x[i]); else v = x[i];
        s += v * v;
    }
    s = block_reduce<false>(s, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;   // fixed grid -> deterministic second stage on the host side tensor
}

// ------------------------------------------------------------------------------------------ AdamW
// hp (device): [lr, beta1, beta2, eps, weight_decay, bias_corr1, bias_corr2, grad_scale] so a captured graph can be replayed.
// Every thread owns 8 consecutive elements (n must be a multiple of 8; shards are multiples of 128).
template <typename T> __device__ __forceinline__ void load8_any(const T* p, float (&f)[8]) {
    if constexpr (sizeof(T) == 2) {
        load8(reinterpret_cast<const bf16*>(p), f);
    } else {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
}
template <typename T> __device__ __forceinline__ void store8_any(T* p, const float (&f)[8]) {
    if constexpr (sizeof(T) == 2) {
        store8(reinterpret_cast<bf16*>(p), f);
    } else {
        *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
}

template <typename P, typename G>
__global__ void __launch_bounds__(256) adamw_fp32_kernel(P* __restrict__ p, const G* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                                                         const uint8_t* __restrict__ decay_mask, const float* __restrict__ hp, size_t n) {
    const float lr = hp[0], b1 = hp[1], b2 = hp[2], eps = hp[3], wd = hp[4], bc1 = hp[5], bc2 = hp[6], gs = hp[7];
    if (gs == 0.f) return;   // clip scale 0 = the step's gradient was not finite: weights and moments stay as they are
    const float ibc1 = 1.f / bc1, ibc2 = 1.f / bc2;
    const size_t nvec = n / 8;
    for (size_t vi = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; vi < nvec; vi += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t i = vi * 8;
        float pv[8], gv[8], mv[8], vv[8];
        load8_any(p + i, pv);
        load8_any(g + i, gv);
        load8_any(m + i, mv);
        load8_any(v + i, vv);
        uint2 mk = make_uint2(0, 0);
        if (decay_mask) mk = *reinterpret_cast<const uint2*>(decay_mask + i);
        const uint8_t* mb = reinterpret_cast<const uint8_t*>(&mk);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float gk = gv[k] * gs;
            mv[k] = b1 * mv[k] + (1.f - b1) * gk;
            vv[k] = b2 * vv[k] + (1.f - b2) * gk * gk;
            const float dec = mb[k] ? wd : 0.f;
            pv[k] = pv[k] * (1.f - lr * dec) - lr * (mv[k] * ibc1) / (sqrtf(vv[k] * ibc2) + eps);
        }
        store8_any(m + i, mv);
        store8_any(v + i, vv);
        store8_any(p + i, pv);
    }
}

// 8-bit state: momentum int8 through softsign (2x/(1+|x|) of the group-normalised value), variance uint8 of sqrt(v),
// groups of 32 with fp16 scales.  Four adjacent lanes (8 elements each) form one group; the group abs-max is two shuffles.
// n must be a multiple of 32.  The kernel moves 10.25 bytes per parameter, so the work per element has to stay below about
// 40 issued instructions to be bound by memory and not by instruction issue.  Hence:
//  * element pairs go through the packed fp32 instructions of sm_100 (fma / mul / add .f32x2: two results per issue slot);
//  * momentum codes are decoded through a 256-entry shared-memory table, variance codes by splicing the byte into the
//    mantissa of 2^23 (one byte-permute), and both are re-encoded by adding 1.5 * 2^23, whose low mantissa byte then IS the
//    rounded two's-complement code (no float<->int conversions, which share an issue port with the special-function unit);
//  * square root and the two reciprocals per element use the hardware approximations;
//  * the weight-decay mask is one byte per 128 parameters (BLOCK_MASK) instead of one per parameter.
__device__ __forceinline__ float sqrt_fast(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_fast(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 splat2(float x) { return make_float2(x, x); }
constexpr float kRoundMagic = 12582912.f;   // 1.5 * 2^23: adding it rounds to the nearest integer and leaves it in the low mantissa bits

// Weights, gradients and codes reach the registers through a ring of shared-memory slots (cp.async; every thread copies and
// reads only its own 8 elements, so the ring needs no barrier): three trips' worth of loads are outstanding while one is computed, 110 KB
// per SM.  The group scales are two bytes each, below what cp.async moves, and are fetched one trip ahead into registers.  With loads and
// arithmetic of a trip one after the other, DRAM idled during the arithmetic of all three CTAs: 64 M parameters in bf16
// on B200 170 -> 146 us (4.7 TB/s).
// Four slots, or three where weights and gradients are both fp32: four of those leave room for two CTAs per SM only, and then the arithmetic
// is short of warps (64 M parameters 183 us with loads and arithmetic in turn, 195 with four slots, 169 with three).
constexpr int ADAM8_THREADS = 256;
template <typename P, typename G> constexpr int adam8_stages() { return sizeof(P) + sizeof(G) >= 8 ? 3 : 4; }
template <typename P, typename G> constexpr int adam8_slot_bytes() { return ADAM8_THREADS * (8 * static_cast<int>(sizeof(P) + sizeof(G)) + 16); }
template <int BYTES> __device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
    if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
template <typename P, typename G, bool BLOCK_MASK>
__global__ void __launch_bounds__(ADAM8_THREADS, 3) adamw_8bit_kernel(P* __restrict__ p, const G* __restrict__ g, int8_t* __restrict__ m8, uint8_t* __restrict__ v8,
                                                            __half* __restrict__ ms, __half* __restrict__ vs, const uint8_t* __restrict__ decay_mask,
                                                            const float* __restrict__ hp, size_t n) {
    extern __shared__ __align__(16) uint8_t ring[];
    // softsign decode table of the momentum code, indexed by code + 128: y = c/127, m = y / (2 - |y|) (times the group scale)
    __shared__ float m_lut[256];
    {
        const float y = static_cast<float>(static_cast<int>(threadIdx.x) - 128) * (1.f / 127.f);
        m_lut[threadIdx.x] = y / (2.f - fabsf(y));
    }
    __syncthreads();
    const float lr = hp[0], b1 = hp[1], b2 = hp[2], eps = hp[3], wd = hp[4], bc1 = hp[5], bc2 = hp[6], gs = hp[7];
    if (gs == 0.f) return;   // skipped update (non-finite gradient norm): nothing is read or written
    const float2 gs2 = splat2(gs), b1_2 = splat2(b1), omb1_2 = splat2(1.f - b1), b2_2 = splat2(b2), rt_omb2 = splat2(sqrtf(1.f - b2)),
                 sib2_2 = splat2(rsqrtf(bc2)), eps_2 = splat2(eps), nstep_2 = splat2(-lr / bc1), one_2 = splat2(1.f), magic_2 = splat2(kRoundMagic),
                 c254_2 = splat2(254.f), nbias_2 = splat2(-8388608.f);
    const float decay_on = 1.f - lr * wd;
    const char* lut_bytes = reinterpret_cast<const char*>(m_lut);
    const size_t nvec = n / 8;
    constexpr int PB = 8 * sizeof(P), GB = 8 * sizeof(G), SLOT = adam8_slot_bytes<P, G>(), STAGES = adam8_stages<P, G>();
    constexpr int OFF_G = ADAM8_THREADS * PB, OFF_M = OFF_G + ADAM8_THREADS * GB, OFF_V = OFF_M + ADAM8_THREADS * 8;
    const uint32_t ring0 = smem_u32(ring);
    const size_t stride = static_cast<size_t>(gridDim.x) * ADAM8_THREADS;
    auto request = [&](size_t vi, int slot) {      // one commit group per trip, empty behind the end
        if (vi < nvec) {
            const uint32_t d = ring0 + slot * SLOT;
#pragma unroll
            for (int k = 0; k < PB; k += 16) cp_async<16>(d + threadIdx.x * PB + k, reinterpret_cast<const uint8_t*>(p + vi * 8) + k);
#pragma unroll
            for (int k = 0; k < GB; k += 16) cp_async<16>(d + OFF_G + threadIdx.x * GB + k, reinterpret_cast<const uint8_t*>(g + vi * 8) + k);
            cp_async<8>(d + OFF_M + threadIdx.x * 8, m8 + vi * 8);
            cp_async<8>(d + OFF_V + threadIdx.x * 8, v8 + vi * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const size_t first = blockIdx.x * static_cast<size_t>(ADAM8_THREADS) + threadIdx.x;
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) request(first + k * stride, k);
    uint2 next_mk = make_uint2(0x01010101u, 0x01010101u);
    float next_sm = 0.f, next_sq = 0.f;
    auto fetch_scales = [&](size_t vi) {
        if (vi < nvec) {
            next_sm = __half2float(ms[vi >> 2]);
            next_sq = __half2float(vs[vi >> 2]);
            if (decay_mask) {
                if (BLOCK_MASK) next_mk.x = decay_mask[vi >> 4] ? 0x01010101u : 0u;
                else next_mk = *reinterpret_cast<const uint2*>(decay_mask + vi * 8);
            }
        }
    };
    fetch_scales(first);
    int slot = 0;
    // warp-uniform trip count so the shuffles always see all 32 lanes
    for (size_t base = blockIdx.x * static_cast<size_t>(ADAM8_THREADS) + (threadIdx.x & ~31); base < nvec; base += stride) {
        const size_t vi = base + (threadIdx.x & 31), idx = vi * 8;
        const bool live = vi < nvec;
        request(vi + (STAGES - 1) * stride, (slot + STAGES - 1) % STAGES);   // the slot that the previous trip emptied
        const uint2 mk = next_mk;
        const float sm = next_sm, sq = next_sq;
        fetch_scales(vi + stride);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        const uint8_t* cell = ring + slot * SLOT;
        slot = slot + 1 == STAGES ? 0 : slot + 1;
        {
            float pv[8], gv[8];
            load8_any(reinterpret_cast<const P*>(cell + threadIdx.x * PB), pv);
            load8_any(reinterpret_cast<const G*>(cell + OFF_G + threadIdx.x * GB), gv);
            const uint2 mraw = *reinterpret_cast<const uint2*>(cell + OFF_M + threadIdx.x * 8), vraw = *reinterpret_cast<const uint2*>(cell + OFF_V + threadIdx.x * 8);
            float2 mv[4], sv[4];
            float am = 0.f, av = 0.f;
            if (live) {
                const uint32_t mw[2] = {mraw.x ^ 0x80808080u, mraw.y ^ 0x80808080u};   // two's-complement codes -> table indices
                const uint32_t vw[2] = {vraw.x, vraw.y};
                const uint8_t* mb = reinterpret_cast<const uint8_t*>(&mk);
                const float2 smu2 = splat2(sm), squ2 = splat2(sq * (1.f / 255.f));
                const float2 dec_vec = splat2(mk.x ? decay_on : 1.f);
#pragma unroll
                for (int j = 0; j < 4; ++j) {       // elements 2j and 2j + 1
                    const uint32_t mword = mw[j >> 1], vword = vw[j >> 1];
                    const int b0 = (2 * j) & 3, b1i = b0 + 1;
                    // table lookups: byte b of the word, times 4, as a byte offset into the table
                    const uint32_t o0 = b0 == 0 ? (mword << 2) & 0x3FCu : (mword >> (8 * b0 - 2)) & 0x3FCu;
                    const uint32_t o1 = (mword >> (8 * b1i - 2)) & 0x3FCu;
                    float2 mi = mul2(make_float2(*reinterpret_cast<const float*>(lut_bytes + o0), *reinterpret_cast<const float*>(lut_bytes + o1)), smu2);
                    // variance codes: 0x4B0000cc is the float 2^23 + cc
                    const float2 vcode = make_float2(__uint_as_float(__byte_perm(vword, 0x4B000000u, 0x7440u | b0)),
                                                     __uint_as_float(__byte_perm(vword, 0x4B000000u, 0x7440u | b1i)));
                    const float2 r = mul2(add2(vcode, nbias_2), squ2);
                    float2 vi2 = mul2(r, r);
                    const float2 gk = mul2(make_float2(gv[2 * j], gv[2 * j + 1]), gs2);
                    mi = fma2(b1_2, mi, mul2(omb1_2, gk));
                    const float2 gc = mul2(gk, rt_omb2);
                    vi2 = fma2(gc, gc, mul2(b2_2, vi2));
                    const float2 sd = make_float2(sqrt_fast(vi2.x), sqrt_fast(vi2.y));     // sqrt(v)
                    const float2 den = fma2(sd, sib2_2, eps_2);
                    const float2 q = mul2(mi, make_float2(rcp_fast(den.x), rcp_fast(den.y)));
                    const float2 dec = BLOCK_MASK ? dec_vec : make_float2(mb[2 * j] ? decay_on : 1.f, mb[2 * j + 1] ? decay_on : 1.f);
                    const float2 pn = fma2(q, nstep_2, mul2(make_float2(pv[2 * j], pv[2 * j + 1]), dec));
                    pv[2 * j] = pn.x;
                    pv[2 * j + 1] = pn.y;
                    mv[j] = mi;
                    sv[j] = sd;
                    am = fmaxf(am, fmaxf(fabsf(mi.x), fabsf(mi.y)));
                    av = fmaxf(av, fmaxf(sd.x, sd.y));
                }
                store8_any(p + idx, pv);
            }
            am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
            am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
            av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 1));
            av = fmaxf(av, __shfl_xor_sync(0xffffffffu, av, 2));
            if (live) {
                // fp16 scales rounded up, so normalised values stay within [-1, 1] (up to one rounding of the product, which cannot
                // move a code past +-127 / 255)
                const __half hm = __float2half_ru(fmaxf(am, 1e-30f)), hv = __float2half_ru(fmaxf(av, 1e-30f));
                const float fm = fmaxf(__half2float(hm), 6e-8f), fv = fmaxf(__half2float(hv), 6e-8f);
                const float2 im2 = splat2(rcp_fast(fm)), iv2 = splat2(255.f * rcp_fast(fv));
                uint32_t mcode[4], vcode[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 xn = mul2(mv[j], im2);
                    const float2 ax = make_float2(fabsf(xn.x), fabsf(xn.y));
                    const float2 den = add2(ax, one_2);
                    const float2 y = mul2(xn, make_float2(rcp_fast(den.x), rcp_fast(den.y)));
                    const float2 mc = fma2(y, c254_2, magic_2);          // low mantissa byte = round(254 x / (1 + |x|)) in two's complement
                    const float2 vc = fma2(sv[j], iv2, magic_2);         // low mantissa byte = round(255 s / scale)
                    mcode[j] = __byte_perm(__float_as_uint(mc.x), __float_as_uint(mc.y), 0x0040u);
                    vcode[j] = __byte_perm(__float_as_uint(vc.x), __float_as_uint(vc.y), 0x0040u);
                }
                uint2 mo, vo;
                mo.x = __byte_perm(mcode[0], mcode[1], 0x5410u);
                mo.y = __byte_perm(mcode[2], mcode[3], 0x5410u);
                vo.x = __byte_perm(vcode[0], vcode[1], 0x5410u);
                vo.y = __byte_perm(vcode[2], vcode[3], 0x5410u);
                *reinterpret_cast<uint2*>(m8 + idx) = mo;
                *reinterpret_cast<uint2*>(v8 + idx) = vo;
                if ((threadIdx.x & 3) == 0) { ms[idx >> 5] = __float2half(fm); vs[idx >> 5] = __float2half(fv); }
            }
        }
    }
}

// ============================================================================================ launchers
static inline int grid_for(size_t work_items, int threads, int num_sms, int per_sm = 8) {
    size_t g = (work_items + threads - 1) / threads;
    const size_t cap = static_cast<size_t>(num_sms) * per_sm;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

void rmsnorm_fwd(const void* x, const void* residual, const void* w, void* res_out, void* y, float* rstd, void* y_fp8, const float* fp8_scale,
                 float* amax, int rows, int C, float eps, cudaStream_t s) {
    int threads = C / 8;
    threads = threads > 256 ? 256 : (threads < 32 ? 32 : (threads + 31) / 32 * 32);
    const int iters = (C + threads * 8 - 1) / (threads * 8);
#define SG_RF(IT)                                                                                                                              \
    rmsnorm_fwd_kernel<IT><<<rows, threads, 0, s>>>((const bf16*)x, (const bf16*)residual, (const bf16*)w, (bf16*)res_out, (bf16*)y, rstd,     \
                                                    (uint8_t*)y_fp8, fp8_scale, amax, C, eps)
    if (iters <= 1) SG_RF(1);
    else if (iters <= 2) SG_RF(2);
    else if (iters <= 4) SG_RF(4);
    else SG_RF(0);
#undef SG_RF
}
int rmsnorm_bwd_blocks(int rows, int num_sms) { return rows < num_sms * 2 ? rows : num_sms * 2; }
static int rmsnorm_bwd_threads(int C) { return C <= 1024 ? 128 : RB_THREADS; }
static int rmsnorm_bwd_iters(int C) {
    const int per = rmsnorm_bwd_threads(C) * 8;
    const int n = (C + per - 1) / per;
    return n <= 1 ? 1 : (n <= 2 ? 2 : (n <= 4 ? 4 : 8));
}
// CTAs for a [rows, C] problem: as many per SM as the register budget of the variant allows (see the kernel comment)
int rmsnorm_bwd_blocks_wide(int rows, int C, int num_sms) {
    const int per_sm = C <= 1024 ? 8 : (C <= 4096 ? 3 : 2);
    return rows < num_sms * per_sm ? rows : num_sms * per_sm;
}
void rmsnorm_bwd_n(const void* dy, const void* x, const void* w, const float* rstd, const void* d_res, void* dx, float* dw_partial, float* dw, int rows,
                   int C, int blocks, cudaStream_t s) {
    const int threads = rmsnorm_bwd_threads(C);
#define SG_RB(IT) rmsnorm_bwd_kernel<IT><<<blocks, threads, 0, s>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, rstd, (const bf16*)d_res, (bf16*)dx, dw_partial, rows, C)
    switch (rmsnorm_bwd_iters(C)) {
        case 1: SG_RB(1); break;
        case 2: SG_RB(2); break;
        case 4: SG_RB(4); break;
        default: SG_RB(8); break;
    }
#undef SG_RB
    column_sum_kernel<<<(C + CS_COLS - 1) / CS_COLS, CS_THREADS, 0, s>>>(dw_partial, dw, blocks, C);
}
void rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* d_res, void* dx, float* dw_partial, float* dw, int rows,
                 int C, int num_sms, cudaStream_t s) {
    rmsnorm_bwd_n(dy, x, w, rstd, d_res, dx, dw_partial, dw, rows, C, rmsnorm_bwd_blocks(rows, num_sms), s);
}
// blocks of 256 threads over the M / 8 column vectors; enough row-blocks to give every SM eight resident blocks
static int swiglu_threads(int M) {
    const int t = (M / 8 + 31) / 32 * 32;
    return t < 256 ? t : 256;       // narrow expert projections: no idle warps in the block
}
static dim3 swiglu_grid(size_t rows, int M, int num_sms) {
    const int threads = swiglu_threads(M);
    const unsigned gx = static_cast<unsigned>((M / 8 + threads - 1) / threads);
    size_t gy = (static_cast<size_t>(num_sms) * (2048 / threads) + gx - 1) / gx;
    if (gy > rows) gy = rows;
    if (gy < 1) gy = 1;
    if (gy > 65535) gy = 65535;
    return dim3(gx, static_cast<unsigned>(gy));
}
void swiglu_fwd(const void* x, void* y, void* y_fp8, const float* fp8_scale, float* amax, size_t rows, int M, int num_sms, cudaStream_t s,
                const int* rows_limit) {
    swiglu_fwd_kernel<<<swiglu_grid(rows, M, num_sms), swiglu_threads(M), 0, s>>>((const bf16*)x, (bf16*)y, (uint8_t*)y_fp8, fp8_scale, amax, rows, M, rows_limit);
}
void swiglu_bwd(const void* dy, const void* x, void* dx, size_t rows, int M, int num_sms, cudaStream_t s, const int* rows_limit, void* dx_fp8,
                const float* fp8_scale, float* amax_out) {
    swiglu_bwd_kernel<<<swiglu_grid(rows, M, num_sms), swiglu_threads(M), 0, s>>>((const bf16*)dy, (const bf16*)x, (bf16*)dx, rows, M, rows_limit,
                                                                             (uint8_t*)dx_fp8, fp8_scale, amax_out);
}
// Zero the output matrices of groups that own no rows (their wgrad tiles are never scheduled): out [G, per_group] of `elem` bytes.
__global__ void __launch_bounds__(256) zero_empty_groups_kernel(uint4* __restrict__ out, const int* __restrict__ offsets, size_t vec_per_group) {
    const int g = blockIdx.y;
    if (offsets[g + 1] != offsets[g]) return;
    uint4* dst = out + static_cast<size_t>(g) * vec_per_group;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < vec_per_group; i += static_cast<size_t>(gridDim.x) * blockDim.x)
        dst[i] = make_uint4(0, 0, 0, 0);
}
void zero_empty_groups(void* out, const int* offsets, int groups, size_t bytes_per_group, cudaStream_t s) {
    zero_empty_groups_kernel<<<dim3(32, groups), 256, 0, s>>>((uint4*)out, offsets, bytes_per_group / 16);
}
void qk_norm_rope_fwd(const void* qkv, const void* qw, const void* kw, const int* pos, void* out, float* q_rstd, float* k_rstd, size_t tokens, int Hq,
                      int Hkv, float eps, float theta, int lim_h, int lim_w, int num_sms, cudaStream_t s) {
#define SG_QR(TOK)                                                                                                                               \
    qk_norm_rope_kernel<false, TOK><<<grid_for(tokens, TOK, num_sms, 64 / TOK), 256, 0, s>>>((const bf16*)qkv, nullptr, (const bf16*)qw, (const bf16*)kw, \
                                                                                             pos, (bf16*)out, q_rstd, k_rstd, nullptr, nullptr, tokens, \
                                                                                             Hq, Hkv, eps, log2f(theta), lim_h, lim_w)
    if (Hq + 2 * Hkv > ROPE_SPLIT_HEADS) SG_QR(4);
    else SG_QR(8);
#undef SG_QR
}
void qk_norm_rope_bwd(const void* d_out, const void* qkv_pre, const void* qw, const void* kw, const int* pos, void* d_qkv, float* q_rstd,
                      float* k_rstd, float* dqw, float* dkw, size_t tokens, int Hq, int Hkv, float eps, float theta, int lim_h, int lim_w, int num_sms,
                      cudaStream_t s) {
    qk_norm_rope_kernel<true, 8><<<grid_for(tokens, 8, num_sms, 4), 256, 0, s>>>((const bf16*)d_out, (const bf16*)qkv_pre, (const bf16*)qw,
                                                                                     (const bf16*)kw, pos, (bf16*)d_qkv, q_rstd, k_rstd, dqw, dkw, tokens,
                                                                                     Hq, Hkv, eps, log2f(theta), lim_h, lim_w);
}
void embedding_fwd(const int* tokens, const void* table, void* out, size_t n, int C, int V, int* error_flag, int num_sms, cudaStream_t s) {
    embedding_fwd_kernel<<<grid_for(n * (C / 8), 256, num_sms), 256, 0, s>>>(tokens, (const bf16*)table, (bf16*)out, n, C, V, error_flag);
}
void embedding_bwd(const int* tokens, const void* d_out, void* d_table, int grad_fp32, size_t n, int C, int num_sms, cudaStream_t s) {
    const int grid = grid_for(n * (C / 2), 256, num_sms);
    if (grad_fp32) embedding_bwd_kernel<float><<<grid, 256, 0, s>>>(tokens, (const bf16*)d_out, (float*)d_table, n, C);
    else embedding_bwd_kernel<bf16><<<grid, 256, 0, s>>>(tokens, (const bf16*)d_out, (bf16*)d_table, n, C);
}
void embedding_bwd_sorted(const int* sorted_ids, const long long* order, const void* d_out, void* d_table, int grad_fp32, int n, int C, int V, int vec,
                          cudaStream_t s) {
    if (n <= 0) return;
    const int cols = vec == 8 ? EMB_COLS : 2 * EMB_COLS;       // narrow rows: two passes of a CTA, or its launch costs more than its work
    const dim3 grid(n, (C + cols - 1) / cols);
#define SG_EB(G, VEC) embedding_bwd_sorted_kernel<G, VEC><<<grid, EMB_COLS / VEC, 0, s>>>(sorted_ids, order, (const bf16*)d_out, (G*)d_table, n, C, V)
    if (grad_fp32) { if (vec == 8) SG_EB(float, 8); else if (vec == 2) SG_EB(float, 2); else SG_EB(float, 1); }
    else { if (vec == 8) SG_EB(bf16, 8); else if (vec == 2) SG_EB(bf16, 2); else SG_EB(bf16, 1); }
#undef SG_EB
}
void zero_fill(void* p, size_t bytes, int num_sms, cudaStream_t s) { zero_fill_kernel<<<grid_for(bytes / 16, 256, num_sms), 256, 0, s>>>((uint4*)p, bytes / 16); }
void cross_entropy_fwd_bwd(void* logits, const int* targets, float* loss, const float* scale_ptr, float scale_host, int rows, int V, int ld,
                           int write_grad, const float* row_weight, const int* kd_idx, const float* kd_logp, int kd_k, float kd_weight, float* kd_loss,
                           cudaStream_t s) {
    cross_entropy_fwd_bwd_kernel<false><<<rows, 1024, 0, s>>>((bf16*)logits, nullptr, nullptr, targets, loss, scale_ptr, scale_host, V, ld, write_grad, row_weight,
                                                              kd_idx, kd_logp, kd_k, kd_weight, kd_loss);
}
void cross_entropy_fwd_bwd_fp8(const void* logits, void* d8, const float* q_scale, const int* targets, float* loss, const float* scale_ptr, float scale_host, int rows,
                               int V, int ld, cudaStream_t s) {
    cross_entropy_fwd_bwd_kernel<true><<<rows, 1024, 0, s>>>((bf16*)logits, (uint8_t*)d8, q_scale, targets, loss, scale_ptr, scale_host, V, ld, 1, nullptr, nullptr,
                                                             nullptr, 0, 0.f, nullptr);
}
void quantize_fp8(const void* x, void* q, const float* scale, float* amax, size_t n, int e5m2, int num_sms, cudaStream_t s, const int* rows_limit,
                  int row_len) {
    const int grid = grid_for(n / 8, 256, num_sms);
    if (e5m2) quantize_fp8_kernel<true><<<grid, 256, 0, s>>>((const bf16*)x, (uint8_t*)q, scale, amax, n, rows_limit, row_len);
    else quantize_fp8_kernel<false><<<grid, 256, 0, s>>>((const bf16*)x, (uint8_t*)q, scale, amax, n, rows_limit, row_len);
}
void dequantize_fp8(const void* q, const float* scale, void* out, size_t n, int e5m2, int num_sms, cudaStream_t s) {
    if (n == 0) return;
    const int grid = grid_for((n + 15) / 16, 256, num_sms);
    if (e5m2) dequantize_fp8_kernel<true><<<grid, 256, 0, s>>>((const uint8_t*)q, scale, (bf16*)out, n);
    else dequantize_fp8_kernel<false><<<grid, 256, 0, s>>>((const uint8_t*)q, scale, (bf16*)out, n);
}
void amax_bf16(const void* x, float* amax, size_t n, int num_sms, cudaStream_t s, const int* rows_limit, int row_len) {
    amax_kernel<<<grid_for(n / 8, 256, num_sms), 256, 0, s>>>((const bf16*)x, amax, n, rows_limit, row_len);
}
void sumsq(const void* x, int is_fp32, float* partial, int nblocks, size_t n, cudaStream_t s) {
    if (is_fp32) sumsq_kernel<float><<<nblocks, 512, 0, s>>>((const float*)x, partial, n);
    else sumsq_kernel<bf16><<<nblocks, 512, 0, s>>>((const bf16*)x, partial, n);
}
void adamw_fp32(void* p, int p_fp32, const void* g, int g_fp32, float* m, float* v, const uint8_t* mask, const float* hp, size_t n, int num_sms,
                cudaStream_t s) {
    const int grid = grid_for(n / 8, 256, num_sms);
    if (p_fp32 && g_fp32) adamw_fp32_kernel<float, float><<<grid, 256, 0, s>>>((float*)p, (const float*)g, m, v, mask, hp, n);
    else if (p_fp32) adamw_fp32_kernel<float, bf16><<<grid, 256, 0, s>>>((float*)p, (const bf16*)g, m, v, mask, hp, n);
    else if (g_fp32) adamw_fp32_kernel<bf16, float><<<grid, 256, 0, s>>>((bf16*)p, (const float*)g, m, v, mask, hp, n);
    else adamw_fp32_kernel<bf16, bf16><<<grid, 256, 0, s>>>((bf16*)p, (const bf16*)g, m, v, mask, hp, n);
}
const char* adamw_8bit(void* p, int p_fp32, const void* g, int g_fp32, void* m8, void* v8, void* ms, void* vs, const uint8_t* mask, int block_mask,
                const float* hp, size_t n, int num_sms, cudaStream_t s) {
#define SG_A8(PT, GT, BM)                                                                                                                       \
    do {                                                                                                                                        \
        constexpr int smem = adam8_stages<PT, GT>() * adam8_slot_bytes<PT, GT>();                                                                 \
        static_assert(3 * (smem + 2048) <= 227 * 1024, "three CTAs per SM");                                                                     \
        static std::atomic<uint64_t> limit{0};                                                                                                  \
        if (!raise_smem_limit(reinterpret_cast<const void*>(adamw_8bit_kernel<PT, GT, BM>), smem, limit)) return "raising the shared-memory limit failed (8-bit AdamW)"; \
        const int grid = grid_for(n / 8, ADAM8_THREADS, num_sms, 3);   /* the resident CTAs, each with a full ring */      \
        adamw_8bit_kernel<PT, GT, BM><<<grid, ADAM8_THREADS, smem, s>>>((PT*)p, (const GT*)g, (int8_t*)m8, (uint8_t*)v8, (__half*)ms, (__half*)vs, mask, hp, n); \
    } while (0)
    if (block_mask) {
        if (p_fp32 && g_fp32) SG_A8(float, float, true); else if (p_fp32) SG_A8(float, bf16, true); else if (g_fp32) SG_A8(bf16, float, true); else SG_A8(bf16, bf16, true);
    } else {
        if (p_fp32 && g_fp32) SG_A8(float, float, false); else if (p_fp32) SG_A8(float, bf16, false); else if (g_fp32) SG_A8(bf16, float, false); else SG_A8(bf16, bf16, false);
    }
#undef SG_A8
    return cudaGetLastError() == cudaSuccess ? nullptr : "8-bit AdamW launch failed";
}

}  // namespace sg
