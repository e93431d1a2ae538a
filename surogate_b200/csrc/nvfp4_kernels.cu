// NVFP4 quantisation for sm_100a: E2M1 values with two-level scaling — one FP8 (UE4M3) scale per 16 elements of
// the contraction dimension and one fp32 scale per tensor.
//
//   global encode  ge = (448 * 6) / amax(tensor)                 (device scalar, from an abs-max pass)
//   block scale    sf = e4m3( amax(block16) * ge / 6 )           (stored; decodes to sfd)
//   element        q  = e2m1( x * ge / sfd )                     (round-to-nearest-even, or stochastic for gradients)
//   decode         x ~= q * sfd / ge        =>  GEMM result is scaled by 1 / (ge_a * ge_b) in its epilogue
//
// Scale factors are written in the 128x4 "atom" layout the tensor core reads through TMEM: for row r and 16-element
// block kb, byte ((r/128)*atoms_k + kb/4)*512 + (r%32)*16 + ((r%128)/32)*4 + kb%4.
//
// Kernels: row-wise quantise (blocks along the contiguous dimension), transpose-quantise (blocks along the row
// dimension of the input, i.e. the quantised transpose; optional 16x16 random Hadamard transform applied along the
// block before quantisation, used for weight-gradient operands), 2-D 16x16 weight blocks (one scale shared by a
// 16x16 tile so W and W^T quantise consistently), and dequantise (tests, bf16 fallback GEMM).
//
// Replaces recipes/nvfp4/kernels/{quant_fp4,quant_nvfp4_cutlass,hadamard}.cu of the reference.
#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nvfp4_kernels.h"

namespace sg {

using bf16 = __nv_bfloat16;
using bf162 = __nv_bfloat162;

__device__ __forceinline__ size_t sf_offset(int r, int kb, int atoms_k) {
    return (static_cast<size_t>(r >> 7) * atoms_k + (kb >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (kb & 3);
}

// counter-based hash -> uniform float in [0,1)
__device__ __forceinline__ float hash_uniform(uint32_t seed, uint64_t idx) {
    uint64_t z = idx + 0x9E3779B97F4A7C15ull * (static_cast<uint64_t>(seed) + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return static_cast<float>(static_cast<uint32_t>(z >> 40)) * (1.0f / 16777216.0f);
}

// two e2m1 codes (4 bits: sign | 3-bit magnitude index into {0, .5, 1, 1.5, 2, 3, 4, 6}) in one byte, low nibble first; round to
// nearest even on the grid, saturating: one conversion instruction per pair instead of a chain of seven compares per element.
// The addition turns -0 into +0, so that a zero always has code 0.
__device__ __forceinline__ uint32_t e2m1x2_rn(float lo, float hi) {
    return __nv_cvt_float2_to_fp4x2(make_float2(lo + 0.f, hi + 0.f), __NV_E2M1, cudaRoundNearest);
}
__device__ __forceinline__ float2 e2m1x2_value(uint32_t codes) {
    return __half22float2(__half2(__nv_cvt_fp4x2_to_halfraw2(static_cast<__nv_fp4x2_storage_t>(codes), __NV_E2M1)));
}
__device__ __forceinline__ float e2m1_value(uint32_t code) {
    const float mag[8] = {0.f, 0.5f, 1.f, 1.5f, 2.f, 3.f, 4.f, 6.f};
    const float m = mag[code & 7];
    return (code & 8) ? -m : m;
}
// stochastic rounding between the two neighbouring grid points (unbiased for |v| <= 6).  From 1 upwards the grid is the floats with
// one mantissa bit, so the lower neighbour is a truncation and its code a shift; below 1 it is 0 or 0.5.
__device__ __forceinline__ uint32_t e2m1_sr(float v, float u) {
    const uint32_t sign = v < 0.f ? 8u : 0u;
    const float a = fminf(fabsf(v), 6.f);
    const uint32_t bits = __float_as_uint(a);
    const bool big = a >= 1.f, half = a >= 0.5f;
    const uint32_t lo = big ? (bits >> 22) - 252u : (half ? 1u : 0u);
    const float base = big ? __uint_as_float(bits & 0xFFC00000u) : (half ? 0.5f : 0.f);
    const float inv_gap = big ? __uint_as_float((255u << 23) - (bits & 0x7F800000u)) : 2.f;   // 1 / (2^e / 2)
    return sign | (lo + (u < (a - base) * inv_gap ? 1u : 0u));                                  // a = 6 has no remainder: stays code 7
}

__device__ __forceinline__ float decode_e4m3(uint8_t b) {
    __nv_fp8_e4m3 t;
    t.__x = b;
    return static_cast<float>(t);
}

// quantise one block of 16 floats: returns 8 packed bytes in `out` (two uint32) and the scale byte
template <bool SR>
__device__ __forceinline__ uint8_t quant_block16(const float (&v)[16], float ge, float forced_amax, uint32_t seed, uint64_t base_idx, uint32_t (&out)[2]) {
    float amax = forced_amax;
    if (forced_amax < 0.f) {
        amax = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
    }
    const uint8_t sfb = __nv_cvt_float_to_fp8(__fdiv_rn(__fmul_rn(amax, ge), 6.f), __NV_SATFINITE, __NV_E4M3);
    const float sfd = decode_e4m3(sfb);
    const float mul = sfd > 0.f ? ge / sfd : 0.f;
    out[0] = out[1] = 0;
#pragma unroll
    for (int i = 0; i < 16; i += 2) {      // element 2j in the low nibble of byte j
        const float s0 = v[i] * mul, s1 = v[i + 1] * mul;
        const uint32_t c = SR ? e2m1_sr(s0, hash_uniform(seed, base_idx + i)) | (e2m1_sr(s1, hash_uniform(seed, base_idx + i + 1)) << 4) : e2m1x2_rn(s0, s1);
        out[i >> 3] |= c << ((i & 7) * 4);
    }
    return sfb;
}

// Four-over-six (round to nearest only): the block is quantised twice, once with its abs-max mapped to the top grid value 6 and
// once mapped to 4 (the grid {0, .5, 1, 1.5, 2, 3, 4} then has no gap between 4 and 6 to fall into), and the mapping with the smaller
// squared reconstruction error is kept.  `err_group` > 1 shares the decision between that many adjacent lanes (16 for the 16 x 16
// weight tiles, whose rows must agree on one scale).  The tensor encode factor is 1536 (= 256 * 6 = 384 * 4), so that both block
// scales stay inside the UE4M3 range.
__device__ __forceinline__ uint8_t quant_block16_4o6(const float (&v)[16], float ge, float forced_amax, uint32_t (&out)[2], int err_group) {
    float amax = forced_amax;
    if (forced_amax < 0.f) {
        amax = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
    }
    uint8_t sfb[2];
    uint32_t codes[2][2];
    float err[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        sfb[t] = __nv_cvt_float_to_fp8(__fdiv_rn(__fmul_rn(amax, ge), t == 0 ? 6.f : 4.f), __NV_SATFINITE, __NV_E4M3);
        const float sfd = decode_e4m3(sfb[t]);
        const float mul = sfd > 0.f ? ge / sfd : 0.f;
        codes[t][0] = codes[t][1] = 0;
        float e = 0.f;
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const float s0 = v[i] * mul, s1 = v[i + 1] * mul;
            const uint32_t c = e2m1x2_rn(s0, s1);
            const float2 q = e2m1x2_value(c);
            // error in units of x * ge; the operations are spelled out because nearly equal sums decide here
            const float d0 = __fmul_rn(__fsub_rn(q.x, __fmul_rn(v[i], mul)), sfd), d1 = __fmul_rn(__fsub_rn(q.y, __fmul_rn(v[i + 1], mul)), sfd);
            e = __fmaf_rn(d1, d1, __fmaf_rn(d0, d0, e));
            codes[t][i >> 3] |= c << ((i & 7) * 4);
        }
        err[t] = e;
    }
    for (int o = err_group >> 1; o > 0; o >>= 1) {
        err[0] += __shfl_xor_sync(0xffffffffu, err[0], o);
        err[1] += __shfl_xor_sync(0xffffffffu, err[1], o);
    }
    const int pick = err[1] < err[0] ? 1 : 0;
    out[0] = pick ? codes[1][0] : codes[0][0];
    out[1] = pick ? codes[1][1] : codes[0][1];
    return pick ? sfb[1] : sfb[0];
}

__device__ __forceinline__ void load16(const bf16* p, float (&v)[16]) {
    const uint4 a = *reinterpret_cast<const uint4*>(p), b = *reinterpret_cast<const uint4*>(p + 8);
    const bf162* pa = reinterpret_cast<const bf162*>(&a);
    const bf162* pb = reinterpret_cast<const bf162*>(&b);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pb[i]);
        v[2 * i] = x.x; v[2 * i + 1] = x.y; v[8 + 2 * i] = y.x; v[8 + 2 * i + 1] = y.y;
    }
}

// in-register 16-point Hadamard with random signs (orthonormal: scaled by 1/4)
__device__ __forceinline__ void hadamard16(float (&v)[16], uint32_t sign_mask) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if ((sign_mask >> i) & 1u) v[i] = -v[i];
#pragma unroll
    for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if ((i & h) == 0) {
                const float a = v[i], b = v[i + h];
                v[i] = a + b;
                v[i + h] = a - b;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= 0.25f;
}

// ------------------------------------------------------------------------------------------ output tile
// Both quantisers work on tiles of 128 output rows x 128 elements (8 blocks of 16): the codes (64 bytes a row) and the scales (two
// 512-byte atoms) are collected in shared memory and leave as whole sectors.  Written straight from the threads that compute them, each
// scale is a one-byte store into a sector of its own, and the codes of a transpose are 8-byte stores a whole row apart.
// Stochastic rounding issues about 500 instructions per block of 16, so a tensor of few tiles is bound by the SMs that it occupies: with at
// most one tile per SM, tiles are cut into QT_FEW_ROWS rows (each a quarter of the words of its two atoms).
constexpr int QT_ROWS = 128, QT_FEW_ROWS = 32, QT_COLS = 128, QT_BLOCKS = QT_COLS / 16, QT_PITCH = QT_COLS / 2 + 8;
template <int ROWS> struct QTile {
    uint8_t q[ROWS * QT_PITCH];
    alignas(16) uint8_t sf[QT_ROWS * QT_BLOCKS];
    __device__ __forceinline__ void put(int r, int b, const uint32_t (&codes)[2], uint8_t scale) {
        *reinterpret_cast<uint2*>(q + r * QT_PITCH + b * 8) = make_uint2(codes[0], codes[1]);
        sf[(b >> 2) * 512 + (r & 31) * 16 + (r >> 5) * 4 + (b & 3)] = scale;
    }
    // `rows` x `kblocks`: the whole output; (row0, kb0): this tile's origin.  Scales of rows and blocks behind the end are zero, so the
    // buffer needs no clearing beforehand.
    __device__ __forceinline__ void write(uint8_t* __restrict__ qg, uint8_t* __restrict__ sfg, int row0, int kb0, int rows, int kblocks, int atoms_k) const {
        for (int i = threadIdx.x; i < ROWS * QT_BLOCKS; i += blockDim.x) {
            const int r = i / QT_BLOCKS, b = i % QT_BLOCKS;
            if (row0 + r < rows && kb0 + b < kblocks)
                *reinterpret_cast<uint2*>(qg + (static_cast<size_t>(row0 + r) * kblocks + kb0 + b) * 8) = *reinterpret_cast<const uint2*>(q + r * QT_PITCH + b * 8);
        }
        const int atom0 = kb0 >> 2;
        if (threadIdx.x < 64 && atom0 + (threadIdx.x >> 5) < atoms_k) {
            uint4* atom = reinterpret_cast<uint4*>(sfg + (static_cast<size_t>(row0 >> 7) * atoms_k + atom0) * 512);
            if (ROWS == QT_ROWS) atom[threadIdx.x] = reinterpret_cast<const uint4*>(sf)[threadIdx.x];
            else reinterpret_cast<uint32_t*>(atom + threadIdx.x)[(row0 >> 5) & 3] = reinterpret_cast<const uint32_t*>(sf)[threadIdx.x * 4];
        }
    }
};

// ------------------------------------------------------------------------------------------ row-wise quantise
// x [rows, K] bf16 (K % 16 == 0) -> q [rows, K/2] bytes, sf in atom layout.  block2d: scales are shared by 16x16 tiles (rows % 16 == 0).
// 256 threads per 128 x 128 tile, four blocks each.  Bound by instruction issue: about 12 per element with four-over-six (both
// candidates' codes and error sums), about 30 with stochastic rounding (the hash).  24576 x 4096 on B200: four-over-six 958 -> 95 us
// (2.7 TB/s of the 258 MB it must move), plain 151 -> 64 us, stochastic 476 -> 197 us; before, the codes came from a chain of compares,
// their values from a table in local memory, and every scale byte was a store of its own.
// Stochastic, 256 x 1024: scale bytes stored one by one 5.8 us, whole tiles 7.7 us, 32 rows 3.4 us.
template <bool SR, int ROWS>
__global__ void __launch_bounds__(256) nvfp4_quantize_rows_kernel(const bf16* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ sf,
                                                                  const float* __restrict__ amax_tensor, int rows, int K, int atoms_k, uint32_t seed,
                                                                  int block2d, int four_over_six) {
    __shared__ QTile<ROWS> out_tile;
    const float at = __ldg(amax_tensor);
    const float ge = at > 0.f ? __fdiv_rn(four_over_six ? 1536.f : 2688.f, at) : 1.f;
    const int kblocks = K / 16;
    const int tiles_k = (kblocks + QT_BLOCKS - 1) / QT_BLOCKS;
    const int row0 = static_cast<int>(blockIdx.x / tiles_k) * ROWS, kb0 = static_cast<int>(blockIdx.x % tiles_k) * QT_BLOCKS;
#pragma unroll 1
    for (int it = 0; it < ROWS * QT_BLOCKS / 256; ++it) {
        int r, b;
        if (block2d) {   // lanes walk down the 16 rows of a 16x16 tile, so that its abs-max and its decision are 16-lane shuffles
            const int tile = it * 16 + (threadIdx.x >> 4);
            r = (tile / QT_BLOCKS) * 16 + (threadIdx.x & 15);
            b = tile % QT_BLOCKS;
        } else {
            const int i = it * 256 + threadIdx.x;
            r = i / QT_BLOCKS;
            b = i % QT_BLOCKS;
        }
        const bool live = row0 + r < rows && kb0 + b < kblocks;   // rows is a multiple of 16 in the tile path: 16-lane groups agree
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
        if (live) load16(x + static_cast<size_t>(row0 + r) * K + (kb0 + b) * 16, v);
        float forced = -1.f;
        if (block2d) {
            float m = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) m = fmaxf(m, fabsf(v[i]));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            forced = m;
        }
        uint32_t out[2];
        uint8_t sfb;
        if (!SR && four_over_six) sfb = quant_block16_4o6(v, ge, forced, out, block2d ? 16 : 1);
        else sfb = quant_block16<SR>(v, ge, forced, seed, static_cast<uint64_t>(row0 + r) * K + (kb0 + b) * 16, out);
        out_tile.put(r, b, out, live ? sfb : static_cast<uint8_t>(0));
    }
    __syncthreads();
    out_tile.write(q, sf, row0, kb0, rows, kblocks, atoms_k);
}

// ------------------------------------------------------------------------------------------ transpose-quantise
// x [R, C] bf16 -> quantised x^T: q [C, R/2], sf for (row = c, block = r/16).  R % 64 == 0, C % 64 == 0.
// The 128 x 128 input tile passes through shared memory as bf16; a lane owns two adjacent columns (4-byte reads, no bank conflicts).
// 24576 x 4096 on B200: four-over-six 1284 -> 98 us, with the Hadamard transform 1316 -> 118 us, stochastic with it 349 -> 221 us.
// Stochastic, 256 x 1024: 64 x 64 tiles 6.2 us, whole tiles 7.7 us, 32 rows 3.9 us.
template <bool SR, bool RHT, int ROWS, int THREADS>
__global__ void __launch_bounds__(THREADS) nvfp4_quantize_transpose_kernel(const bf16* __restrict__ x, uint8_t* __restrict__ q, uint8_t* __restrict__ sf,
                                                                       const float* __restrict__ amax_tensor, int R, int C, int atoms_k, uint32_t seed,
                                                                       uint32_t sign_mask, int four_over_six) {
    constexpr int QX_PITCH = ROWS + 8;        // bf16 elements per staged row
    __shared__ QTile<ROWS> out_tile;
    __shared__ alignas(16) bf16 tile[QT_COLS * QX_PITCH];
    const int tiles_c = (C + QT_ROWS - 1) / QT_ROWS * (QT_ROWS / ROWS);
    const int c0 = static_cast<int>(blockIdx.x % tiles_c) * ROWS, r0 = static_cast<int>(blockIdx.x / tiles_c) * QT_COLS;
#pragma unroll
    for (int it = 0; it < QT_COLS * ROWS / 8 / THREADS; ++it) {
        const int i = it * THREADS + threadIdx.x, rr = i / (ROWS / 8), cv = (i % (ROWS / 8)) * 8;
        uint4 raw = make_uint4(0, 0, 0, 0);
        if (r0 + rr < R && c0 + cv < C) raw = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(r0 + rr) * C + c0 + cv);
        *reinterpret_cast<uint4*>(tile + rr * QX_PITCH + cv) = raw;
    }
    __syncthreads();
    const float at = __ldg(amax_tensor);
    // the Hadamard transform is orthonormal, so the tensor abs-max bound grows by at most 4x; keep head-room for it
    const float enc = (!SR && four_over_six) ? 1536.f : 2688.f;
    const float ge = at > 0.f ? (RHT ? enc / (at * 2.f) : enc / at) : 1.f;
#pragma unroll 1
    for (int it = 0; it < ROWS / 2 * QT_BLOCKS / THREADS; ++it) {
        const int i = it * THREADS + threadIdx.x, pair = i % (ROWS / 2), rb = i / (ROWS / 2);   // columns 2 pair, 2 pair + 1; 16-row block
        bf162 raw[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) raw[k] = *reinterpret_cast<const bf162*>(tile + (rb * 16 + k) * QX_PITCH + 2 * pair);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 2 * pair + h;
            float v[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = __bfloat162float(h ? raw[k].y : raw[k].x);
            if (RHT) hadamard16(v, sign_mask);
            uint32_t out[2];
            const uint8_t sfb = (!SR && four_over_six) ? quant_block16_4o6(v, ge, -1.f, out, 1)
                                                        : quant_block16<SR>(v, ge, -1.f, seed, static_cast<uint64_t>(c0 + c) * R + r0 + rb * 16, out);
            out_tile.put(c, rb, out, c0 + c < C && r0 + rb * 16 < R ? sfb : static_cast<uint8_t>(0));
        }
    }
    __syncthreads();
    out_tile.write(q, sf, c0, r0 >> 4, C, R >> 4, atoms_k);
}

// ------------------------------------------------------------------------------------------ dequantise
__global__ void __launch_bounds__(256) nvfp4_dequantize_kernel(const uint8_t* __restrict__ q, const uint8_t* __restrict__ sf,
                                                               const float* __restrict__ amax_tensor, float amax_div, bf16* __restrict__ out, int rows,
                                                               int K, int atoms_k, float encode) {
    const float at = __ldg(amax_tensor);
    const float inv_ge = at > 0.f ? at * amax_div / encode : 1.f;
    const int kblocks = K / 16;
    const size_t total = static_cast<size_t>(rows) * kblocks;
    for (size_t b = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; b < total; b += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int r = static_cast<int>(b / kblocks), kb = static_cast<int>(b % kblocks);
        const uint2 raw = *reinterpret_cast<const uint2*>(q + static_cast<size_t>(r) * (K / 2) + kb * 8);
        const float s = decode_e4m3(sf[sf_offset(r, kb, atoms_k)]) * inv_ge;
        const uint32_t w[2] = {raw.x, raw.y};
        bf16 o[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = __float2bfloat16_rn(e2m1_value((w[i >> 3] >> ((i & 7) * 4)) & 15u) * s);
        *reinterpret_cast<uint4*>(out + static_cast<size_t>(r) * K + kb * 16) = *reinterpret_cast<const uint4*>(&o[0]);
        *reinterpret_cast<uint4*>(out + static_cast<size_t>(r) * K + kb * 16 + 8) = *reinterpret_cast<const uint4*>(&o[8]);
    }
}

// ============================================================================================ launchers
static int q_grid(size_t items, int num_sms) {
    size_t g = (items + 255) / 256;
    const size_t cap = static_cast<size_t>(num_sms) * 8;
    return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}
void nvfp4_quantize_rows(const void* x, void* q, void* sf, const float* amax_tensor, int rows, int K, int stochastic, uint32_t seed, int block2d,
                         int num_sms, cudaStream_t s, int four_over_six) {
    const int atoms_k = (K / 16 + 3) / 4;
    if (rows <= 0 || K <= 0) return;
    const unsigned grid = static_cast<unsigned>((rows + QT_ROWS - 1) / QT_ROWS) * static_cast<unsigned>((K / 16 + QT_BLOCKS - 1) / QT_BLOCKS);
#define SG_QR(SR, ROWS, FOS)                                                                                                                            \
    nvfp4_quantize_rows_kernel<SR, ROWS><<<grid * (QT_ROWS / ROWS), 256, 0, s>>>((const bf16*)x, (uint8_t*)q, (uint8_t*)sf, amax_tensor, rows, K, atoms_k, seed, \
                                                                                 block2d, FOS)
    if (stochastic && grid <= static_cast<unsigned>(num_sms)) SG_QR(true, QT_FEW_ROWS, 0);
    else if (stochastic) SG_QR(true, QT_ROWS, 0);
    else SG_QR(false, QT_ROWS, four_over_six);
#undef SG_QR
}
void nvfp4_quantize_transpose(const void* x, void* q, void* sf, const float* amax_tensor, int R, int C, int stochastic, int hadamard, uint32_t seed,
                              uint32_t sign_mask, int num_sms, cudaStream_t s, int four_over_six) {
    const int atoms_k = (R / 16 + 3) / 4;
    if (R <= 0 || C <= 0) return;
    const unsigned grid = static_cast<unsigned>((C + QT_ROWS - 1) / QT_ROWS) * static_cast<unsigned>((R + QT_COLS - 1) / QT_COLS);
    const bf16* xp = (const bf16*)x;
    uint8_t* qp = (uint8_t*)q;
    uint8_t* sp = (uint8_t*)sf;
#define SG_QX(SR, RHT, ROWS, TH)                                                                                                                        \
    nvfp4_quantize_transpose_kernel<SR, RHT, ROWS, TH><<<grid * (QT_ROWS / ROWS), TH, 0, s>>>(xp, qp, sp, amax_tensor, R, C, atoms_k, seed, sign_mask, four_over_six)
    const bool few = grid <= static_cast<unsigned>(num_sms);
    if (stochastic && hadamard) { if (few) SG_QX(true, true, QT_FEW_ROWS, 128); else SG_QX(true, true, QT_ROWS, 256); }
    else if (stochastic) { if (few) SG_QX(true, false, QT_FEW_ROWS, 128); else SG_QX(true, false, QT_ROWS, 256); }
    else if (hadamard) SG_QX(false, true, QT_ROWS, 256);
    else SG_QX(false, false, QT_ROWS, 256);
#undef SG_QX
}
void nvfp4_dequantize(const void* q, const void* sf, const float* amax_tensor, float amax_div, void* out, int rows, int K, int num_sms, cudaStream_t s,
                      float encode) {
    const int atoms_k = (K / 16 + 3) / 4;
    nvfp4_dequantize_kernel<<<q_grid(static_cast<size_t>(rows) * (K / 16), num_sms), 256, 0, s>>>((const uint8_t*)q, (const uint8_t*)sf, amax_tensor,
                                                                                                  amax_div, (bf16*)out, rows, K, atoms_k, encode);
}

}  // namespace sg
