// Dense GEMM for sm_100a: D[M,N] = alpha * sa * sb * (A[M,K] . B[N,K]^T) (+ D), fp32 accumulation in TMEM.
//
// * Inputs bf16 (tcgen05 kind::f16) or FP8 e4m3/e5m2 in any mix (kind::f8f6f4).
// * Each operand may be K-major ([rows, K] row-major) or MN-major ([K, rows] row-major).  Forward (x.W^T),
//   dgrad (dy.W) and wgrad (dy^T.x) therefore all read the tensors as they lie in memory: no transposed
//   copies of weights or activations are ever made, for bf16 or FP8.
// * Persistent, warp-specialised: warp 0 issues TMA loads into a multi-stage shared-memory ring, warp 1
//   issues tcgen05.mma (one elected thread), warps 2-5 drain the accumulator from TMEM (tcgen05.ld), apply
//   the scales and write bf16 / fp32.  Two accumulators (2 x BN TMEM columns) let the epilogue of tile i
//   overlap the main loop of tile i+1.
// * Optional epilogue extras: accumulate into D (gradient accumulation), running abs-max of the output.
// * No cluster multicast anywhere (loads are per-CTA), so the same kernel is used at any GPU count.
//
// Replaces the cuBLASLt calls of the reference (csrc/src/kernels/matmul.cpp:447-1000).
#include <cuda_fp8.h>

#include <algorithm>

#include "gemm_sm100.h"
#include "launch_limits.h"
#include "sm100_ptx.cuh"

namespace sg {

constexpr int BM = 128;
constexpr int TILE_K_BYTES = 128;   // one swizzle row
constexpr int A_STAGE_BYTES = BM * TILE_K_BYTES;
constexpr int GEMM_THREADS = 192;
constexpr int GROUP_M = 8;

template <int BN> struct Cfg {
    static constexpr int B_STAGE_BYTES = BN * TILE_K_BYTES;
    static constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
    static constexpr int STAGES = (BN == 256) ? 4 : 6;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align slack*/ + 256 /*barriers*/;
    static constexpr int TMEM_COLS = 2 * BN;
};

// What one output tile needs to know.  Coordinates are TMA coordinates (elements).
struct TileInfo {
    int a_row0;   // A: row (K-major) or M-column (MN-major) coordinate of the tile
    int b_row0;   // B: row (K-major) or N-column (MN-major) coordinate of the tile
    int a_k0;     // first contraction coordinate in A
    int b_k0;     // first contraction coordinate in B
    int num_k;    // contraction blocks
    int d_row0, d_col0;   // output tile origin
    int m_end, n_end;     // exclusive store limits
    long long d_off;      // element offset of this tile's output matrix inside D
};

// Tile schedules.  mode 0: one dense problem.  mode 1: rows of A / D are grouped (MoE forward and dgrad): group g owns rows
// [offs[g], offs[g+1]) (multiples of 128) and uses B block g.  mode 2: the contraction is grouped (MoE wgrad): group g
// contracts rows [offs[g], offs[g+1]) of both operands into output matrix g.
__device__ __forceinline__ int find_group(const int* tile_start, int num_groups, int tile) {
    int lo = 0, hi = num_groups;  // largest g with tile_start[g] <= tile
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tile_start[mid] <= tile) lo = mid; else hi = mid;
    }
    return lo;
}

template <int BN>
__device__ __forceinline__ TileInfo get_tile(const GemmParams& p, const int* tile_start, int tile, int BK) {
    TileInfo t;
    const int num_n = (p.N + BN - 1) / BN;
    if (p.mode == 0) {
        const int num_m = (p.M + BM - 1) / BM;
        const int per_group = GROUP_M * num_n;
        const int group = tile / per_group;
        const int first_m = group * GROUP_M;
        const int gsize = min(num_m - first_m, GROUP_M);
        const int r = tile - group * per_group;
        const int m_blk = first_m + r % gsize, n_blk = r / gsize;
        t.a_row0 = t.d_row0 = m_blk * BM;
        t.b_row0 = t.d_col0 = n_blk * BN;
        t.a_k0 = t.b_k0 = 0;
        t.num_k = (p.K + BK - 1) / BK;
        t.m_end = p.M;
        t.n_end = p.N;
        t.d_off = 0;
    } else if (p.mode == 1) {
        const int g = find_group(tile_start, p.num_groups, tile);
        const int local = tile - tile_start[g];
        const int m_tiles = (p.group_offsets[g + 1] - p.group_offsets[g]) / BM;
        const int m_blk = local % m_tiles, n_blk = local / m_tiles;
        t.a_row0 = t.d_row0 = p.group_offsets[g] + m_blk * BM;
        t.d_col0 = n_blk * BN;
        // B block g: K-major weights are stacked on rows ([G*N, K]); MN-major weights are stacked on the contraction ([G*K, N])
        t.b_row0 = p.b_mn ? n_blk * BN : g * p.N + n_blk * BN;
        t.a_k0 = 0;
        t.b_k0 = p.b_mn ? g * p.K : 0;
        t.num_k = (p.K + BK - 1) / BK;
        t.m_end = p.group_offsets[g + 1];
        t.n_end = p.N;
        t.d_off = 0;
    } else {
        const int num_m = (p.M + BM - 1) / BM;
        const int per = num_m * num_n;
        const int g = find_group(tile_start, p.num_groups, tile);
        const int local = tile - tile_start[g];
        const int m_blk = local % num_m, n_blk = local / num_m;
        t.a_row0 = t.d_row0 = m_blk * BM;
        t.b_row0 = t.d_col0 = n_blk * BN;
        t.a_k0 = t.b_k0 = p.group_offsets[g];
        t.num_k = (p.group_offsets[g + 1] - p.group_offsets[g]) / BK;
        t.m_end = p.M;
        t.n_end = p.N;
        t.d_off = static_cast<long long>(g) * p.M * p.N;
        (void)per;
    }
    return t;
}

// 32 accumulator columns of one output row, straight from registers: 16-byte stores, optional D += and running abs-max.
__device__ __forceinline__ void store_direct_32(const GemmParams& p, const TileInfo& t, int row, int col0, const uint32_t (&r)[32], float scale,
                                                float& amax) {
    if (row >= t.m_end || col0 >= t.n_end) return;
    if (p.out_fp32) {
        float* drow = reinterpret_cast<float*>(p.D) + t.d_off + static_cast<size_t>(row) * p.ldd + col0;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            if (col0 + g * 4 < t.n_end) {
                float4 v = make_float4(__uint_as_float(r[g * 4]) * scale, __uint_as_float(r[g * 4 + 1]) * scale, __uint_as_float(r[g * 4 + 2]) * scale,
                                       __uint_as_float(r[g * 4 + 3]) * scale);
                float4* dst = reinterpret_cast<float4*>(drow + g * 4);
                if (p.accumulate) {
                    const float4 o = *dst;
                    v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
                }
                amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                *dst = v;
            }
        }
    } else {
        __nv_bfloat16* drow = reinterpret_cast<__nv_bfloat16*>(p.D) + t.d_off + static_cast<size_t>(row) * p.ldd + col0;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            if (col0 + g * 8 < t.n_end) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[g * 8 + i]) * scale;
                uint4* dst = reinterpret_cast<uint4*>(drow + g * 8);
                if (p.accumulate) {
                    const uint4 o = *dst;
                    const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&o);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(ob[i]);
                        v[2 * i] += f.x;
                        v[2 * i + 1] += f.y;
                    }
                }
                uint4 out;
                __nv_bfloat162* pb = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    pb[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                    amax = fmaxf(amax, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
                }
                *dst = out;
            }
        }
    }
}

constexpr int MAX_GROUPS = 256;

// ------------------------------------------------------------------------------------------------ units of work
// A unit is one output tile, or one of `splits` equal pieces of its contraction.  Whole waves of tiles stay whole; only the tiles from
// `split_from` on are cut, so that the last wave (or the only one, for small outputs with a long contraction) fills the chip.  A piece
// leaves its fp32 accumulator in the workspace; the warp that arrives last at its 32 rows adds the pieces in order of the contraction
// (the same order in every run) and stores the result.  Nobody waits for anybody.
struct Unit {
    int tile, kb0, kb1;
    int piece;   // -1: a whole tile
};
// Kernels for whole problems (SPLIT = false) are instantiations of their own: the code of the pieces costs registers and 0.1-0.3 us of a short launch.
template <bool SPLIT> __device__ __forceinline__ int num_units(const GemmParams& p, int num_tiles) {
    return SPLIT ? p.split_from + (num_tiles - p.split_from) * p.splits : num_tiles;
}
template <bool SPLIT> __device__ __forceinline__ Unit get_unit(const GemmParams& p, int num_tiles, int num_k, int unit) {
    if (!SPLIT || unit < p.split_from) return Unit{unit, 0, num_k, -1};
    const int r = unit - p.split_from, n = num_tiles - p.split_from;
    const int s = r / n;
    return Unit{p.split_from + r % n, s * num_k / p.splits, (s + 1) * num_k / p.splits, s};
}
// Workspace of one warp's 32 rows x COLS columns: 16-byte vectors, lanes side by side (whole lines per store), pieces `stride` floats apart.
// `valid` = columns that exist.
template <int COLS> __device__ __forceinline__ void park_piece(uint32_t t_row, float4* ws, int lane, int valid) {
#pragma unroll 1
    for (int c = 0; c < COLS && c < valid; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
            ws[(c / 4 + j) * 32 + lane] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
    }
}
__device__ __forceinline__ void sum_pieces(const float4* ws, size_t stride, int pieces, int lane, int c, uint32_t (&r)[32]) {
    float4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __ldcg(ws + (c / 4 + j) * 32 + lane);
    // the next piece is requested before this one is added
    float4 w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = __ldcg(ws + stride + (c / 4 + j) * 32 + lane);
    for (int s = 1; s < pieces; ++s) {
        float4 x[8];
        const size_t next = (s + 1 < pieces ? s + 1 : s) * stride;
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __ldcg(ws + next + (c / 4 + j) * 32 + lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) { v[j].x += w[j].x; v[j].y += w[j].y; v[j].z += w[j].z; v[j].w += w[j].w; w[j] = x[j]; }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        r[4 * j] = __float_as_uint(v[j].x);
        r[4 * j + 1] = __float_as_uint(v[j].y);
        r[4 * j + 2] = __float_as_uint(v[j].z);
        r[4 * j + 3] = __float_as_uint(v[j].w);
    }
}
// True in the warp that completes these rows: all pieces are in the workspace and visible to it.
__device__ __forceinline__ bool last_piece(int* counter, int pieces, int lane) {
    __threadfence();
    __syncwarp();
    int old = 0;
    if (lane == 0) old = atomicAdd(counter, 1);
    old = __shfl_sync(0xffffffffu, old, 0);
    if (old != pieces - 1) return false;
    __threadfence();
    return true;
}

template <int BN, bool SPLIT>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p) {
    using C = Cfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem_base + C::STAGES * C::STAGE_BYTES;
    // barrier layout (8 B each): full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (C::STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * C::STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * C::STAGES + 2 + a); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int elems_per_row = TILE_K_BYTES / p.elem_bytes;  // K elements per stage (K-major) = BK
    const int BK = elems_per_row;
    __shared__ int tile_start[MAX_GROUPS + 1];
    __shared__ int num_tiles_sh;
    if (p.mode == 0) {
        if (threadIdx.x == 0) num_tiles_sh = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
    } else if (threadIdx.x == 0) {
        // prefix of tiles per group (<= 256 groups: a serial scan by one thread costs well under a microsecond)
        const int num_n = (p.N + BN - 1) / BN;
        int acc = 0;
        for (int g = 0; g < p.num_groups; ++g) {
            tile_start[g] = acc;
            const int rows = p.group_offsets[g + 1] - p.group_offsets[g];
            if (p.mode == 1) acc += (rows / BM) * num_n;
            else acc += rows > 0 ? ((p.M + BM - 1) / BM) * num_n : 0;   // empty groups contribute no tiles
        }
        tile_start[p.num_groups] = acc;
        num_tiles_sh = acc;
    }

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 128);
        }
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 2) {
        tmem_alloc(smem_u32(&tmem_base_slot), C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    const int num_tiles = num_tiles_sh;
    const int units = num_units<SPLIT>(p, num_tiles);      // grouped problems are never split: a unit is a tile

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            const int a_chunks = p.a_mn ? (BM * p.elem_bytes) / TILE_K_BYTES : 1;
            const int b_chunks = p.b_mn ? (BN * p.elem_bytes) / TILE_K_BYTES : 1;
            const int chunk_bytes = BK * TILE_K_BYTES;   // MN-major chunk: BK rows of 128 B
            bool ok = true;
            for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
                const Unit u = get_unit<SPLIT>(p, num_tiles, (p.K + BK - 1) / BK, unit);
                const TileInfo t = get_tile<BN>(p, tile_start, u.tile, BK);
                const int m0 = t.a_row0, n0 = t.b_row0;
                const int kb1 = !SPLIT || u.piece < 0 ? t.num_k : u.kb1;
                for (int kb = u.kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1u, &abort_flag)) { ok = false; break; }
                    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
                    const uint32_t sb = sa + A_STAGE_BYTES;
                    mbar_expect_tx(full_bar(stage), C::STAGE_BYTES);
                    const int ka = t.a_k0 + kb * BK, kbb = t.b_k0 + kb * BK;
                    if (!p.a_mn) {
                        tma_load_2d(sa, &tmA, ka, m0, full_bar(stage));
                    } else {
                        for (int c = 0; c < a_chunks; ++c) tma_load_2d(sa + c * chunk_bytes, &tmA, m0 + c * elems_per_row, ka, full_bar(stage));
                    }
                    if (!p.b_mn) {
                        tma_load_2d(sb, &tmB, kbb, n0, full_bar(stage));
                    } else {
                        for (int c = 0; c < b_chunks; ++c) tma_load_2d(sb + c * chunk_bytes, &tmB, n0 + c * elems_per_row, kbb, full_bar(stage));
                    }
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            uint32_t acc_phase[2] = {0, 0};
            int local_tile = 0;
            const uint32_t idesc = make_idesc(p.a_fmt, p.b_fmt, p.a_mn, p.b_mn, BM, BN);
            const uint32_t lbo = BK * TILE_K_BYTES;                 // MN-major: stride between 128-byte MN chunks
            const uint32_t a_kstep = p.a_mn ? (BK / 4) * TILE_K_BYTES : 32;
            const uint32_t b_kstep = p.b_mn ? (BK / 4) * TILE_K_BYTES : 32;
            bool ok = true;
            for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x, ++local_tile) {
                const int acc = local_tile & 1;
                if (!mbar_wait(tempty_bar(acc), acc_phase[acc] ^ 1u, &abort_flag)) { ok = false; break; }
                acc_phase[acc] ^= 1u;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                const Unit u = get_unit<SPLIT>(p, num_tiles, (p.K + BK - 1) / BK, unit);
                const int num_k = !SPLIT || u.piece < 0 ? get_tile<BN>(p, tile_start, u.tile, BK).num_k : u.kb1 - u.kb0;
                for (int kb = 0; kb < num_k; ++kb) {
                    if (!mbar_wait(full_bar(stage), phase, &abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_base + stage * C::STAGE_BYTES;
                    const uint32_t sb = sa + A_STAGE_BYTES;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint64_t da = make_smem_desc(sa + j * a_kstep, p.a_mn ? lbo : 16, 1024);
                        const uint64_t db = make_smem_desc(sb + j * b_kstep, p.b_mn ? lbo : 16, 1024);
                        const uint32_t accum = (kb > 0 || j > 0) ? 1u : 0u;
                        if (p.elem_bytes == 2) mma_f16(d_tmem, da, db, idesc, accum);
                        else mma_f8(d_tmem, da, db, idesc, accum);
                    }
                    tc_commit(empty_bar(stage));   // frees the smem stage once these MMAs have read it
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
                }
                if (ok) tc_commit(tfull_bar(acc));   // accumulator complete
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..5)
        const int quad = warp & 3;          // TMEM lane quarter this warp may access
        uint32_t acc_phase[2] = {0, 0};
        int local_tile = 0;
        float scale = p.alpha;
        if (p.scale_a) scale *= __ldg(p.scale_a);
        if (p.scale_b) scale *= __ldg(p.scale_b);
        float amax = 0.f;
        bool ok = true;
        for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x, ++local_tile) {
            const Unit u = get_unit<SPLIT>(p, num_tiles, (p.K + BK - 1) / BK, unit);
            const TileInfo t = get_tile<BN>(p, tile_start, u.tile, BK);
            const int acc = local_tile & 1;
            if (!mbar_wait(tfull_bar(acc), acc_phase[acc], &abort_flag)) { ok = false; break; }
            acc_phase[acc] ^= 1u;
            tc_fence_after();
            const int row = t.d_row0 + quad * 32 + lane;
            const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
            if (SPLIT && u.piece >= 0) {
                const int slot = (u.tile - p.split_from) * 4 + quad, slots = (num_tiles - p.split_from) * 4;
                float4* ws = reinterpret_cast<float4*>(p.workspace) + static_cast<size_t>(slot) * (32 * BN / 4);
                const size_t stride = static_cast<size_t>(slots) * (32 * BN / 4);
                const bool rows = t.d_row0 + quad * 32 < t.m_end;        // the same in every piece of the tile
                if (rows) park_piece<BN>(t_row, ws + u.piece * stride, lane, t.n_end - t.d_col0);
                tc_fence_before();
                mbar_arrive(tempty_bar(acc));
                if (rows && last_piece(p.counters + slot, p.splits, lane)) {
#pragma unroll 1
                    for (int c = 0; c < BN && t.d_col0 + c < t.n_end; c += 32) {
                        uint32_t r[32];
                        sum_pieces(ws, stride, p.splits, lane, c, r);
                        store_direct_32(p, t, row, t.d_col0 + c, r, scale, amax);
                    }
                }
                continue;
            }
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                uint32_t r[32];
                tmem_ld_32x32(t_row + c, r);
                tmem_ld_wait();
                store_direct_32(p, t, row, t.d_col0 + c, r, scale, amax);
            }
            tc_fence_before();
            mbar_arrive(tempty_bar(acc));
        }
        if (p.amax_out) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            if (lane == 0 && amax > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.amax_out), __float_as_uint(amax));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && abort_flag && p.error_flag) atomicExch(p.error_flag, 1);
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------ CTA-pair kernel
// 256 x 256 output tile per CLUSTER of two CTAs (tcgen05 cta_group::2).  Each CTA stages its own 128 rows of A and its own 128 of
// the tile's 256 B rows (16 KB + 16 KB per stage instead of 16 + 32 for the single-CTA 128 x 256 tile, so six stages fit and every
// byte of B is read from shared memory by one SM, not two); the leader CTA's MMA thread issues M = 256, N = 256 instructions that
// fill 128 TMEM lanes x 256 columns in both CTAs.  Loads are per-CTA TMA copies (no cluster broadcast) that complete on the
// leader's barrier; the MMA completion is committed to both CTAs' barriers.  The epilogue leaves through shared memory: every
// warp packs its 32 rows x 128 bytes into a swizzled staging tile and one lane issues a TMA store (or a TMA add for fp32
// accumulation), so global writes are whole 128-byte lines and the tensor map clips the edges.  bf16 accumulation (ACC) fetches D the
// same way: a warp's four 32 x 64 tiles of D are requested into its staging tiles before the accumulator is complete, summed there in
// fp32, rounded once and stored (8192 x 17408 += 16 deep on B200 643 -> 203 us, 151936 x 4096 += 4096 deep in FP8 2733 -> 1970 us; read
// and added row by row from registers before).  Only an fp32 abs-max of accumulated values keeps the register
// path.  Dense problems only (mode 0).
constexpr int PAIR_BM = 256, PAIR_BN = 256;
constexpr int PAIR_B_BYTES = 128 * TILE_K_BYTES;                 // this CTA's half of the B tile
constexpr int PAIR_STAGE_BYTES = A_STAGE_BYTES + PAIR_B_BYTES;   // 32 KB
// staging tiles of 32 rows x 128 bytes per epilogue warp: two in turn, or with ACC one per 64-column chunk of D, paid for with one ring
// stage (the ring is no slower with five: it is bound by operand bandwidth, not by latency)
template <bool ACC> struct PairCfg {
    static constexpr int STAGES = ACC ? 5 : 6;
    static constexpr int EPI_BUFS = ACC ? 4 : 2;
    static constexpr int EPI_WARP_BYTES = EPI_BUFS * 4096;
    static constexpr int SMEM_BYTES = STAGES * PAIR_STAGE_BYTES + 4 * EPI_WARP_BYTES + 1024 /*align slack*/ + 384 /*barriers*/;
};

struct PairTile {
    int m0, n0;   // origin of the 256 x 256 tile
};
__device__ __forceinline__ PairTile pair_tile(const GemmParams& p, int tile) {
    const int num_m = (p.M + PAIR_BM - 1) / PAIR_BM, num_n = (p.N + PAIR_BN - 1) / PAIR_BN;
    const int per_group = p.pair_group_m * num_n;
    const int group = tile / per_group;
    const int first_m = group * p.pair_group_m;
    const int gsize = min(num_m - first_m, p.pair_group_m);
    const int r = tile - group * per_group;
    return PairTile{(first_m + r % gsize) * PAIR_BM, (r / gsize) * PAIR_BN};
}

template <bool ACC, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmD,
                 const GemmParams p, const int use_tma_store) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // same offset in both CTAs: the MMA applies one descriptor to both
    constexpr int PAIR_STAGES = PairCfg<ACC>::STAGES;
    const uint32_t epi_base = smem_base + PAIR_STAGES * PAIR_STAGE_BYTES;
    const uint32_t bar_base = epi_base + 4 * PairCfg<ACC>::EPI_WARP_BYTES;
    // barriers (8 B each): full[STAGES] (used in the leader), empty[STAGES], tmem_full[2], tmem_empty[2] (used in the leader), with ACC
    // d_full[4 warps][4 tiles]
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (PAIR_STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * PAIR_STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * PAIR_STAGES + 2 + a); };
    auto d_bar = [&](int w, int b) { return bar_base + 8u * (2 * PAIR_STAGES + 4 + w * 4 + b); };
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int BK = TILE_K_BYTES / p.elem_bytes;
    const int num_tiles = ((p.M + PAIR_BM - 1) / PAIR_BM) * ((p.N + PAIR_BN - 1) / PAIR_BN);
    const int num_k = (p.K + BK - 1) / BK;
    const int units = num_units<SPLIT>(p, num_tiles);
    const int first_unit = blockIdx.x >> 1, unit_step = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < PAIR_STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 8);      // one lane of each epilogue warp of both CTAs
        }
        if (ACC)
            for (int i = 0; i < 16; ++i) mbar_init(d_bar(i >> 2, i & 3), 1);
        fence_barrier_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        if (use_tma_store) tma_prefetch_desc(&tmD);
    }
    if (warp == 2) {
        tmem_alloc_pair(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();     // both CTAs' barriers are initialised before either CTA signals the other
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (one per CTA)
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            const int a_chunks = p.a_mn ? (BM * p.elem_bytes) / TILE_K_BYTES : 1;
            const int b_chunks = p.b_mn ? (128 * p.elem_bytes) / TILE_K_BYTES : 1;
            const int chunk_bytes = BK * TILE_K_BYTES;
            bool ok = true;
            // optional L2 prefetch cursor: runs `pair_prefetch` contraction blocks ahead of the load cursor (across tile boundaries)
            int pf_unit = first_unit, pf_kb = 0, pf_end = 0, pf_m0 = 0, pf_n0 = 0;
            auto pf_origin = [&]() {
                const Unit u = get_unit<SPLIT>(p, num_tiles, num_k, pf_unit);
                const PairTile t = pair_tile(p, u.tile);
                pf_kb = u.kb0;
                pf_end = u.kb1;
                pf_m0 = t.m0 + static_cast<int>(rank) * 128;
                pf_n0 = t.n0 + static_cast<int>(rank) * 128;
            };
            auto pf_step = [&]() {
                if (pf_unit >= units) return;
                const int k0 = pf_kb * BK;
                if (!p.a_mn) tma_prefetch_l2_2d(&tmA, k0, pf_m0);
                else for (int c = 0; c < a_chunks; ++c) tma_prefetch_l2_2d(&tmA, pf_m0 + c * BK, k0);
                if (!p.b_mn) tma_prefetch_l2_2d(&tmB, k0, pf_n0);
                else for (int c = 0; c < b_chunks; ++c) tma_prefetch_l2_2d(&tmB, pf_n0 + c * BK, k0);
                if (++pf_kb == pf_end) {
                    pf_unit += unit_step;
                    if (pf_unit < units) pf_origin();
                }
            };
            if (p.pair_prefetch > 0 && first_unit < units) {
                pf_origin();
                for (int i = 0; i < PAIR_STAGES + p.pair_prefetch; ++i) pf_step();
            }
            for (int unit = first_unit; unit < units && ok; unit += unit_step) {
                const Unit u = get_unit<SPLIT>(p, num_tiles, num_k, unit);
                const PairTile t = pair_tile(p, u.tile);
                const int m0 = t.m0 + static_cast<int>(rank) * 128, n0 = t.n0 + static_cast<int>(rank) * 128;
                for (int kb = u.kb0; kb < u.kb1; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1u, &abort_flag)) { ok = false; break; }
                    if (p.pair_prefetch > 0) pf_step();
                    const uint32_t sa = smem_base + stage * PAIR_STAGE_BYTES;
                    const uint32_t sb = sa + A_STAGE_BYTES;
                    const uint32_t bar = mapa_shared(full_bar(stage), 0);                 // the leader's barrier counts both CTAs' bytes
                    if (leader) mbar_expect_tx(full_bar(stage), 2 * PAIR_STAGE_BYTES);
                    const int k0 = kb * BK;
                    if (!p.a_mn) {
                        tma_load_2d_pair(sa, &tmA, k0, m0, bar);
                    } else {
                        for (int c = 0; c < a_chunks; ++c) tma_load_2d_pair(sa + c * chunk_bytes, &tmA, m0 + c * BK, k0, bar);
                    }
                    if (!p.b_mn) {
                        tma_load_2d_pair(sb, &tmB, k0, n0, bar);
                    } else {
                        for (int c = 0; c < b_chunks; ++c) tma_load_2d_pair(sb + c * chunk_bytes, &tmB, n0 + c * BK, k0, bar);
                    }
                    if (++stage == PAIR_STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader CTA only)
        if (leader && elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            uint32_t acc_phase[2] = {0, 0};
            int local_tile = 0;
            const uint32_t idesc = make_idesc(p.a_fmt, p.b_fmt, p.a_mn, p.b_mn, PAIR_BM, PAIR_BN);
            const uint32_t lbo = BK * TILE_K_BYTES;
            const uint32_t a_kstep = p.a_mn ? (BK / 4) * TILE_K_BYTES : 32;
            const uint32_t b_kstep = p.b_mn ? (BK / 4) * TILE_K_BYTES : 32;
            bool ok = true;
            for (int unit = first_unit; unit < units && ok; unit += unit_step, ++local_tile) {
                const int acc = local_tile & 1;
                if (!mbar_wait_cluster(tempty_bar(acc), acc_phase[acc] ^ 1u, &abort_flag)) { ok = false; break; }
                acc_phase[acc] ^= 1u;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * PAIR_BN;
                const Unit u = get_unit<SPLIT>(p, num_tiles, num_k, unit);
                for (int kb = 0; kb < u.kb1 - u.kb0; ++kb) {
                    if (!mbar_wait_cluster(full_bar(stage), phase, &abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sa = smem_base + stage * PAIR_STAGE_BYTES;
                    const uint32_t sb = sa + A_STAGE_BYTES;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint64_t da = make_smem_desc(sa + j * a_kstep, p.a_mn ? lbo : 16, 1024);
                        const uint64_t db = make_smem_desc(sb + j * b_kstep, p.b_mn ? lbo : 16, 1024);
                        const uint32_t accum = (kb > 0 || j > 0) ? 1u : 0u;
                        if (p.elem_bytes == 2) mma_f16_pair(d_tmem, da, db, idesc, accum);
                        else mma_f8_pair(d_tmem, da, db, idesc, accum);
                    }
                    tc_commit_pair(empty_bar(stage), 3);   // both CTAs' stage is free once these MMAs have read it
                    if (++stage == PAIR_STAGES) { stage = 0; phase ^= 1u; }
                }
                if (ok) tc_commit_pair(tfull_bar(acc), 3);  // both CTAs' halves of the accumulator are complete
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..5 of both CTAs; each CTA drains its own 128 rows)
        const int quad = warp & 3;
        uint32_t acc_phase[2] = {0, 0};
        int local_tile = 0;
        float scale = p.alpha;
        if (p.scale_a) scale *= __ldg(p.scale_a);
        if (p.scale_b) scale *= __ldg(p.scale_b);
        float amax = 0.f;
        bool ok = true;
        const uint32_t tempty_leader[2] = {mapa_shared(tempty_bar(0), 0), mapa_shared(tempty_bar(1), 0)};
        const uint32_t stage_smem = epi_base + quad * PairCfg<ACC>::EPI_WARP_BYTES;
        uint8_t* stage_ptr = smem_raw + (stage_smem - smem_u32(smem_raw));
        int buf = 0, stores_in_flight = 0;
        uint32_t d_phase = 0;      // ACC: parity of each staging tile's next arrival
        // ACC: request this warp's tiles of D (the stores that last used the staging tiles have finished reading them)
        auto fetch_d = [&](const PairTile& pt, int row_w) {
            if (!ACC || row_w >= p.M) return;
            if (lane == 0) {
                tma_store_wait_read<0>();
                for (int i = 0; i < PairCfg<ACC>::EPI_BUFS && pt.n0 + i * 64 < p.N; ++i) {
                    mbar_expect_tx(d_bar(quad, i), 4096);
                    tma_load_2d(stage_smem + i * 4096, &tmD, pt.n0 + i * 64, row_w, d_bar(quad, i));
                }
            }
            __syncwarp();
        };
        // the finished 32 rows x 256 columns of this warp leave; `load` supplies 32 columns of raw accumulators
        auto emit = [&](const PairTile& pt, int row_w, auto&& load) {
            if (use_tma_store) {
                const int cols_per_store = p.out_fp32 ? 32 : 64;
                if (row_w < p.M) {
#pragma unroll 1
                    for (int c = 0; c < PAIR_BN && pt.n0 + c < p.N; c += cols_per_store) {
                        uint32_t r0[32], r1[32];
                        load(c, r0);
                        if (!p.out_fp32) load(c + 32, r1);
                        if (ACC) {
                            buf = c / 64;
                            if (!mbar_wait(d_bar(quad, buf), (d_phase >> buf) & 1u, &abort_flag)) { ok = false; break; }
                            d_phase ^= 1u << buf;
                        } else if (stores_in_flight >= 2) {      // the store that last read this staging tile has finished reading it
                            if (lane == 0) tma_store_wait_read<1>();
                            __syncwarp();
                        }
                        tmem_ld_wait();
                        uint8_t* srow = stage_ptr + buf * 4096 + lane * 128;
                        if (!ACC && p.out_fp32) {
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                const float4 v = make_float4(__uint_as_float(r0[u * 4]) * scale, __uint_as_float(r0[u * 4 + 1]) * scale,
                                                             __uint_as_float(r0[u * 4 + 2]) * scale, __uint_as_float(r0[u * 4 + 3]) * scale);
                                amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                                *reinterpret_cast<float4*>(srow + ((u ^ (lane & 7)) << 4)) = v;
                            }
                        } else {
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                uint4* cell = reinterpret_cast<uint4*>(srow + ((u ^ (lane & 7)) << 4));
                                uint4 o = ACC ? *cell : make_uint4(0, 0, 0, 0);
                                __nv_bfloat162* pb = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const int e = (u & 3) * 8 + 2 * i;
                                    float a = __uint_as_float(u < 4 ? r0[e] : r1[e]) * scale, b = __uint_as_float(u < 4 ? r0[e + 1] : r1[e + 1]) * scale;
                                    if (ACC) {
                                        const float2 d = __bfloat1622float2(pb[i]);
                                        a += d.x;
                                        b += d.y;
                                    }
                                    amax = fmaxf(amax, fmaxf(fabsf(a), fabsf(b)));
                                    pb[i] = __floats2bfloat162_rn(a, b);
                                }
                                *cell = o;
                            }
                        }
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            if (!ACC && p.accumulate) tma_reduce_add_2d(&tmD, stage_smem + buf * 4096, pt.n0 + c, row_w);
                            else tma_store_2d(&tmD, stage_smem + buf * 4096, pt.n0 + c, row_w);
                            tma_store_commit();
                        }
                        ++stores_in_flight;
                        if (!ACC) buf ^= 1;
                    }
                }
            } else {
                TileInfo t;
                t.m_end = p.M;
                t.n_end = p.N;
                t.d_off = 0;
                const int row = row_w + lane;
#pragma unroll 1
                for (int c = 0; c < PAIR_BN && pt.n0 + c < p.N; c += 32) {
                    uint32_t r[32];
                    load(c, r);
                    tmem_ld_wait();
                    store_direct_32(p, t, row, pt.n0 + c, r, scale, amax);
                }
            }
        };
        for (int unit = first_unit; unit < units && ok; unit += unit_step, ++local_tile) {
            const Unit u = get_unit<SPLIT>(p, num_tiles, num_k, unit);
            const PairTile pt = pair_tile(p, u.tile);
            const int acc = local_tile & 1;
            const int row_w = pt.m0 + static_cast<int>(rank) * 128 + quad * 32;   // first row of this warp
            const uint32_t t_row = tmem_base + acc * PAIR_BN + (static_cast<uint32_t>(quad * 32) << 16);
            if (!SPLIT || u.piece < 0) fetch_d(pt, row_w);
            if (!mbar_wait(tfull_bar(acc), acc_phase[acc], &abort_flag)) { ok = false; break; }
            acc_phase[acc] ^= 1u;
            tc_fence_after();
            if (!SPLIT || u.piece < 0) {
                emit(pt, row_w, [&](int c, uint32_t(&r)[32]) { tmem_ld_32x32(t_row + c, r); });
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(tempty_leader[acc]);
            } else {
                const int slot = ((u.tile - p.split_from) * 2 + static_cast<int>(rank)) * 4 + quad, slots = (num_tiles - p.split_from) * 8;
                float4* ws = reinterpret_cast<float4*>(p.workspace) + static_cast<size_t>(slot) * (32 * PAIR_BN / 4);
                const size_t stride = static_cast<size_t>(slots) * (32 * PAIR_BN / 4);
                const bool rows = row_w < p.M;
                if (rows) park_piece<PAIR_BN>(t_row, ws + u.piece * stride, lane, (p.N - pt.n0 + 63) & ~63);   // the reader takes 64 columns at a time
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(tempty_leader[acc]);
                if (rows && last_piece(p.counters + slot, p.splits, lane)) {
                    fetch_d(pt, row_w);
                    emit(pt, row_w, [&](int c, uint32_t(&r)[32]) { sum_pieces(ws, stride, p.splits, lane, c, r); });
                }
            }
        }
        if (use_tma_store && lane == 0) tma_store_wait_all();
        if (p.amax_out) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            if (lane == 0 && amax > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.amax_out), __float_as_uint(amax));
        }
    }

    tc_fence_before();
    cluster_sync_all();   // neither CTA leaves (or frees TMEM) while the other may still signal its barriers or read its shared memory
    if (threadIdx.x == 0 && abort_flag && p.error_flag) atomicExch(p.error_flag, 1);
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------------------------ host side
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn get_encode_fn() {
    static EncodeFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess || !ptr)
            return nullptr;
        fn = reinterpret_cast<EncodeFn>(ptr);
    }
    return fn;
}

const char* make_tensor_map_2d(CUtensorMap* map, const void* base, int elem_bytes, uint64_t inner, uint64_t outer, uint64_t row_stride_bytes,
                               uint32_t box_inner, uint32_t box_outer) {
    EncodeFn enc = get_encode_fn();
    if (!enc) return "cuTensorMapEncodeTiled unavailable";
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return "TMA base address must be 16-byte aligned";
    if (row_stride_bytes % 16 != 0) return "TMA row stride must be a multiple of 16 bytes";
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_stride_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : (elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8);
    CUresult r = enc(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? nullptr : "cuTensorMapEncodeTiled failed";
}

template <int BN, bool SPLIT> static const char* launch(const GemmOperand& A, const GemmOperand& B, const GemmParams& p, int num_sms, cudaStream_t stream) {
    using C = Cfg<BN>;
    const int BK = TILE_K_BYTES / p.elem_bytes;
    CUtensorMap tmA, tmB;
    const char* e;
    // K-major: inner = K, outer = rows, box {BK, rows_per_tile}.  MN-major: inner = rows, outer = K, box {128 B of rows, BK}.
    // Extents of the stored 2-D operands.  Grouped modes: a_rows / b_rows are the totals over all groups.
    const uint64_t a_rows = p.mode == 0 ? (p.a_mn ? p.K : p.M) : p.a_total_rows;
    const uint64_t b_rows = p.mode == 0 ? (p.b_mn ? p.K : p.N) : p.b_total_rows;
    if (!p.a_mn) e = make_tensor_map_2d(&tmA, A.ptr, p.elem_bytes, p.K, a_rows, A.row_stride_bytes, BK, BM);
    else e = make_tensor_map_2d(&tmA, A.ptr, p.elem_bytes, p.M, a_rows, A.row_stride_bytes, BK, BK);
    if (e) return e;
    if (!p.b_mn) e = make_tensor_map_2d(&tmB, B.ptr, p.elem_bytes, p.K, b_rows, B.row_stride_bytes, BK, BN);
    else e = make_tensor_map_2d(&tmB, B.ptr, p.elem_bytes, p.N, b_rows, B.row_stride_bytes, BK, BK);
    if (e) return e;
    static std::atomic<uint64_t> limit{0};
    if (!raise_smem_limit(reinterpret_cast<const void*>(gemm_tcgen05_kernel<BN, SPLIT>), C::SMEM_BYTES, limit)) return "raising the shared-memory limit failed (GEMM)";
    int units = p.mode == 0 ? ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) : num_sms;  // grouped: tile count lives on the device
    if (SPLIT) units = p.split_from + (units - p.split_from) * p.splits;
    const int grid = units < num_sms ? units : num_sms;
    gemm_tcgen05_kernel<BN, SPLIT><<<grid, GEMM_THREADS, C::SMEM_BYTES, stream>>>(tmA, tmB, p);
    return cudaGetLastError() == cudaSuccess ? nullptr : "gemm kernel launch failed";
}

static const char* launch_pair(const GemmOperand& A, const GemmOperand& B, GemmParams p, int num_sms, cudaStream_t stream) {
    const int BK = TILE_K_BYTES / p.elem_bytes;
    // L2 prefetch is off unless asked for: measured on B200 it costs 3-5 % (the kernel is bound by operand delivery bandwidth, not by
    // DRAM latency: four, five and six ring stages run at the same speed, half the operand bytes run 15-18 % faster)
    if (p.pair_group_m <= 0) {
        // The group's A panel (group_m x 256 rows x K) is re-read from L2 by every tile of the sweep over N while B streams through
        // once per group: make the panel as tall as a quarter of the L2 allows, so B is fetched from DRAM as few times as possible.
        const long long panel_row_bytes = static_cast<long long>(PAIR_BM) * p.K * p.elem_bytes;
        long long g = (32ll << 20) / (panel_row_bytes > 0 ? panel_row_bytes : 1);
        g = g < 4 ? 4 : (g > 32 ? 32 : g);
        p.pair_group_m = static_cast<int>(g);
    }
    CUtensorMap tmA, tmB, tmD;
    const char* e;
    if (!p.a_mn) e = make_tensor_map_2d(&tmA, A.ptr, p.elem_bytes, p.K, p.M, A.row_stride_bytes, BK, BM);
    else e = make_tensor_map_2d(&tmA, A.ptr, p.elem_bytes, p.M, p.K, A.row_stride_bytes, BK, BK);
    if (e) return e;
    if (!p.b_mn) e = make_tensor_map_2d(&tmB, B.ptr, p.elem_bytes, p.K, p.N, B.row_stride_bytes, BK, 128);
    else e = make_tensor_map_2d(&tmB, B.ptr, p.elem_bytes, p.N, p.K, B.row_stride_bytes, BK, BK);
    if (e) return e;
    // The shared-memory epilogue serves everything but an fp32 abs-max that must include the accumulated values (the TMA add does not
    // return them).
    const int d_bytes = p.out_fp32 ? 4 : 2;
    int use_tma_store = !(p.accumulate && p.out_fp32 && p.amax_out);
    if (use_tma_store) {
        e = make_tensor_map_2d(&tmD, p.D, d_bytes, p.N, p.M, static_cast<uint64_t>(p.ldd) * d_bytes, 128 / d_bytes, 32);
        if (e) use_tma_store = 0;
    }
    if (!use_tma_store) tmD = tmA;
    const bool acc = use_tma_store && p.accumulate && !p.out_fp32;
    const int num_tiles = ((p.M + PAIR_BM - 1) / PAIR_BM) * ((p.N + PAIR_BN - 1) / PAIR_BN);
    const int units = p.splits > 1 ? p.split_from + (num_tiles - p.split_from) * p.splits : num_tiles;
    const int clusters = units < num_sms / 2 ? units : num_sms / 2;
    auto run = [&](auto* kernel, int smem, std::atomic<uint64_t>& limit) -> const char* {
        if (!raise_smem_limit(reinterpret_cast<const void*>(kernel), smem, limit)) return "raising the shared-memory limit failed (pair GEMM)";
        kernel<<<2 * clusters, GEMM_THREADS, smem, stream>>>(tmA, tmB, tmD, p, use_tma_store);
        return cudaGetLastError() == cudaSuccess ? nullptr : "pair gemm kernel launch failed";
    };
    static std::atomic<uint64_t> limit[4];
    if (acc) return p.splits > 1 ? run(gemm_pair_kernel<true, true>, PairCfg<true>::SMEM_BYTES, limit[3]) : run(gemm_pair_kernel<true, false>, PairCfg<true>::SMEM_BYTES, limit[2]);
    return p.splits > 1 ? run(gemm_pair_kernel<false, true>, PairCfg<false>::SMEM_BYTES, limit[1]) : run(gemm_pair_kernel<false, false>, PairCfg<false>::SMEM_BYTES, limit[0]);
}

// ------------------------------------------------------------------------------------------------ choice of kernel and split
// Which kernel runs a dense problem, and into how many pieces the contraction of its last wave of tiles is cut, by estimated time.  A wave
// costs its contraction (128-byte blocks) or its epilogue, whichever is longer, and the last one both; a piece costs its trip through the
// workspace, the warp that adds them every piece; nothing is faster than its operands and output from memory.  The constants are a
// least-squares fit to 68 000 timings on B200 (11 500 problems, every kernel and split that they allow);
// blocks cost the same in bf16 and FP8.  The estimate is good to 10-20 %, so the count of pair tiles decides (a wave of them: pairs) unless
// the other kernel is estimated 8 % faster, and a split has to promise 5 %.
//   pair   : full rate, but 74 tiles of 256 x 256 to a wave.  [1024, 3072] = 16384 deep (48 tiles) in three pieces 164 -> 93 us, [6144, 1024] (96
//            tiles, the last 22 in three pieces) 204 -> 157 us, [4096, 4096] = 151936 deep in bf16 (256 tiles, 34 in two) 4530 -> 3939 us.
//   single : four times as many tiles, for small outputs; also the narrow ones (N <= 128), where a pair would multiply padding:
//            [4096, 16] = 17408 deep 91 -> 45 us in four pieces.  Its fp32 accumulation goes row by row from registers: [64, 151936] += 64
//            deep takes 94 us, pairs 34 us.
namespace {
struct Shape {
    int tiles, slots;                               // output tiles, tiles that run at once
    float fixed_us, block_us, epilogue_us;          // once; per contraction block of a wave; per wave
    float piece_us, reader_us, split_us;            // per wave of pieces; per piece for the warp that adds them; once per split problem
    int tile_floats;
};
struct Split {
    float us;
    int from, pieces;
};
constexpr int MAX_PIECES = 8;
constexpr int MIN_PIECE_BLOCKS = 4;
constexpr float SPLIT_GAIN = 0.95f, KERNEL_GAIN = 0.92f;
constexpr float STREAM_BYTES_PER_US = 4.0e6f;

Split best_split(const Shape& h, int num_k, float stream_us) {
    const int full = h.tiles / h.slots, rest = h.tiles % h.slots;
    const float k_us = num_k * h.block_us, wave_us = std::max(k_us, h.epilogue_us);
    const int waves = full + (rest ? 1 : 0);
    Split best{std::max(stream_us, h.fixed_us + (waves - 1) * wave_us + k_us + h.epilogue_us), h.tiles, 1};
    for (int s = 2; rest && s <= MAX_PIECES && num_k / s >= MIN_PIECE_BLOCKS && rest * s <= 3 * h.slots; ++s) {
        const int piece_waves = (rest * s + h.slots - 1) / h.slots;
        const float us = h.fixed_us + full * wave_us + piece_waves * (((num_k + s - 1) / s) * h.block_us + h.piece_us) + s * h.reader_us + h.split_us + h.epilogue_us;
        if (std::max(stream_us, us) < best.us * SPLIT_GAIN) best = Split{std::max(stream_us, us), h.tiles - rest, s};
    }
    return best;
}
}  // namespace

GemmPlan gemm_plan_sm100(const GemmParams& p, int num_sms) {
    GemmPlan plan{0, 1, 0, 0, 0};
    if (p.mode != 0 || p.M <= 0 || p.N <= 0 || p.K <= 0) return plan;
    const int num_k = static_cast<int>((static_cast<long long>(p.K) * p.elem_bytes + TILE_K_BYTES - 1) / TILE_K_BYTES);
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    const int out = (p.out_fp32 ? 2 : 0) + (p.accumulate ? 1 : 0), mn = (p.a_mn ? 1 : 0) + (p.b_mn ? 1 : 0);   // bf16, bf16 +=, fp32, fp32 +=
    constexpr float pair_out[4] = {4.0f, 5.4f, 5.2f, 5.8f}, single_out[4] = {3.7f, 7.7f, 5.3f, 13.0f}, single_block[3] = {0.26f, 0.27f, 0.32f};
    const Shape pair{up(p.M, PAIR_BM) * up(p.N, PAIR_BN), num_sms / 2, 1.6f, 0.41f, pair_out[out], 7.2f, 1.2f, 1.5f, PAIR_BM * PAIR_BN};
    // operands of fewer than 16 rows, or with stored rows below 32 bytes, arrive slowly: 2-5 us more per piece
    const bool short_rows = (p.a_mn && p.M * p.elem_bytes < 32) || (p.b_mn && p.N * p.elem_bytes < 32);
    const float single_piece = p.M < 16 || short_rows ? 11.3f : 6.3f;
    const Shape single{up(p.M, BM) * up(p.N, 128), num_sms, 0.4f, single_block[mn], single_out[out], single_piece, 0.4f, 0.4f, BM * 128};
    const float stream_us = (static_cast<float>(p.elem_bytes) * p.K * (static_cast<float>(p.M) + p.N) +
                             (p.out_fp32 ? 4.f : 2.f) * (p.accumulate ? 2.f : 1.f) * p.M * p.N) / STREAM_BYTES_PER_US;
    const Split sp = best_split(pair, num_k, stream_us), ss = best_split(single, num_k, stream_us);
    // stored rows below 32 bytes slow single CTAs more than pairs, beyond the estimate: 16 x 151936 in FP8, 512 deep, 98 and 78 us
    int use_pair = p.N > 128 && (pair.tiles >= pair.slots ? short_rows || !(ss.us < KERNEL_GAIN * sp.us) : sp.us < KERNEL_GAIN * ss.us);
    if (p.tile_n != 0) use_pair = p.tile_n == 512;
    plan.pair = use_pair;
    if (p.tile_n == 256 || p.tile_n == 128) return plan;        // forced single-CTA tiles: never split
    const Split& c = use_pair ? sp : ss;
    if (c.pieces > 1) {
        const Shape& h = use_pair ? pair : single;
        const size_t cut = static_cast<size_t>(h.tiles - c.from);
        plan.splits = c.pieces;
        plan.split_from = c.from;
        plan.workspace_floats = cut * c.pieces * h.tile_floats;
        plan.num_counters = cut * (use_pair ? 8 : 4);
    }
    return plan;
}

const char* gemm_sm100(const GemmOperand& A, const GemmOperand& B, GemmParams p, int num_sms, cudaStream_t stream) {
    if (p.M <= 0 || p.N <= 0 || p.K <= 0) return nullptr;
    if (p.mode != 0 && (p.num_groups <= 0 || p.num_groups > MAX_GROUPS || !p.group_offsets)) return "gemm_sm100: grouped mode needs 1..256 groups and offsets";
    if (p.N % 8 != 0 || p.ldd % 8 != 0) return "gemm_sm100: N and ldd must be multiples of 8";
    if ((reinterpret_cast<uintptr_t>(p.D) & 15) != 0) return "gemm_sm100: D must be 16-byte aligned";
    const GemmPlan plan = gemm_plan_sm100(p, num_sms);
    if (p.workspace && p.counters) {        // a caller without them gets the same kernel, unsplit
        p.splits = plan.splits;
        p.split_from = plan.split_from;
        if (plan.splits > 1 && cudaMemsetAsync(p.counters, 0, plan.num_counters * sizeof(int), stream) != cudaSuccess) return "gemm_sm100: clearing the counters failed";
    } else {
        p.splits = 1;
    }
    if (plan.pair) return launch_pair(A, B, p, num_sms, stream);
    // 128-wide N tiles when the wide tile would leave SMs idle or N is small
    const long tiles256 = static_cast<long>((p.M + BM - 1) / BM) * ((p.N + 255) / 256);
    const bool narrow = p.mode == 0 ? p.tile_n != 256 : p.N <= 128 || (p.tile_n == 128) || (p.tile_n == 0 && tiles256 < num_sms);
    if (p.splits > 1) return launch<128, true>(A, B, p, num_sms, stream);      // only the narrow tiles are ever cut
    return narrow ? launch<128, false>(A, B, p, num_sms, stream) : launch<256, false>(A, B, p, num_sms, stream);
}

}  // namespace sg
