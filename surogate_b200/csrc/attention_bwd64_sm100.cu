// Flash-attention backward (causal, GQA, head_dim 128; nothing but O and the log-sum-exp is kept from forward, scores are recomputed):
//
// One kernel template serves both passes.  A CTA keeps a RESIDENT pair of 128-row tiles and streams 64-row tile pairs through
// a 4-stage TMA ring; the gradient accumulators stay in TMEM for the whole CTA.
//   dK/dV pass: resident (K, V) of one 128-key tile of one KV head, streamed (Q, dO) tiles of the G query heads that share it:
//               X = S^T, Y = dP^T, P^T = exp2(S^T - lse), dS^T = P^T o (dP^T - delta) scale; dV += P^T dO, dK += dS^T Q.
//   dQ pass   : resident (Q, dO) of one 128-query tile, streamed (K, V) tiles: X = S, Y = dP, dS = P o (dP - delta) scale; dQ += dS K.
// dS is scaled before it is rounded to bf16, at no cost: delta comes times -scale, so that the difference and the scale are one fused
// multiply-add.  Scaling the finished dK / dQ instead had an error against fp64 that was 0.2-0.8 % larger over four shapes.
//
// Two groups of four softmax warps take alternate items.  Each group has its own pair of score accumulators (X, Y) in TMEM, reads them,
// and writes P and dS as bf16 over them, from where the accumulating MMAs take their A operand: no copy in shared memory, no proxy
// fence, and the room this leaves holds the fourth ring stage.  The MMA warp issues, per item, the accumulation of item i and then the
// scores of item i + 2 into the same TMEM columns.  Only MMAs of the same accumulator and shape are ordered among themselves, so the scores
// wait for a commit of the MMA that reads P (or dS) there: X(i + 2) for dV's, while dK's runs, and Y(i + 2) for dK's (dQ's), while X(i + 2)
// runs, so that the tensor pipe has work during both waits.  While one group computes, the other's MMAs run.  Bound by the tensor pipe: a score MMA with 64 columns re-reads its resident operand
// from shared memory at the full 128 bytes per cycle, which makes an item 1280 (dK/dV) or 1024 (dQ) cycles; measured 1540 and 1190, where
// one set of eight warps that took one item at a time and paid each wait, TMEM read and fence in full needed 2155 for dK/dV.
// Both passes and the row statistics on B200, L2 flushed: 2 x 4096 x 32/8 heads 1312 -> 980 us, 1 x 8192 x 40/8 2906 -> 2201 us, 8 x 2048 x
// 16/8 702 -> 562 us.
//
// The row statistics are laid out [B, Hq, T] beforehand (fa_delta_kernel), so that the 64 of a query tile arrive with the tile.
// The GQA reduction of dK / dV happens in the TMEM accumulators (no atomics).  Every mbarrier wait is bounded.
// Optional per-row lower bound `lo[b, t]` (HAS_LO; packed documents and sliding windows, see attention_fwd64_sm100.cu): the dQ pass
// starts at key tile lo[first query] / 64; the dK/dV pass stops at `kv_qend[b, key tile]`, the first 64-row query tile in which no
// query can see the key tile any more (lo is non-decreasing, so that is one number per key tile).
#include <cuda_bf16.h>
#include <math_constants.h>

#include "attention_sm100.h"
#include "gemm_sm100.h"
#include "launch_limits.h"
#include "sm100_ptx.cuh"

namespace sg {
namespace fb64 {

constexpr int D = 128;
constexpr int T128 = 128 * D * 2;     // 32 KB tile of 128 rows: two halves of 16 KB
constexpr int H128 = 16384;
constexpr int T64 = 64 * D * 2;       // 16 KB tile of 64 rows: two halves of 8 KB
constexpr int H64 = 8192;
constexpr int THREADS = 320;      // TMA warp, MMA warp, two groups of 4 softmax warps (one per TMEM lane quadrant)
constexpr float LOG2E = 1.4426950408889634f;

struct Params {
    __nv_bfloat16* d_qkv;
    const float* neg_lse2;   // [B, Hq, T]: -lse * log2(e)
    const float* neg_delta;  // [B, Hq, T]: -delta * scale
    int T, Hq, Hkv;
    float scale, scale_log2;
    int* error_flag;
    long long* prof;   // optional [16]: per-phase cycle counters of one softmax thread of each pass (development aid)
    const int* lo;       // optional [B, T]: first key each query may attend
    const int* kv_qend;  // with lo: [B, T / 128] exclusive end, in 64-row query tiles, of the queries that attend each 128-key tile
};

#define FB_PROF(k)                                   \
    do {                                             \
        if (do_prof) {                               \
            const long long now_ = clock64();        \
            acc_[k] += now_ - t_;                    \
            t_ = now_;                               \
        }                                            \
    } while (0)

// columns [64*half, 64*half+64) of a finished 128x128 fp32 accumulator -> bf16 row in global memory
__device__ __forceinline__ void store_acc128(uint32_t t_acc, uint32_t lane_sel, __nv_bfloat16* dst_row, int half) {
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
        const int c = half * 2 + cc;
        uint32_t raw[32];
        tmem_ld_32x32(t_acc + lane_sel + c * 32, raw);
        tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            uint4 o;
            __nv_bfloat162* po = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i) po[i] = __floats2bfloat162_rn(__uint_as_float(raw[u * 8 + 2 * i]), __uint_as_float(raw[u * 8 + 2 * i + 1]));
            *reinterpret_cast<uint4*>(dst_row + c * 32 + u * 8) = o;
        }
    }
}
// D[128, 64] = A[128 rows, d] . B[64 rows, d]^T  (contraction d = 128: 2 halves x 4 steps)
__device__ __forceinline__ void mma_128x64_kk(uint32_t d_tmem, uint32_t a128, uint32_t b64, uint32_t idesc) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
            mma_f16(d_tmem, make_smem_desc(a128 + c * H128 + ks * 32, 16, 1024), make_smem_desc(b64 + c * H64 + ks * 32, 16, 1024), idesc,
                    (c > 0 || ks > 0) ? 1u : 0u);
}
// D[128, 128] (+)= A[128 lanes x 64 contraction] (bf16 in TMEM, two to a column) . B stored [64 contraction rows][128 cols] (two 8 KB halves)
__device__ __forceinline__ void mma_acc_k64(uint32_t d_tmem, uint32_t a_tmem, uint32_t b64, uint32_t idesc, bool acc) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
        mma_f16_ts(d_tmem, a_tmem + ks * 8, make_smem_desc(b64 + ks * 2048, H64, 1024), idesc, (acc || ks > 0) ? 1u : 0u);
}

// ------------------------------------------------------------------------------------------------ the kernel
// R1 | R2 | ring (S1, S2) x 4 | barriers | row statistics of the ring's query tiles (dK/dV pass): 64 x -lse2, -delta, lo
constexpr int RING = 4;
constexpr int OFF_R2 = T128, OFF_RING = 2 * T128, STAGE = 2 * T64, OFF_BAR = OFF_RING + RING * STAGE, OFF_VEC = OFF_BAR + 256;
constexpr int VEC = 3 * 64 * 4;
constexpr int SMEM = OFF_VEC + RING * VEC;
// barriers: 0 res_full | 1-4 ring_full | 5-8 ring_empty | 9,10 xy_full | 11,12 pds_full | 13 x_free | 14 y_free | 15 done
constexpr int B_RES = 0, B_RFULL = 1, B_REMPTY = B_RFULL + RING, B_XY = B_REMPTY + RING, B_PDS = B_XY + 2, B_XFREE = B_PDS + 2, B_YFREE = B_XFREE + 1,
              B_DONE = B_YFREE + 1;

template <bool IS_DQ, bool HAS_LO>
__global__ void __launch_bounds__(THREADS, 1) fa_bwd64_kernel(const __grid_constant__ CUtensorMap tm_qkv128, const __grid_constant__ CUtensorMap tm_qkv64,
                                                              const __grid_constant__ CUtensorMap tm_do128, const __grid_constant__ CUtensorMap tm_do64,
                                                              const Params p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t s0 = smem_u32(smem);
    const uint32_t s_r1 = s0, s_r2 = s0 + OFF_R2, s_ring = s0 + OFF_RING, bars = s0 + OFF_BAR, s_vec = s0 + OFF_VEC;
    auto bar = [&](int i) { return bars + 8u * i; };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_BAR + 128);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_BAR + 136);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.z, row0 = b * p.T;
    const int G = p.Hq / p.Hkv;
    // dK/dV: tile = key tile kb (light-to-heavy order is reversed: early key tiles see the most query tiles), head = KV head
    // dQ   : tile = query tile (late tiles first), head = query head
    const int tile = IS_DQ ? (gridDim.x - 1 - blockIdx.x) : blockIdx.x;
    const int head = blockIdx.y;
    const int hk = IS_DQ ? head / G : head;
    // streamed 64-row tiles [first_ct, first_ct + per_head): keys from the lower bound of the tile's first query up to the diagonal
    // (dQ), queries from the diagonal to the last one that can still see this key tile (dK/dV)
    const int first_ct = IS_DQ ? (HAS_LO ? __ldg(p.lo + row0 + tile * 128) / 64 : 0) : 2 * tile;
    const int last_ct = IS_DQ ? 2 * (tile + 1) : (HAS_LO ? __ldg(p.kv_qend + b * (p.T / 128) + tile) : p.T / 64);
    const int per_head = last_ct - first_ct;
    const int n_items = IS_DQ ? per_head : G * per_head;
    const int kcol = (p.Hq + hk) * D, vcol = (p.Hq + p.Hkv + hk) * D;

    if (threadIdx.x == 0) {
        *abort_flag = (s0 & 1023u) ? 1 : 0;
        for (int i = 0; i <= B_DONE; ++i) mbar_init(bar(i), i == B_PDS || i == B_PDS + 1 ? 128 : 1);
        fence_barrier_init();
    }
    if (warp == 2) { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t t_x[2] = {tmem, tmem + 64}, t_y[2] = {tmem + 128, tmem + 192}, t_a1 = tmem + 256, t_a2 = tmem + 384;
    const bool bad = *abort_flag != 0;

    if (warp == 0 && !bad) {
        if (elect_one()) {
            mbar_expect_tx(bar(B_RES), 2 * T128);
            const int rr = row0 + tile * 128;
            if (IS_DQ) {
                tma_load_2d(s_r1, &tm_qkv128, head * D, rr, bar(B_RES));
                tma_load_2d(s_r1 + H128, &tm_qkv128, head * D + 64, rr, bar(B_RES));
                tma_load_2d(s_r2, &tm_do128, head * D, rr, bar(B_RES));
                tma_load_2d(s_r2 + H128, &tm_do128, head * D + 64, rr, bar(B_RES));
            } else {
                tma_load_2d(s_r1, &tm_qkv128, kcol, rr, bar(B_RES));
                tma_load_2d(s_r1 + H128, &tm_qkv128, kcol + 64, rr, bar(B_RES));
                tma_load_2d(s_r2, &tm_qkv128, vcol, rr, bar(B_RES));
                tma_load_2d(s_r2 + H128, &tm_qkv128, vcol + 64, rr, bar(B_RES));
            }
            for (int i = 0; i < n_items; ++i) {
                const int st = i % RING;
                if (!mbar_wait(bar(B_REMPTY + st), ((i / RING) & 1) ^ 1u, abort_flag)) break;
                mbar_expect_tx(bar(B_RFULL + st), STAGE + (IS_DQ ? 0 : (HAS_LO ? VEC : 512)));
                const uint32_t d1 = s_ring + st * STAGE, d2 = d1 + T64;
                if (IS_DQ) {
                    const int kr = row0 + (first_ct + i) * 64;
                    tma_load_2d(d1, &tm_qkv64, kcol, kr, bar(B_RFULL + st));
                    tma_load_2d(d1 + H64, &tm_qkv64, kcol + 64, kr, bar(B_RFULL + st));
                    tma_load_2d(d2, &tm_qkv64, vcol, kr, bar(B_RFULL + st));
                    tma_load_2d(d2 + H64, &tm_qkv64, vcol + 64, kr, bar(B_RFULL + st));
                } else {
                    const int h = hk * G + i / per_head, q0 = (first_ct + i % per_head) * 64, qr = row0 + q0;
                    const size_t stat = (static_cast<size_t>(b) * p.Hq + h) * p.T + q0;
                    const uint32_t dv = s_vec + st * VEC;
                    bulk_load(dv, p.neg_lse2 + stat, 256, bar(B_RFULL + st));
                    bulk_load(dv + 256, p.neg_delta + stat, 256, bar(B_RFULL + st));
                    if (HAS_LO) bulk_load(dv + 512, p.lo + qr, 256, bar(B_RFULL + st));
                    tma_load_2d(d1, &tm_qkv64, h * D, qr, bar(B_RFULL + st));
                    tma_load_2d(d1 + H64, &tm_qkv64, h * D + 64, qr, bar(B_RFULL + st));
                    tma_load_2d(d2, &tm_do64, h * D, qr, bar(B_RFULL + st));
                    tma_load_2d(d2 + H64, &tm_do64, h * D + 64, qr, bar(B_RFULL + st));
                }
            }
        }
    } else if (warp == 1 && !bad) {
        if (elect_one()) {
            const uint32_t idesc_s = make_idesc(1, 1, 0, 0, 128, 64), idesc_acc = make_idesc(1, 1, 0, 1, 128, 128);
            auto issue_xy = [&](int i) {
                if (!mbar_wait(bar(B_RFULL + i % RING), (i / RING) & 1, abort_flag)) return false;
                tc_fence_after();
                const uint32_t c1 = s_ring + (i % RING) * STAGE, c2 = c1 + T64;
                // item i - 2 left P and dS in these columns; in the dQ pass X holds no operand, only scores that have been read
                if (!IS_DQ && i >= 2) {
                    if (!mbar_wait(bar(B_XFREE), i & 1, abort_flag)) return false;
                    tc_fence_after();
                }
                mma_128x64_kk(t_x[i & 1], s_r1, c1, idesc_s);     // S^T = K Q^T      |  S  = Q K^T
                if (i >= 2) {
                    if (!mbar_wait(bar(B_YFREE), i & 1, abort_flag)) return false;
                    tc_fence_after();
                }
                mma_128x64_kk(t_y[i & 1], s_r2, c2, idesc_s);     // dP^T = V dO^T    |  dP = dO V^T
                tc_commit(bar(B_XY + (i & 1)));
                return true;
            };
            bool ok = mbar_wait(bar(B_RES), 0, abort_flag);
            for (int i = 0; i < 2 && i < n_items && ok; ++i) ok = issue_xy(i);
            for (int i = 0; i < n_items && ok; ++i) {
                if (!mbar_wait(bar(B_PDS + (i & 1)), (i >> 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after();
                const uint32_t c1 = s_ring + (i % RING) * STAGE, c2 = c1 + T64;
                if (!IS_DQ) {
                    mma_acc_k64(t_a2, t_x[i & 1], c2, idesc_acc, i > 0);             // dV += P^T dO
                    tc_commit(bar(B_XFREE));
                }
                mma_acc_k64(t_a1, t_y[i & 1], c1, idesc_acc, i > 0);                 // dK += dS^T Q   |  dQ += dS K
                tc_commit(bar(B_YFREE));
                tc_commit(bar(B_REMPTY + i % RING));
                if (i + 2 < n_items) ok = issue_xy(i + 2);                            // over P and dS of item i, behind their last reads
            }
            if (ok && n_items > 0) tc_commit(bar(B_DONE));
        }
    } else if (warp >= 2 && !bad) {
        const int quad = warp & 3, r = quad * 32 + lane;
        const int group = (warp - 2) >> 2;               // items group, group + 2, ...
        const int row_abs = tile * 128 + r;              // key position (dK/dV) or query position (dQ)
        const uint32_t lane_sel = static_cast<uint32_t>(quad * 32) << 16;
        const uint32_t tx = t_x[group] + lane_sel, ty = t_y[group] + lane_sel;
        float row_neg_lse2 = 0.f, row_dl = 0.f;
        int row_lo = 0;
        if (IS_DQ) {
            const size_t idx = (static_cast<size_t>(b) * p.Hq + head) * p.T + row_abs;
            row_neg_lse2 = p.neg_lse2[idx];
            row_dl = p.neg_delta[idx];
            if (HAS_LO) row_lo = __ldg(p.lo + row0 + row_abs);
        }
        const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), ds_scale2 = make_float2(p.scale, p.scale);
        bool ok = true;
        const bool do_prof = p.prof != nullptr && threadIdx.x == 64 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0;
        long long acc_[6] = {0, 0, 0, 0, 0, 0};
        long long t_ = clock64();
        for (int i = group; i < n_items && ok; i += 2) {
            const int st = i % RING;
            const int ct = first_ct + (IS_DQ ? i : i % per_head);     // index of the streamed 64-row tile inside the sequence
            const float* neg_lse2 = reinterpret_cast<const float*>(smem + OFF_VEC + st * VEC);
            const float* dl = neg_lse2 + 64;
            const int* q_lo = reinterpret_cast<const int*>(dl + 64);
            if (!IS_DQ && !mbar_wait(bar(B_RFULL + st), (i / RING) & 1, abort_flag)) { ok = false; break; }
            FB_PROF(0);
            if (!mbar_wait(bar(B_XY + group), (i >> 1) & 1, abort_flag)) { ok = false; break; }
            tc_fence_after();
            FB_PROF(1);
            uint32_t pb[32], sb[32];      // P and dS of this row, two bf16 to a register
            // causal mask: a key may not be later than the query.  dK/dV: row = key, column = query; dQ: row = query, column = key.
            const bool diag = IS_DQ ? (ct >= 2 * tile) : (ct < 2 * tile + 2);
            // lower bound: a key before the query's first visible key contributes nothing (q_lo is non-decreasing)
            const bool cut = HAS_LO && (IS_DQ ? (ct * 64 < row_lo) : (tile * 128 < q_lo[63]));
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                uint32_t x[32], y[32];
                tmem_ld_32x32(tx + hf * 32, x);
                tmem_ld_32x32(ty + hf * 32, y);
                tmem_ld_wait();
                FB_PROF(2);
                const int c0 = ct * 64 + hf * 32;
                if (diag) {
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (IS_DQ ? (c0 + c > row_abs) : (row_abs > c0 + c)) x[c] = 0xFF800000u;      // -inf: P = 0
                }
                if (cut) {
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (IS_DQ ? (c0 + c < row_lo) : (row_abs < q_lo[hf * 32 + c])) x[c] = 0xFF800000u;
                }
#pragma unroll
                for (int c = 0; c < 32; c += 4) {
                    float4 nl = make_float4(row_neg_lse2, row_neg_lse2, row_neg_lse2, row_neg_lse2), d4 = make_float4(row_dl, row_dl, row_dl, row_dl);
                    if (!IS_DQ) {
                        nl = *reinterpret_cast<const float4*>(neg_lse2 + hf * 32 + c);
                        d4 = *reinterpret_cast<const float4*>(dl + hf * 32 + c);
                    }
#pragma unroll
                    for (int k = 0; k < 4; k += 2) {
                        const float2 e = fma2(make_float2(__uint_as_float(x[c + k]), __uint_as_float(x[c + k + 1])), scale2, k ? make_float2(nl.z, nl.w) : make_float2(nl.x, nl.y));
                        const float2 pr = make_float2(ex2_approx(e.x), ex2_approx(e.y));
                        const float2 nd = k ? make_float2(d4.z, d4.w) : make_float2(d4.x, d4.y);
                        const float2 ds = mul2(pr, fma2(make_float2(__uint_as_float(y[c + k]), __uint_as_float(y[c + k + 1])), ds_scale2, nd));
                        const __nv_bfloat162 hp = __floats2bfloat162_rn(pr.x, pr.y), hs = __floats2bfloat162_rn(ds.x, ds.y);
                        if (!IS_DQ) pb[hf * 16 + (c + k) / 2] = reinterpret_cast<const uint32_t&>(hp);
                        sb[hf * 16 + (c + k) / 2] = reinterpret_cast<const uint32_t&>(hs);
                    }
                }
                FB_PROF(3);
            }
            if (!IS_DQ) tmem_st_32x32(tx, pb);
            tmem_st_32x32(ty, sb);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(bar(B_PDS + group));
            FB_PROF(5);
        }
        if (do_prof) {
            long long* dst = p.prof + (IS_DQ ? 8 : 0);
            for (int k = 0; k < 6; ++k) dst[k] = acc_[k];
            dst[6] = (n_items + 1) / 2;
        }
        if (ok && n_items > 0 && mbar_wait(bar(B_DONE), 0, abort_flag)) {
            tc_fence_after();
            const size_t width = static_cast<size_t>(p.Hq + 2 * p.Hkv) * D;
            __nv_bfloat16* base = p.d_qkv + static_cast<size_t>(row0 + row_abs) * width;
            if (IS_DQ) {
                store_acc128(t_a1, lane_sel, base + head * D, group);
            } else {
                store_acc128(t_a1, lane_sel, base + kcol, group);
                store_acc128(t_a2, lane_sel, base + vcol, group);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && p.error_flag) atomicExch(p.error_flag, IS_DQ ? 8 : 9);
    if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

}  // namespace fb64

const char* flash_attn_bwd64_sm100(const void* qkv, const void* d_out, const float* neg_lse2, const float* neg_delta, void* d_qkv, int B, int T, int Hq, int Hkv,
                                   float softmax_scale, int* error_flag, cudaStream_t stream, long long* prof, const int* lo, const int* kv_qend) {
    using namespace fb64;
    if (T % 128 != 0) return "flash_attn_bwd: T must be a multiple of 128";
    CUtensorMap q128, q64, do128, do64;
    const uint64_t width = static_cast<uint64_t>(Hq + 2 * Hkv) * D, owidth = static_cast<uint64_t>(Hq) * D, rows = static_cast<uint64_t>(B) * T;
    const char* e = nullptr;
    if ((e = make_tensor_map_2d(&q128, qkv, 2, width, rows, width * 2, 64, 128))) return e;
    if ((e = make_tensor_map_2d(&q64, qkv, 2, width, rows, width * 2, 64, 64))) return e;
    if ((e = make_tensor_map_2d(&do128, d_out, 2, owidth, rows, owidth * 2, 64, 128))) return e;
    if ((e = make_tensor_map_2d(&do64, d_out, 2, owidth, rows, owidth * 2, 64, 64))) return e;
    static std::atomic<uint64_t> limit[4];
    auto raise = [](auto* kernel, std::atomic<uint64_t>& done) { return raise_smem_limit(reinterpret_cast<const void*>(kernel), SMEM, done); };
    if (!(lo ? raise(fa_bwd64_kernel<true, true>, limit[3]) && raise(fa_bwd64_kernel<false, true>, limit[1])
             : raise(fa_bwd64_kernel<true, false>, limit[2]) && raise(fa_bwd64_kernel<false, false>, limit[0])))
        return "raising the shared-memory limit failed (flash_attn_bwd64)";
    if ((lo == nullptr) != (kv_qend == nullptr)) return "flash_attn_bwd: the lower bounds and the per-key-tile query ends come together";
    Params p{static_cast<__nv_bfloat16*>(d_qkv), neg_lse2, neg_delta, T, Hq, Hkv, softmax_scale, softmax_scale * LOG2E, error_flag, prof, lo, kv_qend};
    if (lo) {
        fa_bwd64_kernel<false, true><<<dim3(T / 128, Hkv, B), THREADS, SMEM, stream>>>(q128, q64, do128, do64, p);
        fa_bwd64_kernel<true, true><<<dim3(T / 128, Hq, B), THREADS, SMEM, stream>>>(q128, q64, do128, do64, p);
    } else {
        fa_bwd64_kernel<false, false><<<dim3(T / 128, Hkv, B), THREADS, SMEM, stream>>>(q128, q64, do128, do64, p);
        fa_bwd64_kernel<true, false><<<dim3(T / 128, Hq, B), THREADS, SMEM, stream>>>(q128, q64, do128, do64, p);
    }
    return cudaGetLastError() == cudaSuccess ? nullptr : "flash_attn_bwd64 launch failed";
}

// Row statistics of the backward in the layout it reads, [B, Hq, T]: -scale * sum_d dO * O and -lse * log2(e).  Half a warp per (token, head);
// a block takes 16 consecutive tokens of one head, so its results are two whole sectors.
__global__ void __launch_bounds__(256) fa_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse,
                                                       float* __restrict__ neg_lse2, float* __restrict__ neg_delta, int T, int Hq, float scale,
                                                       unsigned blocks) {
    const int sub = threadIdx.x & 15;
    for (unsigned blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
        const unsigned h = blk % Hq;
        const size_t tok = static_cast<size_t>(blk / Hq) * 16 + (threadIdx.x >> 4);      // T is a multiple of 16: a block stays in one sequence
        const size_t it = tok * Hq + h;
        const uint4 a = *reinterpret_cast<const uint4*>(o + it * 128 + sub * 8), g = *reinterpret_cast<const uint4*>(d_o + it * 128 + sub * 8);
        const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
        const __nv_bfloat162* pg = reinterpret_cast<const __nv_bfloat162*>(&g);
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pg[i]);
            s += x.x * y.x + x.y * y.y;
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (sub == 0) {
            const size_t dst = (tok / T * Hq + h) * T + tok % T;
            neg_delta[dst] = -s * scale;
            neg_lse2[dst] = -lse[it] * fb64::LOG2E;
        }
    }
}

const char* flash_attn_bwd_sm100(const void* qkv, const void* out, const void* d_out, const float* lse, float* stats, void* d_qkv, int B, int T, int Hq,
                                 int Hkv, float softmax_scale, int* error_flag, int num_sms, cudaStream_t stream, const int* lo, const int* kv_qend,
                                 long long* prof) {
    if (T % 128 != 0) return "flash_attn_bwd: T must be a multiple of 128";
    const unsigned blocks = static_cast<unsigned>(static_cast<size_t>(B) * T / 16 * Hq);
    if (blocks == 0) return nullptr;
    const unsigned cap = static_cast<unsigned>(num_sms) * 32;
    float* neg_delta = stats + static_cast<size_t>(B) * T * Hq;
    fa_delta_kernel<<<blocks < cap ? blocks : cap, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out), lse, stats,
                                                                      neg_delta, T, Hq, softmax_scale, blocks);
    return flash_attn_bwd64_sm100(qkv, d_out, stats, neg_delta, d_qkv, B, T, Hq, Hkv, softmax_scale, error_flag, stream, prof, lo, kv_qend);
}

}  // namespace sg
