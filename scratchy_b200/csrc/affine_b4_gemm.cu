// MLX affine int4 (groups of 32, 64, 128): prefill GEMM on tcgen05 tensor cores, M > 128 (from 97 on where k is short).
//
//   y[m,n] = bf16( sum_k x[m,k] * w[n,k] (+ bias[n]) ),  w = the bit-exact bf16 dequantisation of the codes
//
// Persistent, warp-specialised CTA (736 threads), one per SM.  A tile is 128 channels (the rows of the MMA) by `width` tokens (its
// columns, 96 to 192):
//   warps 0-15   dequantise: four groups of four warps take the halves (64 k) of alternate 128-k chunks; a thread expands 64 codes of
//                one channel and writes them to TMEM with tcgen05.st, where the MMA reads its A operand: no swizzled shared-memory
//                image and no proxy fence, and the shared memory holds activations in flight instead
//   warps 16-19  epilogue: tcgen05.ld (lane = channel, column = token), one rounding to bf16 (or f32 partials), stores of 32
//                consecutive channels of a token per warp
//   warp 20      producer of the packed weights: one tiled copy per chunk (affine_b4_tc.cuh), ahead of the preceding kernel
//   warp 21      producer of the activations: tiled TMA loads of 64 k x the tokens (128-byte swizzle, zeros outside)
//   warp 22      owns TMEM; the warp issues 8 tcgen05.mma (128 x width x 16) per chunk and commits the barriers, a lane elected
//                inside each: 3072 -> 16384 at 4096 tokens 284 us, 297 with the lane elected once and branches around the issue
// TMEM holds two accumulators of 192 columns (the epilogue of a tile overlaps the main loop of the next) and two stages of 64
// columns of dequantised weights.  No multicast: every CTA issues its own loads.
//
// What bounds it: the MMAs, 64 cycles for 128 columns and 96 for 192 (alone in a loop, A in TMEM: the tensor core's full rate), 768 a chunk
// at 192, and for large calls the clock that the power limit leaves: 2048 tokens of 3072 -> 8192 73.7 us (1.40 PFLOP/s, what cuBLAS
// sustains) in a stream of calls, 72.4 with the election inside (70.2 with the plan below).  It was 83.7 us, 1250 cycles a chunk whatever the width, while one lane issued eight bulk copies a chunk
// and the dequantised weights were handed over in stages of a whole chunk.  Wide tiles pay, since a chunk is expanded once for all of a
// tile's tokens.
#include <cuda.h>

#include <algorithm>

#include "affine_b4_tc.cuh"
#include "gemv_common.cuh"
#include "skinny.cuh"

bool affine_b4_gemm_tc_enabled() { return true; }
// Defined in affine_b4_gemm_pair.cu
bool affine_b4_gemm_pair_applies(int M, int N, int K, int sms);
int32_t affine_b4_gemm_pair_launch(scr_ctx* ctx, const CUtensorMap& x_map, const uint8_t* packed, uint16_t* y, int M, int N, int K,
                                   int gs, int out_f32, const uint16_t* bias, cudaStream_t stream, bool* launched);
// Defined in affine_b4_skinny.cu
bool affine_b4_skinny_applies(int M, int N, int K, int sms);
int32_t affine_b4_skinny_launch(scr_ctx* ctx, const uint8_t* packed, const uint16_t* x, uint16_t* y, int M, int N, int K, int gs, int out,
                                const uint16_t* bias, float scale, cudaStream_t stream);
size_t affine_b4_gemm_tc_workspace_plan(int M, int N, int K);
size_t affine_b4_gemm_tc_workspace(int M, int N, int K) { return affine_b4_gemm_tc_workspace_plan(M, N, K); }

#define A4G_BN 128            // channels of a tile
constexpr int A4G_THREADS = 736, A4G_DQ_WARPS = 16;
constexpr int A4G_WIDTH = 192;                                  // tokens of a tile at most (a multiple of 16)
// Activation stages of 64 k; packed-weight and dequantised stages of 128 k, even in number: a stage always belongs to the same
// groups, whose waits take its phases in order.  A dequantised stage is handed over and freed in halves of 64 k
constexpr int A4G_SX = 7, A4G_SP = 4, A4G_SA = 2;
constexpr uint32_t A4G_XSTAGE = A4G_WIDTH * 128u;
constexpr uint32_t A4G_POFF = A4G_SX * A4G_XSTAGE;
constexpr uint32_t A4G_BARS = 320;
constexpr uint32_t A4G_TMEM = 512, A4G_ACOL = 2 * A4G_WIDTH;    // columns; where the dequantised stages start

static __device__ __forceinline__ void a4g_tma_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}

static __device__ __forceinline__ uint4 a4g_lds_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
static __device__ __forceinline__ uint32_t a4g_lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// Finishes the split tiles: sums a tile's ks_tail partial tiles in slab order (deterministic) and stores the
// result, rounded once (or as f32 partials).  One CTA per (tail tile, 8 rows), one float4 per thread.
__global__ void __launch_bounds__(256) affine_b4_gemm_tail_finish_kernel(const float* __restrict__ slabs, int ks_tail, int n_tail,
                                                                         int full, int MT, int tile_rows, int M, int N,
                                                                         uint16_t* __restrict__ y, int out_f32,
                                                                         const uint16_t* __restrict__ bias) {
    const int groups = tile_rows / 8;
    const int tt = blockIdx.x / groups, grp = blockIdx.x - tt * groups;
    const int tile = full + tt;
    const int mt = tile % MT, nb = tile / MT;
    const size_t tile_elems = (size_t)tile_rows * A4G_BN;
    const int rl = grp * 8 + threadIdx.x / (A4G_BN / 4), c4 = (threadIdx.x % (A4G_BN / 4)) * 4;
    const int m = mt * tile_rows + rl, n = nb * A4G_BN + c4;
    if (m >= M || n >= N) return;
    const float* p = slabs + (size_t)tt * tile_elems + (size_t)rl * A4G_BN + c4;
    float4 a = *reinterpret_cast<const float4*>(p);
    for (int k = 1; k < ks_tail; ++k) {
        const float4 b = *reinterpret_cast<const float4*>(p + (size_t)k * n_tail * tile_elems);
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (n + j >= N) break;
        if (out_f32) {
            reinterpret_cast<float*>(y)[(size_t)m * N + n + j] = v[j];
        } else {
            const __nv_bfloat16 o = __float2bfloat16_rn(bias ? v[j] + __uint_as_float(uint32_t(bias[n + j]) << 16) : v[j]);
            y[(size_t)m * N + n + j] = *reinterpret_cast<const uint16_t*>(&o);
        }
    }
}

template <int GS>
__global__ void __launch_bounds__(A4G_THREADS, 1)
affine_b4_gemm_tc_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const uint8_t* __restrict__ packed,
                         uint16_t* __restrict__ y, int M, int N, int RB, int KC, int width, int MT, int out_f32, const uint16_t* __restrict__ bias, int full, int ks_tail, float* __restrict__ slabs,
                         int* __restrict__ status) {
    constexpr uint32_t kBlock = aff_block_bytes(GS), kPStage = 8u * kBlock, kBarOff = A4G_POFF + A4G_SP * kPStage;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar = smem_base + kBarOff;
    auto xfull = [&](int s) { return bar + 8u * s; };
    auto xempty = [&](int s) { return bar + 8u * (A4G_SX + s); };
    auto pfull = [&](int s) { return bar + 8u * (2 * A4G_SX + s); };
    auto pempty = [&](int s) { return bar + 8u * (2 * A4G_SX + A4G_SP + s); };
    auto afull = [&](int s) { return bar + 8u * (2 * A4G_SX + 2 * A4G_SP + s); };
    auto aempty = [&](int s) { return bar + 8u * (2 * A4G_SX + 2 * A4G_SP + 2 * A4G_SA + s); };
    constexpr int kAccSlot = 2 * A4G_SX + 2 * A4G_SP + 4 * A4G_SA;
    auto accf = [&](int b) { return bar + 8u * (kAccSlot + b); };
    auto acce = [&](int b) { return bar + 8u * (kAccSlot + 2 + b); };
    static_assert(8 * (kAccSlot + 5) <= A4G_BARS, "barriers");
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + kBarOff + 8 * (kAccSlot + 4));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    // Work units: the first `full` tiles whole; each of the remaining (tail) tiles as ks_tail units that share its k
    // extent and leave f32 partial tiles in `slabs` for the finishing kernel.
    const int n_tail = MT * (RB / 8) - full, units = full + n_tail * ks_tail;

    if (threadIdx.x == 0) {
        for (int s = 0; s < A4G_SX; ++s) { mbar_init(xfull(s), 1); mbar_init(xempty(s), 1); }
        for (int s = 0; s < A4G_SP; ++s) { mbar_init(pfull(s), 1); mbar_init(pempty(s), A4G_DQ_WARPS / 2); }
        for (int s = 0; s < 2 * A4G_SA; ++s) { mbar_init(afull(s), A4G_DQ_WARPS / 4); mbar_init(aempty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(accf(b), 1); mbar_init(acce(b), 4); }
        fence_mbar_init();
    }
    if (warp == 22) {
        tmem_alloc(smem_u32((const void*)tmem_slot), A4G_TMEM);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    skinny_pdl_trigger();                              // not before this CTA has its TMEM: the next kernel's CTAs could take it first

    if (warp == 20) {
        if (lane == 0) {
            int c = 0;                                 // chunks so far
            for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
                int tile, ks, kc_lo, kc_hi;
                tc_unit(unit, full, ks_tail, KC, tile, ks, kc_lo, kc_hi);
                const int rb0 = (tile / MT) * 8;
                for (int kc = kc_lo; kc < kc_hi; ++kc, ++c) {
                    const int s = c % A4G_SP;
                    if (c == A4G_SP) skinny_pdl_wait();        // only the weights may be touched before the preceding kernel has finished
                    mbar_wait(pempty(s), ((uint32_t)(c / A4G_SP) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                    mbar_arrive_expect_tx(pfull(s), kPStage);
                    affine_load_chunk(smem_base + A4G_POFF + s * kPStage, &w_map, kc, rb0, pfull(s));
                }
            }
        }
    } else if (warp == 21) {
        if (lane == 0) {
            skinny_pdl_wait();
            int s = 0;
            uint32_t ph = 0;
            for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
                int tile, ks, kc_lo, kc_hi;
                tc_unit(unit, full, ks_tail, KC, tile, ks, kc_lo, kc_hi);
                const int m0 = (tile % MT) * width;
                for (int k = 2 * kc_lo; k < 2 * kc_hi; ++k) {
                    mbar_wait(xempty(s), ph ^ 1u, status, TC_ERR_EMPTY_WAIT);
                    mbar_arrive_expect_tx(xfull(s), (uint32_t)width * 128u);
                    a4g_tma_2d(smem_base + s * A4G_XSTAGE, &x_map, k * 64, m0, xfull(s));
                    if (++s == A4G_SX) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 22) {
        skinny_pdl_wait();
        const uint32_t idesc = umma_idesc(1, 1, A4G_BN, (uint32_t)width);
        int s = 0, c = 0, it = 0;
        uint32_t ph = 0;
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x, ++it) {
            int tile, ks, kc_lo, kc_hi;
            tc_unit(unit, full, ks_tail, KC, tile, ks, kc_lo, kc_hi);
            const int buf = it & 1;
            mbar_wait(acce(buf), ((uint32_t)(it >> 1) & 1u) ^ 1u, status, TC_ERR_ACC_EMPTY);
            const uint32_t d = tmem + (uint32_t)(buf * A4G_WIDTH);
            for (int kc = kc_lo; kc < kc_hi; ++kc, ++c) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int a = 2 * (c % A4G_SA) + h;
                    const uint32_t ac = tmem + A4G_ACOL + (uint32_t)(32 * a);
                    const uint64_t bdesc = umma_desc_k_sw128(smem_base + s * A4G_XSTAGE);
                    mbar_wait(xfull(s), ph, status, TC_ERR_FULL_WAIT);
                    mbar_wait(afull(a), (uint32_t)(c / A4G_SA) & 1u, status, TC_ERR_DEQ_WAIT);
                    tc_fence_after();
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4)
                        umma_f16_ta_warp(d, ac + (uint32_t)(8 * k4), bdesc + (uint64_t)(2 * k4), idesc, kc > kc_lo || h > 0 || k4 > 0);
                    umma_commit_warp(aempty(a));
                    umma_commit_warp(xempty(s));
                    if (++s == A4G_SX) { s = 0; ph ^= 1u; }
                }
            }
            umma_commit_warp(accf(buf));
        }
    } else if (warp < A4G_DQ_WARPS) {
        const bool check = *reinterpret_cast<const unsigned int*>(packed + (size_t)RB * KC * kBlock) != 0;
        const int grp = warp >> 2, kh = grp & 1, row = (warp & 3) * 32 + lane, half = (row >> 3) & 1, g = row & 7;
        const uint32_t dst0 = tmem + A4G_ACOL + (uint32_t)(32 * grp) + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t src0 = smem_base + A4G_POFF + (uint32_t)((row >> 4) * kBlock);
        int c = 0;
        bool waited = false;
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
            int tile, ks, kc_lo, kc_hi;
            tc_unit(unit, full, ks_tail, KC, tile, ks, kc_lo, kc_hi);
            for (int kc = kc_lo; kc < kc_hi; ++kc, ++c) {
                if ((c & 1) != grp >> 1) continue;
                const int s = c % A4G_SP;
                if (c >= A4G_SA && !waited) {
                    skinny_pdl_wait();                 // from here on a wait depends on the activations
                    waited = true;
                }
                mbar_wait(pfull(s), (uint32_t)(c / A4G_SP) & 1u, status, TC_ERR_FULL_WAIT);
                const uint32_t blk = src0 + s * kPStage;
                uint4 piece[2];
                uint32_t sb[2];
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    piece[t] = a4g_lds_v4(blk + (uint32_t)(half * 512 + (4 * g + 2 * kh + t) * 16));
                    sb[t] = a4g_lds_u32(blk + 1024u + (uint32_t)(((g << GS) + ((2 * kh + t) >> (2 - GS))) * 8 + half * 4));
                }
                mbar_wait(aempty(grp), ((uint32_t)(c / A4G_SA) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                tc_fence_after();
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    uint32_t w[16];
                    if (check) {
                        affine_dequant_piece<true>(piece[t], sb[t], w);
                    } else {
                        const AffineScaled cs = affine_scaled_consts(sb[t]);     // w * 2^-7: the sums are multiplied by 2^7
                        affine_dequant_word_scaled(piece[t].x, cs, w + 0);
                        affine_dequant_word_scaled(piece[t].y, cs, w + 4);
                        affine_dequant_word_scaled(piece[t].z, cs, w + 8);
                        affine_dequant_word_scaled(piece[t].w, cs, w + 12);
                    }
                    tmem_st_32x16(dst0 + (uint32_t)(16 * t), w);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(afull(grp));
                    mbar_arrive(pempty(s));
                }
            }
        }
    } else {
        const int q = warp & 3;                        // TMEM lane quadrant this warp may read
        const float factor = (*reinterpret_cast<const unsigned int*>(packed + (size_t)RB * KC * kBlock) != 0) ? 1.0f : AFF_SCALED_FACTOR;
        skinny_pdl_wait();                             // y and the slabs may still be in use by a preceding kernel
        int it = 0;
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x, ++it) {
            int tile, ks, kc_lo, kc_hi;
            tc_unit(unit, full, ks_tail, KC, tile, ks, kc_lo, kc_hi);
            const int m0 = (tile % MT) * width, nb = tile / MT, n = nb * A4G_BN + q * 32 + lane, buf = it & 1;
            const bool split = unit >= full && ks_tail > 1;
            const float b = !split && bias && n < N ? __uint_as_float(uint32_t(bias[n]) << 16) : 0.0f;
            mbar_wait(accf(buf), (uint32_t)(it >> 1) & 1u, status, TC_ERR_ACC_FULL);
            tc_fence_after();
            const int tokens = min(width, M - m0);
            const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * A4G_WIDTH);
            // Runs of 16 tokens with no branch between their stores.  (With the bounds and the kind of output looked up for every token
            // a store took 125 cycles and a tile 12 us, longer than the main loop of a k of 512: 3000 tokens of 512 -> 8192 80.2 us,
            // here 25.2; 2048 tokens of 3072 -> 8192 90.5 and 83.9, in a stream of such calls.)
            auto drain = [&](auto* dst, size_t stride, bool real, auto put) {
                for (int c = 0; c < tokens; c += 16, dst += 16 * stride) {
                    uint32_t r[16];
                    tmem_ld_32x16(acc + (uint32_t)c, r);
                    tmem_ld_wait();
                    if (!real) continue;
                    if (c + 16 <= tokens) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) dst[j * stride] = put(__uint_as_float(r[j]) * factor);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c + j < tokens) dst[j * stride] = put(__uint_as_float(r[j]) * factor);
                    }
                }
            };
            auto same = [](float v) { return v; };
            auto rounded = [](float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); };
            const size_t at = (size_t)m0 * N + n;
            if (split) drain(slabs + ((size_t)ks * n_tail + (tile - full)) * (size_t)(width * A4G_BN) + q * 32 + lane, A4G_BN, true, same);
            else if (out_f32) drain(reinterpret_cast<float*>(y) + at, N, n < N, same);
            else if (bias) drain(y + at, N, n < N, [&](float v) { return rounded(v + b); });
            else drain(y + at, N, n < N, rounded);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acce(buf));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 22) {
        tc_fence_after();
        tmem_dealloc(tmem, A4G_TMEM);
    }
}

// ---- host --------------------------------------------------------------------------------
// The tokens of a tile and how the tiles are cut into work units (tc_plan_units).  A 128-k chunk takes about 0.26 us and 1.23 ns a token (148
// tiles of 24 chunks a round: further rounds 9.0 us at 112 tokens, 10.0 at 128, 10.6 at 144, 10.9 at 160, 11.3 at 176, 11.9 at 192), and a tile's drain at
// the end 6.5 ns a token; the width whose rounds fill the GPU best wins.  512 tokens of 3072 -> 8192 26.6 us at 192, 23.1 at 128; 777 of 8192 -> 3072
// 35.4 and at 144 30.1; 200 of 3072 -> 3072 13.0 and at 112 11.1.  A cut costs about 5 us in all.
struct AffineGemmPlan {
    int width, mt, tiles, full, ks_tail;
    float us;                                            // estimate
    int n_tail() const { return tiles - full; }
    size_t slab_floats() const { return ks_tail > 1 ? (size_t)ks_tail * n_tail() * (size_t)(width * A4G_BN) : 0; }
};
static AffineGemmPlan affine_gemm_plan(int M, int N, int K, int sms) {
    const AffineGeom g = affine_geom(N, K, 64);
    AffineGemmPlan best{};
    float least = 1e30f;
    if (M <= 96 || (M <= 128 && K > 1536)) {
        // few tokens of a matrix of more tiles than SMs: whole tiles of just these tokens, no workspace
        best.width = (M + 15) & ~15;
        best.mt = 1;
        best.tiles = best.full = g.RB * 16 / A4G_BN;
        best.ks_tail = 1;
        return best;
    }
    for (int width = A4G_WIDTH; width >= 96; width -= 16) {
        AffineGemmPlan p;
        p.width = width;
        p.mt = scr_ceil_div(M, width);
        p.tiles = p.mt * (g.RB * 16 / A4G_BN);
        const float us = 0.26f + 0.00123f * width;
        p.us = tc_plan_units(p.tiles, g.KC, sms, us, &p.full, &p.ks_tail, 1.6f, 3.4f) * g.KC * us + 0.0065f * width;
        if (p.us < least * 0.99f) {
            least = p.us;
            best = p;
        }
    }
    return best;
}
size_t affine_b4_gemm_tc_workspace_plan(int M, int N, int K) {
    if (affine_b4_skinny_applies(M, N, K, tc_sm_count())) return 0;
    return affine_gemm_plan(M, N, K, tc_sm_count()).slab_floats() * sizeof(float);
}

template <int GS>
static int32_t affine_gemm_launch(scr_ctx* ctx, tc_encode_tiled_fn enc, const CUtensorMap& map, const uint8_t* packed, uint16_t* y, int M, int N, int K, int out_f32,
                                  const uint16_t* bias, const AffineGemmPlan& p, float* slabs, cudaStream_t stream) {
    const AffineGeom g = affine_geom(N, K, 64);
    const int units = p.full + p.n_tail() * p.ks_tail;
    CUtensorMap w_map;
    if (!affine_w_map(&w_map, enc, packed, g.RB, g.KC, GS)) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled failed");
    constexpr size_t smem = A4G_POFF + A4G_SP * 8u * aff_block_bytes(GS) + A4G_BARS + 1024;
    const cudaError_t e = skinny_launch(affine_b4_gemm_tc_kernel<GS>, std::min(units, ctx->sm_count), 1, A4G_THREADS, smem, stream, map, w_map, packed, y, M, N, g.RB,
                                        g.KC, p.width, p.mt, out_f32, bias, p.full, p.ks_tail, slabs, ctx->dev_status);
    if (e != cudaSuccess) return scr_fail(ctx, SCR_E_CUDA, "affine_b4_gemm_tc: %s", cudaGetErrorString(e));
    const int32_t st = scr_check_launch(ctx, "affine_b4_gemm_tc");
    if (st || p.ks_tail == 1) return st;
    affine_b4_gemm_tail_finish_kernel<<<p.n_tail() * (p.width / 8), 256, 0, stream>>>(slabs, p.ks_tail, p.n_tail(), p.full, p.mt, p.width, M, N, y, out_f32,
                                                                                      bias);
    return scr_check_launch(ctx, "affine_b4_gemm_tail_finish");
}

static bool affine_gemm_x_map(CUtensorMap* map, tc_encode_tiled_fn enc, const uint16_t* x, int M, int K, int rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int32_t affine_b4_gemm_tc_launch(scr_ctx* ctx, const uint8_t* packed, const uint16_t* x, uint16_t* y, int M, int N, int K,
                                 int gs, int out_f32, const uint16_t* bias, void* workspace, size_t, cudaStream_t stream) {
    if (((uintptr_t)packed & 127u) != 0) return scr_fail(ctx, SCR_E_ALIGN, "packed weights must be 128-byte aligned for the GEMM path");
    if (!scr_aligned16(y)) return scr_fail(ctx, SCR_E_ALIGN, "y must be 16-byte aligned");
    if (affine_b4_skinny_applies(M, N, K, ctx->sm_count))
        return affine_b4_skinny_launch(ctx, packed, x, y, M, N, K, gs, out_f32 ? GEMV_OUT_F32 : GEMV_OUT_BF16, bias, 1.0f, stream);
    tc_encode_tiled_fn enc = tc_tensor_map_encoder();
    if (!enc) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled entry point not available");
    CUtensorMap map;
    const AffineGemmPlan plan = affine_gemm_plan(M, N, K, ctx->sm_count);
    if (affine_b4_gemm_pair_applies(M, N, K, ctx->sm_count)) {
        bool launched = false;
        if (!affine_gemm_x_map(&map, enc, x, M, K, 128)) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled failed");
        const int32_t st = affine_b4_gemm_pair_launch(ctx, map, packed, y, M, N, K, gs, out_f32, bias, stream, &launched);
        if (st || launched) return st;
    }
    float* slabs = reinterpret_cast<float*>(workspace);
    if (plan.ks_tail > 1 && (!slabs || !scr_aligned16(slabs))) return scr_fail(ctx, SCR_E_WORKSPACE, "split-K needs an aligned workspace");
    if (!affine_gemm_x_map(&map, enc, x, M, K, plan.width)) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled failed");
    return gs == 2 ? affine_gemm_launch<2>(ctx, enc, map, packed, y, M, N, K, out_f32, bias, plan, slabs, stream)
                   : affine_gemm_launch<1>(ctx, enc, map, packed, y, M, N, K, out_f32, bias, plan, slabs, stream);
}
