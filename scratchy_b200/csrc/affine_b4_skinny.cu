// MLX affine int4: GEMM for few tokens (up to 128; from how many on, affine_b4.cu) on tcgen05 tensor cores, weights as the rows of the MMA (skinny.cuh).
//
//   y[m,n] = bf16( sum_k x[m,k] * w[n,k] (+ bias[n]) ),  w = the bit-exact bf16 dequantisation of the codes
//
// with the matvec's ends (a scale, the add into the residual stream, the gate/up pairing).  A unit is 128 channels by one CTA's share of the 128-k
// chunks; 352 threads:
//   warps 0-7    dequantise: two groups of four warps take alternate chunks; a thread expands the 128 codes of ONE channel
//                and writes them to TMEM with tcgen05.st, where the MMA reads its A operand: no swizzled shared-memory
//                image, no proxy fence.  Afterwards they drain the accumulator.
//   warp 8       producer of the packed weights (one tiled copy of 8 blocks per chunk, affine_b4_tc.cuh), which are load-time
//                constants: it starts before the preceding kernel of the stream has finished, and ahead of this kernel's own setting up
//   warp 9       producer of the activations (2 tiled TMA loads of 64 k x the tokens, 128-byte swizzle, zeros outside)
//   warp 10      owns TMEM; the warp issues 8 tcgen05.mma (128 x tokens x 16) per chunk, a lane elected inside each
// A stage of activations and one of dequantised weights go round together: the group's warps and the activations' bytes complete one barrier,
// one commit frees both.  (A wait that passes costs the issuing warp 69 to 89 cycles and a commit 25; the eight MMAs 128 at 32 tokens.)
//
// What bounds it: 1.0 us from the end of the kernel before to the release of the wait and 0.4 to the first activations (2 more on SMs whose CTA of
// the launch before ended last: theirs starts then), then HBM and the way of a chunk round the stages, about 0.25 us a chunk and SM (its 9.2 KB take
// 0.21 from HBM), then about 2 us for the sums and the stores.  Streams of calls: 45 tokens of 8192 -> 3072 8.0 us (16.1 on the 128-token tiles of the
// prefill GEMM, 11.4 with a bulk copy for every block, two CTAs to an SM and two cluster barriers at the end, 8.6 with a barrier pair each for
// activations and weights and the lane elected around the issue); 16 tokens of 3072 -> 16384 9.9 us, 20.1 in the matvec.  Sixteen dequantising
// warps gain nothing (8.7 for the 8.3 of that form), nor do more stages.  The decode step of Llama-3.2-3B at 32 sequences 2.67 -> 2.23 ms.
#include <cuda.h>

#include "affine_b4_tc.cuh"
#include "gemv_common.cuh"
#include "skinny.cuh"

namespace {

constexpr int A4S_GROUPS = 2, A4S_DQ_WARPS = 4 * A4S_GROUPS, A4S_THREADS = 32 * (A4S_DQ_WARPS + 3);

template <int TN>
struct A4SCfg {
    static constexpr int kSA = TN == 128 ? 4 : 3;                                       // stages of activations (128 k) and of dequantised weights in TMEM (64
                                                                        //   columns each beside the accumulator): one a group, and one pair
                                                                        //   of barriers for both
    static constexpr int kSP = TN == 128 ? 8 : 6;                       // packed-weight stages, even: a stage always belongs to the
                                                                        //   same of the two groups, whose waits take its phases in order
    static constexpr uint32_t kACol = TN < 32 ? 32 : TN, kTmemCols = TN == 128 ? 512 : 256;
    static constexpr uint32_t kXStage = TN * 256u;                      // 2 atoms of TN rows x 128 B
    static constexpr uint32_t kPOff = kSA * kXStage;
};

__device__ __forceinline__ uint4 a4s_lds_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t a4s_lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void a4s_tma_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}

// The 128 codes of channel `row` of a chunk -> 64 TMEM columns at `dst` (this warp's lanes).
template <int GS, bool CHECK>
__device__ __forceinline__ void a4s_expand(uint32_t stage, int row, uint32_t dst) {
    const int half = (row >> 3) & 1, g = row & 7;
    const uint32_t blk = stage + (uint32_t)((row >> 4) * aff_block_bytes(GS));
    uint4 piece[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) piece[t] = a4s_lds_v4(blk + (uint32_t)(half * 512 + (4 * g + t) * 16));
    uint32_t sb[1 << GS];
#pragma unroll
    for (int h = 0; h < (1 << GS); ++h) sb[h] = a4s_lds_u32(blk + 1024u + (uint32_t)(((g << GS) + h) * 8 + half * 4));
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const uint32_t s = sb[t >> (2 - GS)];
        uint32_t w[16];
        if (CHECK) {
            affine_dequant_piece<true>(piece[t], s, w);
        } else {
            const AffineScaled c = affine_scaled_consts(s);          // w * 2^-7: the sums are multiplied by 2^7
            affine_dequant_word_scaled(piece[t].x, c, w + 0);
            affine_dequant_word_scaled(piece[t].y, c, w + 4);
            affine_dequant_word_scaled(piece[t].z, c, w + 8);
            affine_dequant_word_scaled(piece[t].w, c, w + 12);
        }
        tmem_st_32x16(dst + 16u * t, w);
    }
}

template <int TN, int GS>
__global__ void __launch_bounds__(A4S_THREADS, TN == 128 ? 1 : 2)
affine_b4_skinny_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const uint8_t* __restrict__ packed,
                        uint16_t* __restrict__ y, int M, int N, int RB, int KC, int split, int over_rings,
                        int out, const uint16_t* __restrict__ bias, float scale, int* __restrict__ status) {
    using C = A4SCfg<TN>;
    constexpr uint32_t kBlock = aff_block_bytes(GS), kPStage = 8u * kBlock, kBarOff = C::kPOff + C::kSP * kPStage, kSumOff = kBarOff + 512u;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar = smem_base + kBarOff;
    auto full = [&](int s) { return bar + 8u * s; };
    auto aempty = [&](int s) { return bar + 8u * (C::kSA + s); };
    auto pfull = [&](int s) { return bar + 8u * (2 * C::kSA + s); };
    auto pempty = [&](int s) { return bar + 8u * (2 * C::kSA + C::kSP + s); };
    constexpr int kSlots = 2 * C::kSA + 2 * C::kSP;
    const uint32_t accf = bar + 8u * kSlots, rbar = accf + 8u;
    static_assert(8 * (kSlots + 3) <= 512, "barriers");
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + kBarOff + 8 * (kSlots + 2));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int tile = blockIdx.x / split, rank = blockIdx.x - tile * split;
    int kc_lo, kc_hi;
    skinny_range(KC, rank, split, kc_lo, kc_hi);
    const int steps = kc_hi - kc_lo;

    // The first weights are on their way before anything else is set up: their copy needs only its own barriers.
    auto load = [&](int i) {
        const int s = i % C::kSP;
        mbar_arrive_expect_tx(pfull(s), kPStage);
        affine_load_chunk(smem_base + C::kPOff + s * kPStage, &w_map, kc_lo + i, tile * 8, pfull(s));
    };
    const int early = min(steps, 2);
    if (warp == A4S_DQ_WARPS) {
        if (lane == 0) {
            for (int s = 0; s < C::kSP; ++s) { mbar_init(pfull(s), 1); mbar_init(pempty(s), 4); }
            fence_mbar_init();
            for (int i = 0; i < early; ++i) load(i);
        }
        __syncwarp();
    } else if (warp == A4S_DQ_WARPS + 1) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
            for (int s = 0; s < C::kSA; ++s) { mbar_init(full(s), 5); mbar_init(aempty(s), 1); }         // a group's warps and the copy's lane
            mbar_init(accf, 1);
            skinny_expect(rbar, M, split, rank, over_rings);
            fence_mbar_init();
        }
        __syncwarp();
    } else if (warp == A4S_DQ_WARPS + 2) {
        tmem_alloc(smem_u32((const void*)tmem_slot), C::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (split > 1 && !over_rings) skinny_cluster_arrive();
    skinny_pdl_trigger();                              // not before this CTA has its TMEM: the next kernel's CTAs could take it first
    auto a_col = [&](int s) { return tmem + C::kACol + (uint32_t)(64 * s); };

    // Only the weights may be touched before the preceding kernel has finished.  A wait that depends on the activations
    // comes after griddepcontrol.wait, so that its bound does not run against that kernel.
    if (warp == A4S_DQ_WARPS) {
        if (lane == 0) {
            for (int i = early; i < steps; ++i) {
                if (i == C::kSP) skinny_pdl_wait();
                mbar_wait(pempty(i % C::kSP), ((uint32_t)(i / C::kSP) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                load(i);
            }
        }
    } else if (warp == A4S_DQ_WARPS + 1) {
        if (lane == 0) {
            skinny_pdl_wait();
            const uint32_t tokens = (uint32_t)(M + 15) & ~15u;
            for (int i = 0; i < steps; ++i) {
                const int s = i % C::kSA;
                mbar_wait(aempty(s), ((uint32_t)(i / C::kSA) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                mbar_arrive_expect_tx(full(s), tokens * 256u);
                const uint32_t xs = smem_base + s * C::kXStage;
                a4s_tma_2d(xs, &x_map, (kc_lo + i) * 128, 0, full(s));
                a4s_tma_2d(xs + TN * 128u, &x_map, (kc_lo + i) * 128 + 64, 0, full(s));
            }
        }
    } else if (warp == A4S_DQ_WARPS + 2) {
        // The warp goes round as a whole, so that the descriptors stay in uniform registers: an MMA of few columns is shorter than its
        // issue from a divergent thread (55 cycles).  One wait and one commit a chunk: each costs about what eight MMAs of 16 columns do.
        skinny_pdl_wait();
        const uint32_t idesc = umma_idesc(1, 1, SKINNY_ROWS, (uint32_t)(M + 15) & ~15u);
        for (int i = 0; i < steps; ++i) {
            const int s = i % C::kSA;
            const uint32_t xs = smem_base + s * C::kXStage, ac = a_col(s);
            const uint64_t b0 = umma_desc_k_sw128(xs), b1 = umma_desc_k_sw128(xs + TN * 128u);
            mbar_wait(full(s), (uint32_t)(i / C::kSA) & 1u, status, TC_ERR_FULL_WAIT);
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < 8; ++k) umma_f16_ta_warp(tmem, ac + (uint32_t)(8 * k), (k < 4 ? b0 : b1) + (uint64_t)(2 * (k & 3)), idesc, i > 0 || k > 0);
            umma_commit_warp(aempty(s));
        }
        umma_commit_warp(accf);
    } else {
        const bool check = *reinterpret_cast<const unsigned int*>(packed + (size_t)RB * KC * kBlock) != 0;
        const int row = (warp & 3) * 32 + lane;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        bool waited = false;
        for (int i = warp >> 2; i < steps; i += A4S_GROUPS) {
            const int s = i % C::kSP, a = i % C::kSA;
            if (i >= C::kSA && !waited) {
                skinny_pdl_wait();
                waited = true;
            }
            mbar_wait(pfull(s), (uint32_t)(i / C::kSP) & 1u, status, TC_ERR_FULL_WAIT);
            mbar_wait(aempty(a), ((uint32_t)(i / C::kSA) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
            tc_fence_after();
            const uint32_t stage = smem_base + C::kPOff + s * kPStage;
            if (check) a4s_expand<GS, true>(stage, row, a_col(a) + lanes);
            else a4s_expand<GS, false>(stage, row, a_col(a) + lanes);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(full(a));
                mbar_arrive(pempty(s));
            }
        }
        skinny_pdl_wait();                             // y may still be read by a preceding kernel
        mbar_wait(accf, 0, status, TC_ERR_ACC_FULL);
    }
    __syncwarp();
    const float factor = (*reinterpret_cast<const unsigned int*>(packed + (size_t)RB * KC * kBlock) != 0) ? 1.0f : AFF_SCALED_FACTOR;
    skinny_pdl_wait();
    const uint32_t sums = over_rings ? 0 : kSumOff;
    auto finish = [&](auto put) {
        skinny_finish<A4S_DQ_WARPS, true>(tmem, smem_base + sums, reinterpret_cast<const float*>(smem_gen + sums), over_rings != 0, rbar, M, split, rank,
                                          tile * SKINNY_ROWS, N, status, put);
    };
    if (out == GEMV_OUT_BF16 && !bias && scale == 1.0f) {          // (the common case without the others' branches)
        finish([&](int m, int n, float a, float b) {
            uint16_t* at = y + (size_t)m * N + n;
            at[0] = __bfloat16_as_ushort(__float2bfloat16_rn(a * factor));
            if (n + 8 < N) at[8] = __bfloat16_as_ushort(__float2bfloat16_rn(b * factor));
        });
    } else if (out == GEMV_OUT_SILU_PAIRS) {                       // n: a gate's channel, n + 8 its up's
        finish([&](int m, int n, float a, float b) {
            const float g = __bfloat162float(__float2bfloat16_rn(a * factor)), u = __bfloat162float(__float2bfloat16_rn(b * factor));
            y[(size_t)m * (N >> 1) + (n >> 4) * 8 + (n & 7)] = __bfloat16_as_ushort(__float2bfloat16_rn(__fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u)));
        });
    } else {
        finish([&](int m, int n, float a, float b) {
            float v[2] = {a * factor, b * factor};
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int c = n + 8 * j;
                if (c >= N) break;
                const size_t at = (size_t)m * N + c;
                if (bias) v[j] += __uint_as_float(uint32_t(bias[c]) << 16);
                if (scale != 1.0f) v[j] *= scale;
                if (out == GEMV_OUT_F32) {
                    reinterpret_cast<float*>(y)[at] = v[j];
                    continue;
                }
                __nv_bfloat16 o = __float2bfloat16_rn(v[j]);
                if (out == GEMV_OUT_RESIDUAL_ADD) o = __float2bfloat16_rn(__fadd_rn(__uint_as_float(uint32_t(y[at]) << 16), __bfloat162float(o)));
                y[at] = __bfloat16_as_ushort(o);
            }
        });
    }
    __syncthreads();
    if (warp == A4S_DQ_WARPS + 2) {
        tc_fence_after();
        tmem_dealloc(tmem, C::kTmemCols);
    }
}

template <int TN, int GS>
int32_t a4s_launch(scr_ctx* ctx, tc_encode_tiled_fn enc, const CUtensorMap& map, const uint8_t* packed, uint16_t* y, int M, int N, int K, int out, const uint16_t* bias,
                   float scale, cudaStream_t stream) {
    using C = A4SCfg<TN>;
    const AffineGeom g = affine_geom(N, K, 64);          // RB / KC only: the same for every group size
    constexpr size_t smem = C::kPOff + C::kSP * 8u * aff_block_bytes(GS) + 512 + 1024;
    static_assert(C::kPOff + C::kSP * 8u * aff_block_bytes(GS) >= skinny_sum_bytes(TN), "the sums fit the rings");
    CUtensorMap w_map;
    if (!affine_w_map(&w_map, enc, packed, g.RB, g.KC, GS)) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled failed");
    static SkinnyResident resident;
    const int tiles = g.RB / 8;
    const SkinnyPlan p = skinny_plan(resident, affine_b4_skinny_kernel<TN, GS>, ctx->device, ctx->sm_count, tiles, g.KC, A4S_THREADS, smem, TN, 3.0f);
    const cudaError_t e = skinny_launch(affine_b4_skinny_kernel<TN, GS>, tiles, p.split, A4S_THREADS, p.smem, stream, map, w_map, packed, y, M, N, g.RB, g.KC, p.split,
                                        p.over_rings, out, bias, scale, ctx->dev_status);
    if (e != cudaSuccess) return scr_fail(ctx, SCR_E_CUDA, "affine_b4_skinny: %s", cudaGetErrorString(e));
    return scr_check_launch(ctx, "affine_b4_skinny");
}

}  // namespace

// Whether the GEMM for few tokens takes this call: up to the 128 that one accumulator and four activation stages hold beside the
// weights (beyond, a second token tile would expand every weight a second time).  Its end grows with the tokens, and where k is short that is most
// of a call: 128 tokens of 512 -> 8192 8.5 us against 5.9 on the prompt kernel's tiles, of 1280 -> 4096 10.8 and 8.0, of 1536 -> 6144 10.3
// and 9.9, but of 2048 -> 2048 9.0 and 9.9.  From 65 tokens on a CTA fills its SM, so that a matrix of more tiles than SMs would run whole units one
// after the other; the prompt kernel's tiles overlap (3072 -> 24576: 96 tokens 30.4 and 20.9 us; 64, two CTAs to an SM here, 20.9 and 20.4).
bool affine_b4_skinny_applies(int M, int N, int K, int sms) {
    if (M <= 64) return true;
    return (M <= 96 || (M <= 128 && K > 1536)) && affine_geom(N, K, 64).RB / 8 <= sms;
}

int32_t affine_b4_skinny_launch(scr_ctx* ctx, const uint8_t* packed, const uint16_t* x, uint16_t* y, int M, int N, int K, int gs, int out,
                                const uint16_t* bias, float scale, cudaStream_t stream) {
    tc_encode_tiled_fn enc = tc_tensor_map_encoder();
    if (!enc) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled entry point not available");
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)((M + 15) & ~15)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return scr_fail(ctx, SCR_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
#define A4S_CASE(TN) (gs == 2 ? a4s_launch<TN, 2>(ctx, enc, map, packed, y, M, N, K, out, bias, scale, stream) \
                              : a4s_launch<TN, 1>(ctx, enc, map, packed, y, M, N, K, out, bias, scale, stream))
    if (M <= 16) return A4S_CASE(16);
    if (M <= 32) return A4S_CASE(32);
    if (M <= 64) return A4S_CASE(64);
    return A4S_CASE(128);
#undef A4S_CASE
}
