// fp8-dynamic-per-channel: GEMM for few tokens (up to 256; from how many on, fp8.cu) on tcgen05 tensor cores (kind::f8f6f4), weights as the rows of the MMA
// (skinny.cuh).
//
//   y[m,n] = bf16( (sum_k x_q[m,k] * w_q[n,k]) * a_scale[m] * w_scale[n] (+ bias[n]) )
//
// A unit is 128 channels by one CTA's share of the 128-k tiles; 352 threads:
//   warps 0-7    drain the accumulator, scale and store
//   warp 8       producer of the weights (one bulk copy of a pre-swizzled 16 KB tile per step), load-time constants: it
//                starts before the quantisation of the activations has finished
//   warp 9       producer of the quantised activations, which lie in the same image: the tokens' rows of a k-tile are one
//                contiguous run (rows past the last token hold whatever the pack held; their columns are never stored)
//   warp 10      owns TMEM; one elected lane issues 4 tcgen05.mma (128 x tokens x 32) per step
//
// What bounds it: the copies into shared memory, 16 KB of weights and 128 bytes per token and step.  250 tokens of 18944 -> 3584
// (with the quantisation) 46.4 us on the 128-token tiles of fp8_gemm.cu and their finishing launch, 32.5 us here.
// One token of 18944 -> 3584 15.3 us (22.0 in the matvec, which quantises in a launch of its own there).
#include "fp8.cuh"
#include "skinny.cuh"

namespace {

constexpr int F8S_THREADS = 352;
constexpr uint32_t F8S_W_STAGE = FP8_TILE_BYTES;

template <int TN>
struct F8SCfg {
    static constexpr int kSW = TN == 256 ? 4 : TN == 128 || TN == 16 ? 6 : 5;                 // weight stages
    static constexpr int kSX = TN == 64 ? 3 : kSW;                                // activation stages
    static constexpr uint32_t kXStage = TN * 128u;
    static constexpr uint32_t kXOff = kSW * F8S_W_STAGE;
    static constexpr uint32_t kBarOff = kXOff + kSX * kXStage;
    static constexpr uint32_t kTotal = kBarOff + 256u + 1024u;
    static constexpr int kCtasPerSm = TN >= 128 ? 1 : 2;
    static constexpr uint32_t kTmemCols = TN < 32 ? 32 : TN;
};

template <int TN>
__global__ void __launch_bounds__(F8S_THREADS, F8SCfg<TN>::kCtasPerSm)
fp8_skinny_kernel(const uint8_t* __restrict__ wpack, const float* __restrict__ w_scale, const uint8_t* __restrict__ xq, const float* __restrict__ a_scale,
                  uint16_t* __restrict__ y, int M, int N, int KT, int M_pad, int split, int over_rings, int out_f32, const uint16_t* __restrict__ bias,
                  int* __restrict__ status) {
    using C = F8SCfg<TN>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar = smem_base + C::kBarOff;
    auto wfull = [&](int s) { return bar + 8u * s; };
    auto wempty = [&](int s) { return bar + 8u * (C::kSW + s); };
    auto xfull = [&](int s) { return bar + 8u * (2 * C::kSW + s); };
    auto xempty = [&](int s) { return bar + 8u * (2 * C::kSW + C::kSX + s); };
    constexpr int kSlots = 2 * C::kSW + 2 * C::kSX;
    static_assert(8 * (kSlots + 3) <= 256, "barriers");
    const uint32_t accf = bar + 8u * kSlots, rbar = accf + 8u;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + C::kBarOff + 8 * (kSlots + 2));

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int tile = blockIdx.x / split, rank = blockIdx.x - tile * split;
    int k_lo, k_hi;
    skinny_range(KT, rank, split, k_lo, k_hi);
    const int steps = k_hi - k_lo;
    const uint32_t tokens = (uint32_t)(M + 15) & ~15u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kSW; ++s) { mbar_init(wfull(s), 1); mbar_init(wempty(s), 1); }
        for (int s = 0; s < C::kSX; ++s) { mbar_init(xfull(s), 1); mbar_init(xempty(s), 1); }
        mbar_init(accf, 1);
        skinny_expect(rbar, M, split, rank, over_rings);
        fence_mbar_init();
    }
    if (warp == 10) {
        tmem_alloc(smem_u32((const void*)tmem_slot), C::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (split > 1 && !over_rings) skinny_cluster_arrive();
    skinny_pdl_trigger();                              // not before this CTA has its TMEM: the next kernel's CTAs could take it first

    // Only the weights may be touched before the preceding kernel has finished.  A wait that depends on the activations
    // comes after griddepcontrol.wait, so that its bound does not run against that kernel.
    if (warp == 8) {
        if (lane == 0) {
            for (int i = 0; i < steps; ++i) {
                const int s = i % C::kSW;
                if (i == C::kSW) skinny_pdl_wait();
                mbar_wait(wempty(s), ((uint32_t)(i / C::kSW) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                mbar_arrive_expect_tx(wfull(s), F8S_W_STAGE);
                bulk_g2s(smem_base + s * F8S_W_STAGE, wpack + ((size_t)tile * KT + k_lo + i) * FP8_TILE_BYTES, F8S_W_STAGE, wfull(s));
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            skinny_pdl_wait();
            for (int i = 0; i < steps; ++i) {
                const int s = i % C::kSX;
                mbar_wait(xempty(s), ((uint32_t)(i / C::kSX) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                mbar_arrive_expect_tx(xfull(s), tokens * 128u);
                bulk_g2s(smem_base + C::kXOff + s * C::kXStage, xq + (size_t)(k_lo + i) * ((size_t)M_pad * 128), tokens * 128u, xfull(s));
            }
        }
    } else if (warp == 10) {
        // The warp goes round as a whole, with one lane elected for the instructions alone, so that the descriptors stay in uniform
        // registers: an MMA of few columns is shorter than its issue from a divergent thread.
        skinny_pdl_wait();
        const bool lead = elect_one();
        const uint32_t idesc = umma_idesc(0, 0, SKINNY_ROWS, tokens);
        for (int i = 0; i < steps; ++i) {
            const int sw = i % C::kSW, sx = i % C::kSX;
            const uint64_t adesc = umma_desc_k_sw128(smem_base + sw * F8S_W_STAGE), bdesc = umma_desc_k_sw128(smem_base + C::kXOff + sx * C::kXStage);
            mbar_wait(wfull(sw), (uint32_t)(i / C::kSW) & 1u, status, TC_ERR_FULL_WAIT);
            mbar_wait(xfull(sx), (uint32_t)(i / C::kSX) & 1u, status, TC_ERR_FULL_WAIT);
            tc_fence_after();
            if (lead) {
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) umma_f8f6f4(tmem, adesc + (uint64_t)(2 * k4), bdesc + (uint64_t)(2 * k4), idesc, i > 0 || k4 > 0);
                umma_commit(wempty(sw));
                umma_commit(xempty(sx));
            }
            __syncwarp();
        }
        if (lead) umma_commit(accf);
    } else {
        skinny_pdl_wait();
        mbar_wait(accf, 0, status, TC_ERR_ACC_FULL);
    }
    __syncwarp();
    skinny_pdl_wait();
    const uint32_t sums = over_rings ? 0 : C::kBarOff + 256u;
    skinny_finish<8, true>(tmem, smem_base + sums, reinterpret_cast<const float*>(smem_gen + sums), over_rings != 0, rbar, M, split, rank, tile * SKINNY_ROWS, N, status,
                         [&](int m, int n, float a, float b) {
        const float as = a_scale[m], v[2] = {a, b};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int c = n + 8 * j;
            if (c >= N) break;
            const float r = __fmul_rn(__fmul_rn(v[j], as), __ldg(w_scale + c));
            if (out_f32) {
                reinterpret_cast<float*>(y)[(size_t)m * N + c] = r;
            } else {
                const __nv_bfloat16 o = __float2bfloat16_rn(bias ? r + __uint_as_float(uint32_t(bias[c]) << 16) : r);
                y[(size_t)m * N + c] = *reinterpret_cast<const uint16_t*>(&o);
            }
        }
    });
    __syncthreads();
    if (warp == 10) {
        tc_fence_after();
        tmem_dealloc(tmem, C::kTmemCols);
    }
}

template <int TN>
SkinnyPlan f8s_plan(const scr_ctx* ctx, const Fp8Geom& g) {
    static SkinnyResident resident;
    return skinny_plan(resident, fp8_skinny_kernel<TN>, ctx->device, ctx->sm_count, g.NT, g.KT, F8S_THREADS, F8SCfg<TN>::kTotal, TN, 4.0f);
}

template <int TN>
int32_t f8s_launch(scr_ctx* ctx, const uint8_t* wpack, const uint8_t* act, int rows, uint16_t* y, int M, int N, int K, const LinearEnds& ends,
                   cudaStream_t stream) {
    using C = F8SCfg<TN>;
    static_assert(C::kBarOff >= skinny_sum_bytes(TN), "the sums fit the rings");
    const Fp8Geom g = fp8_geom(N, K);
    const SkinnyPlan p = f8s_plan<TN>(ctx, g);
    const float* w_scale = reinterpret_cast<const float*>(wpack + (size_t)g.NT * g.KT * FP8_TILE_BYTES);
    const cudaError_t e = skinny_launch(fp8_skinny_kernel<TN>, g.NT, p.split, F8S_THREADS, p.smem, stream, wpack, w_scale, act + fp8_act_scale_bytes(M),
                                        reinterpret_cast<const float*>(act), y, M, N, g.KT, rows, p.split, p.over_rings, ends.out_f32,
                                        ends.bias, ctx->dev_status);
    if (e != cudaSuccess) return scr_fail(ctx, SCR_E_CUDA, "fp8_skinny: %s", cudaGetErrorString(e));
    return scr_check_launch(ctx, "fp8_skinny");
}

}  // namespace

// About what a call of 65 to 256 tokens takes here, in us: a k-tile of a unit 0.40 and 0.0006 a token, and start and end of a launch 2.3 and
// 0.0335 a token (fitted to streams of calls: 3584 x 18944 at 256 tokens 27.4, 3584 x 3584 15.3, 8192 x 1024 15.2, 512 x 512 11.2).
float fp8_skinny_us(const scr_ctx* ctx, int M, int N, int K) {
    const Fp8Geom g = fp8_geom(N, K);
    const int split = M <= 128 ? f8s_plan<128>(ctx, g).split : f8s_plan<256>(ctx, g).split;
    const int rounds = scr_ceil_div(g.NT * split, ctx->sm_count);
    return 2.3f + 0.0335f * M + (float)(rounds * scr_ceil_div(g.KT, split)) * (0.40f + 0.0006f * M);
}

int32_t fp8_skinny_launch(scr_ctx* ctx, const uint8_t* wpack, const uint8_t* act, uint16_t* y, int M, int N, int K, const LinearEnds& ends,
                          cudaStream_t stream) {
    const int rows = scr_ceil_div(M, FP8_TILE) * FP8_TILE;
    if (M <= 32) return f8s_launch<32>(ctx, wpack, act, rows, y, M, N, K, ends, stream);
    if (M <= 64) return f8s_launch<64>(ctx, wpack, act, rows, y, M, N, K, ends, stream);
    if (M <= 128) return f8s_launch<128>(ctx, wpack, act, rows, y, M, N, K, ends, stream);
    return f8s_launch<256>(ctx, wpack, act, rows, y, M, N, K, ends, stream);
}

// Up to 16 tokens, whose pack (`rows` = FP8_FEW_ROWS of a k-tile) only `scr_linear_fp8_dynamic` makes, for itself.
bool fp8_skinny16_even(scr_ctx* ctx, int N, int K) {
    const Fp8Geom g = fp8_geom(N, K);
    const float share = (float)g.NT * g.KT / ctx->sm_count;
    const int rounds = (g.NT + ctx->sm_count - 1) / ctx->sm_count;
    return f8s_plan<16>(ctx, g).units <= 1.6f * share && 20 * g.NT < 19 * rounds * ctx->sm_count;
}

int32_t fp8_skinny16_launch(scr_ctx* ctx, const uint8_t* wpack, const uint8_t* act, uint16_t* y, int M, int N, int K, const LinearEnds& ends,
                            cudaStream_t stream) {
    return f8s_launch<16>(ctx, wpack, act, FP8_FEW_ROWS, y, M, N, K, ends, stream);
}
