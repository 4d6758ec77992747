// bf16 GEMM for few rows of x on tcgen05 tensor cores, the weights as the rows of the MMA (skinny.cuh), with the ends of
// `scr_dense` applied to the finished sums.
//
// A unit is 128 rows of W by one CTA's share of the 64-wide k slices; 352 threads:
//   warps 0-7    drain the accumulator and store
//   warp 8       producer of the weights (one tiled TMA load of 128 rows x 64 k per slice, 128-byte swizzle), load-time
//                constants: it starts before the preceding kernel of the stream has finished, and ahead of this kernel's own setting up
//   warp 9       producer of x (one tiled TMA load per slice, zeros outside)
//   warp 10      owns TMEM; one elected lane issues 4 tcgen05.mma (128 x rows of x x 16) per slice
//
// What bounds it: the weights from HBM; for the small linears the start and end of a launch.  10240 x 3072 (63 MB) at 32 rows
// 14.9 us (4.2 TB/s), 3072 x 8192 11.9 us (13.3 with two CTAs to an SM and cluster barriers, 12.3 with the first weights after the setting up), 128256 x 3072 at 8 rows 120 us (6.5 TB/s), in streams of calls.  Against the 128-row tile of dense_gemm.cu and its finishing launch: a decode step of the 3B Vumipel at 32 sequences
// 4.22 -> 3.59 ms, with that issue 3.31 -> 3.09 ms.
#include "seq_common.cuh"
#include "skinny.cuh"

namespace {

constexpr int DS_THREADS = 352;
constexpr uint32_t DS_W_STAGE = SKINNY_ROWS * 128u;          // 128 rows x 64 bf16

template <int TN>
struct DsCfg {
    static constexpr int kSW = TN == 128 ? 8 : TN == 16 ? 6 : 5;                  // weight stages
    static constexpr int kSX = TN == 128 ? 4 : TN == 64 ? 3 : kSW;                // x stages
    static constexpr uint32_t kXStage = TN * 128u;
    static constexpr uint32_t kXOff = kSW * DS_W_STAGE;
    static constexpr uint32_t kBarOff = kXOff + kSX * kXStage;
    static constexpr uint32_t kTotal = kBarOff + 256u + 1024u;
    static constexpr uint32_t kTmemCols = TN < 32 ? 32 : TN;
    static constexpr int kCtasPerSm = TN == 128 ? 1 : 2;
};

template <int TN, DenseEnd END>
__global__ void __launch_bounds__(DS_THREADS, DsCfg<TN>::kCtasPerSm)
dense_skinny_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, int M, int N, int KT, int NT, int split,
                    int over_rings, int w_fresh, DenseEnds ends, int* __restrict__ status) {
    using C = DsCfg<TN>;
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
    const int g = tile / NT, n0 = (tile - g * NT) * SKINNY_ROWS;
    int k_lo, k_hi;
    skinny_range(KT, rank, split, k_lo, k_hi);
    const int steps = k_hi - k_lo;

    // The first weights are on their way before anything else is set up (unless another kernel writes them): their copy needs only its own
    // barriers.
    auto load = [&](int i) {
        const int s = i % C::kSW;
        mbar_arrive_expect_tx(wfull(s), DS_W_STAGE);
        tma_load_3d(smem_base + s * DS_W_STAGE, &w_map, (k_lo + i) * 64, n0, g, wfull(s));
    };
    const int early = w_fresh ? 0 : min(steps, 2);
    if (warp == 8) {
        if (lane == 0) {
            for (int s = 0; s < C::kSW; ++s) { mbar_init(wfull(s), 1); mbar_init(wempty(s), 1); }
            fence_mbar_init();
            for (int i = 0; i < early; ++i) load(i);
        }
        __syncwarp();
    } else if (warp == 9) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
            for (int s = 0; s < C::kSX; ++s) { mbar_init(xfull(s), 1); mbar_init(xempty(s), 1); }
            mbar_init(accf, 1);
            skinny_expect(rbar, M, split, rank, over_rings);
            fence_mbar_init();
        }
        __syncwarp();
    } else if (warp == 10) {
        tmem_alloc(smem_u32((const void*)tmem_slot), C::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (split > 1 && !over_rings) skinny_cluster_arrive();
    pdl_trigger();                                     // not before this CTA has its TMEM: the next kernel's CTAs could take it first

    // Only the weights may be touched before the preceding kernel has finished.  A wait that depends on x comes after
    // griddepcontrol.wait, so that its bound does not run against that kernel.
    if (warp == 8) {
        if (lane == 0) {
            if (w_fresh) pdl_wait();
            for (int i = early; i < steps; ++i) {
                if (i == C::kSW) pdl_wait();
                mbar_wait(wempty(i % C::kSW), ((uint32_t)(i / C::kSW) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                load(i);
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            pdl_wait();
            const uint32_t rows = (uint32_t)(M + 15) & ~15u;
            for (int i = 0; i < steps; ++i) {
                const int s = i % C::kSX;
                mbar_wait(xempty(s), ((uint32_t)(i / C::kSX) & 1u) ^ 1u, status, TC_ERR_EMPTY_WAIT);
                mbar_arrive_expect_tx(xfull(s), rows * 128u);
                tma_load_3d(smem_base + C::kXOff + s * C::kXStage, &x_map, (k_lo + i) * 64, g, 0, xfull(s));
            }
        }
    } else if (warp == 10) {
        // The warp goes round as a whole, with one lane elected for the instructions alone, so that the descriptors stay in uniform
        // registers: an MMA of few columns is shorter than its issue from a divergent thread.
        pdl_wait();
        const bool lead = elect_one();
        const uint32_t idesc = umma_idesc(1, 1, SKINNY_ROWS, (uint32_t)(M + 15) & ~15u);
        for (int i = 0; i < steps; ++i) {
            const int sw = i % C::kSW, sx = i % C::kSX;
            const uint64_t adesc = umma_desc_k_sw128(smem_base + sw * DS_W_STAGE), bdesc = umma_desc_k_sw128(smem_base + C::kXOff + sx * C::kXStage);
            mbar_wait(wfull(sw), (uint32_t)(i / C::kSW) & 1u, status, TC_ERR_FULL_WAIT);
            mbar_wait(xfull(sx), (uint32_t)(i / C::kSX) & 1u, status, TC_ERR_FULL_WAIT);
            tc_fence_after();
            if (lead) {
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) umma_f16(tmem, adesc + (uint64_t)(2 * k4), bdesc + (uint64_t)(2 * k4), idesc, i > 0 || k4 > 0);
                umma_commit(wempty(sw));
                umma_commit(xempty(sx));
            }
            __syncwarp();
        }
        if (lead) umma_commit(accf);
    } else {
        pdl_wait();
        mbar_wait(accf, 0, status, TC_ERR_ACC_FULL);
    }
    __syncwarp();
    pdl_wait();
    const uint32_t sums = over_rings ? 0 : C::kBarOff + 256u;
    skinny_finish<8, (TN <= 64)>(tmem, smem_base + sums, reinterpret_cast<const float*>(smem_gen + sums), over_rings != 0, rbar, M, split, rank, n0, N, status,
                  [&](int m, int n, float a, float b) { dense_put_two<bf16, END>(ends, m, g, n, N, a, b); });
    __syncthreads();
    if (warp == 10) {
        tc_fence_after();
        tmem_dealloc(tmem, C::kTmemCols);
    }
}

template <int TN, DenseEnd END>
int32_t ds_launch(scr_ctx* ctx, const scr_dense& d, const CUtensorMap& x_map, const CUtensorMap& w_map, cudaStream_t stream) {
    using C = DsCfg<TN>;
    static_assert(C::kBarOff >= skinny_sum_bytes(TN), "the sums fit the rings");
    const int nt = scr_ceil_div(d.N, SKINNY_ROWS), kt = scr_ceil_div(d.K, 64);
    static SkinnyResident resident;
    const SkinnyPlan p = skinny_plan(resident, dense_skinny_kernel<TN, END>, ctx->device, ctx->sm_count, nt * d.groups, kt, DS_THREADS, C::kTotal, TN, 4.0f);
    const cudaError_t e = skinny_launch(dense_skinny_kernel<TN, END>, nt * d.groups, p.split, DS_THREADS, p.smem, stream, x_map, w_map, d.M, d.N, kt, nt,
                                        p.split, p.over_rings, (int)(d.w_fresh != 0), dense_ends(d), ctx->dev_status);
    if (e != cudaSuccess) return scr_fail(ctx, SCR_E_CUDA, "dense_skinny: %s", cudaGetErrorString(e));
    return scr_check_launch(ctx, "dense_skinny");
}

template <DenseEnd END>
int32_t ds_launch_rows(scr_ctx* ctx, const scr_dense& d, const CUtensorMap& x_map, const CUtensorMap& w_map, cudaStream_t stream) {
    if (d.M <= 16) return ds_launch<16, END>(ctx, d, x_map, w_map, stream);
    if (d.M <= 32) return ds_launch<32, END>(ctx, d, x_map, w_map, stream);
    if (d.M <= 64) return ds_launch<64, END>(ctx, d, x_map, w_map, stream);
    return ds_launch<128, END>(ctx, d, x_map, w_map, stream);
}

}  // namespace

// Whether the GEMM for few rows takes this call (up to 128 rows of x, what one accumulator holds), or the tiles of 128 rows by up to 256
// columns of dense_gemm.cu.  Those read x once for two of this kernel's tiles and pay for 128 rows whatever there are: they are ahead
// where W is wide enough that they need no cut of k, and its long ends count where k is short.  Streams of calls, us, few rows / tiles:
//   3072 -> 16384, 33 rows 24.1 / 20.5, 64 27.6 / 20.5, 128 30.7 / 21.4;  3072 -> 128256, 64 rows 154 / 134, 128 220 / 140
//   2048 -> 12288, 33 rows 14.8 / 12.3;  3072 -> 10240, 64 rows 16.7 / 16.6, 65 21.8 / 16.5;  3072 -> 8192, 65 rows 14.2 / 15.4
//   512 -> 3072, 64 rows 6.0 / 5.5, 128 8.0 / 6.5;  3072 -> 3072, 128 rows 11.1 / 13.7;  8192 -> 8192, 128 rows 35.0 / 40.0
// Up to 32 rows, a decode batch, the two are close (3072 -> 16384, 32 rows 22.9 / 20.3, 20 rows 22.2 / 28.2), and only this kernel
// fetches W while the norm before it runs: with the tiles a decode step of the 3B Vumipel at 32 sequences took 3.23 ms, here 3.09.
bool dense_skinny_applies(int M, int N, int K, int groups) {
    const long long tiles = (long long)scr_ceil_div(N, SKINNY_ROWS) * groups;
    if (M <= 16) return true;
    if (M > 128) return false;
    return M <= 32 || (tiles < 96 && (M <= 64 || (tiles < 80 && K > 512)));
}

int32_t dense_skinny_launch(scr_ctx* ctx, const scr_dense& d, cudaStream_t stream) {
    CUtensorMap x_map, w_map;
    const uint64_t xg = d.groups > 1 ? (uint64_t)d.x_group * 2 : (uint64_t)d.K * 2;
    const uint64_t row = (uint64_t)(d.M > 1 ? d.ldx : d.K) * 2;          // (a single row has no use for its stride)
    if (!dense_tensor_map(&x_map, d.x, d.K, d.groups, d.M, xg, row, 1, (d.M + 15) & ~15) ||
        !dense_tensor_map(&w_map, d.w, d.K, d.N, d.groups, (uint64_t)d.K * 2, (uint64_t)d.N * d.K * 2, SKINNY_ROWS, 1))
        return scr_fail(ctx, SCR_E_CUDA, "dense_skinny: tensor map (M %d N %d K %d groups %d)", d.M, d.N, d.K, d.groups);
    switch (dense_end(d)) {
        case END_PARTS: return ds_launch_rows<END_PARTS>(ctx, d, x_map, w_map, stream);
        case END_RESIDUAL: return ds_launch_rows<END_RESIDUAL>(ctx, d, x_map, w_map, stream);
        default: return ds_launch_rows<END_OWN>(ctx, d, x_map, w_map, stream);
    }
}
