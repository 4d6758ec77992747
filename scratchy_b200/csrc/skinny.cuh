// What the GEMMs for few tokens share (affine_b4_skinny.cu, fp8_skinny.cu, dense_skinny.cu): a decode batch, drafted tokens
// to verify, the rest of a prompt.  The roles of the operands are swapped against the prefill GEMMs: the 128 ROWS of the MMA
// are 128 output channels (the weights, which bound such a call) and its columns are the tokens, so a few tokens cost a
// few columns instead of a 128-row tile of padding.  A tile's k extent is shared by a cluster of up to 8 CTAs, one work
// unit each, whose sums meet through distributed shared memory in rank order: no workspace, no second kernel.
#pragma once

#include <atomic>

#include "tc_common.cuh"

constexpr int SKINNY_ROWS = 128;                 // output channels of a tile
constexpr int SKINNY_MAX_SPLIT = 8;              // portable cluster size
constexpr int SKINNY_EPI_WARPS = 8;              // warps 0..7 drain the accumulator

__device__ __forceinline__ void skinny_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void skinny_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void skinny_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}

// The k steps of unit `rank` of `split`: even shares, none empty while split <= steps.
__device__ __forceinline__ void skinny_range(int steps, int rank, int split, int& lo, int& hi) {
    lo = (int)((long long)steps * rank / split);
    hi = (int)((long long)steps * (rank + 1) / split);
}

// Shared memory the sums of a cluster need (they reuse the rings of the main loop): split x per tokens x 128 channels.
__host__ __device__ constexpr size_t skinny_sum_bytes(int tokens) { return (size_t)(tokens + 4 * SKINNY_MAX_SPLIT) * SKINNY_ROWS * 4; }

// The end of a unit, called by every thread of every CTA of the cluster once its role is done; warps 0..7 have seen the
// accumulator complete, so nothing reads or fills this CTA's rings any more.  `d` = the accumulator (lane = channel, column =
// token), `sums` = the start of the rings (shared and generic address).  The tokens are dealt to the cluster's CTAs in runs
// of a multiple of 4 (they travel 16 bytes at a time): a CTA sends every run to its owner, which adds the `split` sums of a value in rank order and passes the channels n and
// n + 8 (n % 16 < 8: a gate and its up, where they are interleaved) to put(token, n, sum, sum8).
template <typename Put>
__device__ __forceinline__ void skinny_finish(uint32_t d, uint32_t sums, const float* sums_gen, int M, int split, int rank, int n0, int N, Put put) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = ((M + split - 1) / split + 3) & ~3;
    if (split > 1) skinny_cluster_sync();
    else __syncthreads();
    if (warp < SKINNY_EPI_WARPS) {
        tc_fence_after();
        const int row = (warp & 3) * 32 + lane;
        for (int c = (warp >> 2) * 16; c < M; c += 32) {
            uint32_t r[16];
            tmem_ld_32x16(d + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, r);
            tmem_ld_wait();
            // [sender][4 tokens][channel][token of the 4]
            int owner = c / per, at = c - owner * per;
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                if (c + j < M) {
                    uint32_t dst = sums + (uint32_t)(((rank * per + at) >> 2) * SKINNY_ROWS + row) * 16u;
                    if (split > 1) asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(dst) : "r"(owner));
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3]) : "memory");
                }
                at += 4;
                if (at == per) { at = 0; ++owner; }
            }
        }
        tc_fence_before();
    }
    if (split > 1) skinny_cluster_sync();
    else __syncthreads();
    const int mine = min(per, M - rank * per);
    for (int i = threadIdx.x; i < mine * (SKINNY_ROWS / 2); i += blockDim.x) {
        const int t = i >> 6, p = i & 63, ch = (p >> 3) * 16 + (p & 7);
        if (n0 + ch >= N) continue;
        const float* part = sums_gen + ((size_t)(t >> 2) * SKINNY_ROWS + ch) * 4 + (t & 3);
        float a[SKINNY_MAX_SPLIT], b[SKINNY_MAX_SPLIT];
#pragma unroll
        for (int k = 0; k < SKINNY_MAX_SPLIT; ++k) {
            a[k] = k < split ? part[(size_t)k * per * SKINNY_ROWS] : 0.0f;
            b[k] = k < split ? part[(size_t)k * per * SKINNY_ROWS + 32] : 0.0f;
        }
#pragma unroll
        for (int k = 1; k < SKINNY_MAX_SPLIT; ++k)
            if (k < split) {
                a[0] += a[k];
                b[0] += b[k];
            }
        put(rank * per + t, n0 + ch, a[0], b[0]);
    }
}

// How many clusters of `split` CTAs of a kernel run at once (a cluster needs its SMs in one GPC, so 148 SMs hold fewer clusters of
// 5 or 6 CTAs than 148 / 6): asked once per kernel, device and size.
constexpr int SKINNY_DEVICES = 64;
struct SkinnyResident {
    std::atomic<int> clusters[SKINNY_DEVICES][SKINNY_MAX_SPLIT + 1];
};
template <typename... KArgs>
static inline int skinny_resident(SkinnyResident& cache, void (*kernel)(KArgs...), int device, int sms, int split, int threads, size_t smem) {
    const bool known = device >= 0 && device < SKINNY_DEVICES;
    int n = known ? cache.clusters[device][split].load(std::memory_order_relaxed) : 0;
    if (n > 0) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sms * split));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
        (void)cudaGetLastError();
        n = sms / split > 0 ? sms / split : 1;
    }
    if (known) cache.clusters[device][split].store(n, std::memory_order_relaxed);
    return n;
}

// CTAs that share a tile's k extent.  A call is rounds of the clusters that run at once; a round lasts as long as a unit, whose
// k steps share the SM with those of the units beside it and which costs `unit_cost` steps beside them.  (Without the rounds
// in the account 24 tiles at 128 tokens were cut six ways, 22 of which run at once: 3072 x 3072 int4 took 19.0 us, now 11.1.)
template <typename... KArgs>
static inline int skinny_split(SkinnyResident& cache, void (*kernel)(KArgs...), int device, int sms, int tiles, int steps, int threads, size_t smem,
                               float unit_cost) {
    int best = 1;
    float least = 1e30f;
    for (int s = 1; s <= SKINNY_MAX_SPLIT && s <= steps; ++s) {
        const int resident = skinny_resident(cache, kernel, device, sms, s, threads, smem), at_once = tiles < resident ? tiles : resident;
        const int rounds = (tiles + resident - 1) / resident, beside = (at_once * s + sms - 1) / sms;
        const float t = (float)rounds * ((float)(beside * ((steps + s - 1) / s)) + unit_cost);
        if (t < least * 0.999f) {
            least = t;
            best = s;
        }
    }
    return best;
}

// One launch of `split`-CTA clusters, overlapping its start with the kernel before it.
template <typename... KArgs, typename... Args>
static inline cudaError_t skinny_launch(void (*kernel)(KArgs...), int tiles, int split, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * split));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = split > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
