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

__device__ __forceinline__ void skinny_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void skinny_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void skinny_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same in two parts: after a CTA's barriers are initialised, and before it touches another CTA's.
__device__ __forceinline__ void skinny_cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void skinny_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
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

// Shared memory the sums of a cluster need (after the rings of the main loop, or over them): split x per tokens x 128 channels.
__host__ __device__ constexpr size_t skinny_sum_bytes(int tokens) { return (size_t)(tokens + 4 * SKINNY_MAX_SPLIT) * SKINNY_ROWS * 4; }

// The tokens are dealt to the cluster's CTAs in runs of a multiple of 4.
__device__ __forceinline__ int skinny_run(int M, int split) { return ((M + split - 1) / split + 3) & ~3; }

// The start of a unit, for thread 0 beside the other barriers: `rbar` completes when the cluster's sums of this CTA's run are here.
__device__ __forceinline__ void skinny_expect(uint32_t rbar, int M, int split, int rank, int over_rings) {
    const int per = skinny_run(M, split), mine = min(per, M - rank * per);
    mbar_init(rbar, 1);
    if (split > 1 && !over_rings && mine > 0) mbar_arrive_expect_tx(rbar, (uint32_t)(split * ((mine + 3) & ~3) * SKINNY_ROWS * 4));
}
// The wait for the sums.  It is bounded by its count alone: every CTA of the cluster sends its sums whatever became of its own waits, and
// none may leave while they are on their way to it.
__device__ __forceinline__ void skinny_wait_sums(uint32_t rbar, int* status) {
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(rbar) : "memory");
        if (ok) return;
    }
    atomicCAS(status, 0, TC_ERR_ACC_FULL);
}

// The end of a unit, called by every thread of every CTA of the cluster once its role is done; warps 0 .. EPI_WARPS - 1 have
// seen the accumulator complete.  `d` = the accumulator (lane = channel, column = token), `sums` = where the cluster's sums go (shared and generic
// address).  A CTA sends every run to its owner, which adds the `split` sums of a value in rank order and passes the channels n and n + 8
// (n % 16 < 8: a gate and its up, where they are interleaved) to put(token, n, sum, sum8).
// Where the sums have memory of their own they travel by asynchronous stores that count on the owner's `rbar`: no barrier of the cluster in the
// end of a unit.  (With one before the stores and one after, 45 tokens of 8192 -> 3072 spent 3.3 of 10 us there.)  Those need a launch with
// clusters, an illegal instruction otherwise.  Else (`over_rings`) the sums lie over the rings, which every CTA must be done with first, and
// plain stores are ahead for their many tokens (250 fp8 tokens of 3584 -> 3584: 17.5 us, 19.0 with asynchronous ones).
// From SKINNY_QUAD_TOKENS on a run has work for every thread four tokens at a time (QUADS; 250 fp8 tokens of 18944 -> 3584 31.4 -> 29.8 us, but the
// bf16 linears of 65 to 128 rows, whose put is longer, lost 2 to 8 %).
constexpr int SKINNY_QUAD_TOKENS = 12;
template <int EPI_WARPS, bool QUADS, typename Put>
__device__ __forceinline__ void skinny_finish(uint32_t d, uint32_t sums, const float* sums_gen, bool over_rings, uint32_t rbar, int M, int split, int rank,
                                              int n0, int N, int* status, Put put) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per = skinny_run(M, split), mine = min(per, M - rank * per);
    const bool async = split > 1 && !over_rings;
    if (async) skinny_cluster_wait();            // the others' barriers are set up (they arrived when theirs were)
    else if (split > 1) skinny_cluster_sync();
    if (warp < EPI_WARPS) {
        tc_fence_after();
        const int row = (warp & 3) * 32 + lane;
        // [sender][4 tokens][channel][token of the 4]
        int owner = 0, at = (warp >> 2) * 16;
        while (at >= per) { at -= per; ++owner; }
        for (int c = (warp >> 2) * 16; c < M; c += EPI_WARPS * 4) {
            uint32_t r[16], dst[4], bar[4];
            tmem_ld_32x16(d + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, r);
            int o = owner, t = at;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t local = sums + (uint32_t)(((rank * per + t) >> 2) * SKINNY_ROWS + row) * 16u;
                const int to = o < split ? o : rank;
                dst[j] = local;
                if (split > 1) {
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst[j]) : "r"(local), "r"(to));
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar[j]) : "r"(rbar), "r"(to));
                }
                t += 4;
                if (t == per) { t = 0; ++o; }
            }
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (c + 4 * j >= M) continue;
                if (async)
                    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
                                 ::"r"(dst[j]), "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3]), "r"(bar[j]) : "memory");
                else
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst[j]), "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3]) : "memory");
            }
            at += EPI_WARPS * 4;
            while (at >= per) { at -= per; ++owner; }
        }
        tc_fence_before();
    }
    if (split == 1) __syncthreads();
    else if (!async) skinny_cluster_sync();
    if (mine <= 0) return;
    if (async) skinny_wait_sums(rbar, status);
    if (QUADS && mine >= SKINNY_QUAD_TOKENS) {   // the 4 tokens that lie together, one 16-byte load for each sum of them
        for (int i = threadIdx.x; i < ((mine + 3) >> 2) * (SKINNY_ROWS / 2); i += blockDim.x) {
            const int p = i & 63, ch = (p >> 3) * 16 + (p & 7);
            if (n0 + ch >= N) continue;
            const float4* part = reinterpret_cast<const float4*>(sums_gen) + (i >> 6) * SKINNY_ROWS + ch;
            float4 a = part[0], b = part[8];
            for (int k = 1; k < split; ++k) {
                part += (per >> 2) * SKINNY_ROWS;
                const float4 c = part[0], e = part[8];
                a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
                b.x += e.x; b.y += e.y; b.z += e.z; b.w += e.w;
            }
            const int t = rank * per + 4 * (i >> 6);
            put(t, n0 + ch, a.x, b.x);
            if (t + 1 < M) put(t + 1, n0 + ch, a.y, b.y);
            if (t + 2 < M) put(t + 2, n0 + ch, a.z, b.z);
            if (t + 3 < M) put(t + 3, n0 + ch, a.w, b.w);
        }
        return;
    }
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
// 5 or 6 CTAs than 148 / 6): asked once per kernel, device, size and whether a CTA has its SM to itself.
constexpr int SKINNY_DEVICES = 64;
struct SkinnyResident {
    std::atomic<int> clusters[SKINNY_DEVICES][2][SKINNY_MAX_SPLIT + 1];
};
template <typename... KArgs>
static inline int skinny_resident(SkinnyResident& cache, void (*kernel)(KArgs...), int device, int sms, int split, bool alone, int threads, size_t smem) {
    const bool known = device >= 0 && device < SKINNY_DEVICES;
    int n = known ? cache.clusters[device][alone][split].load(std::memory_order_relaxed) : 0;
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
    if (scr_smem_limit((const void*)kernel, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
        (void)cudaGetLastError();
        n = sms / split > 0 ? sms / split : 1;
    }
    if (known) cache.clusters[device][alone][split].store(n, std::memory_order_relaxed);
    return n;
}

// How a call is launched: CTAs that share a tile's k extent, shared memory, and whether the sums lie over the rings.
struct SkinnyPlan {
    int split;
    size_t smem;
    int over_rings;
    float units;                                 // k steps that an SM works through, and `unit_cost` for each of its units
};
constexpr size_t SKINNY_ALONE = 118 * 1024;      // dynamic shared memory that leaves no room for a second CTA on the SM

// `rings` = the kernel's shared memory without the sums of `tokens` tokens.  A call whose clusters all run at once has each CTA alone on its
// SM: with two to an SM the launch's own CTAs met on some SMs while others had none, because those of the launch before still sat there
// (of 128 CTAs of 3072 -> 16384 at 32 tokens half were done after 8.6 us and the last after 12.2).  Otherwise it is rounds of the clusters that run
// at once; a round lasts as long as a unit, whose k steps share the SM with those of the units beside it and which costs `unit_cost` steps
// beside them.
template <typename... KArgs>
static inline SkinnyPlan skinny_plan(SkinnyResident& cache, void (*kernel)(KArgs...), int device, int sms, int tiles, int steps, int threads, size_t rings,
                                     int tokens, float unit_cost) {
    const size_t sums = skinny_sum_bytes(tokens);
    const bool own = rings + sums <= 227 * 1024;
    const size_t alone_smem = own ? (rings + sums > SKINNY_ALONE ? rings + sums : SKINNY_ALONE) : rings;
    SkinnyPlan best{1, rings, 1, 0.0f};
    float least = 1e30f;
    for (int s = 1; s <= SKINNY_MAX_SPLIT && s <= steps; ++s) {
        if (tiles <= skinny_resident(cache, kernel, device, sms, s, true, threads, alone_smem)) {
            const float t = (float)((steps + s - 1) / s) + unit_cost;
            if (t < least * 0.999f) {
                least = t;
                best = {s, alone_smem, !own, t};
            }
            continue;
        }
        const int resident = skinny_resident(cache, kernel, device, sms, s, false, threads, rings), at_once = tiles < resident ? tiles : resident;
        const int rounds = (tiles + resident - 1) / resident, beside = (at_once * s + sms - 1) / sms;
        const float t = (float)rounds * ((float)(beside * ((steps + s - 1) / s)) + unit_cost);
        if (t < least * 0.999f) {
            least = t;
            best = {s, rings, 1, t};
        }
    }
    return best;
}

// One launch of `split`-CTA clusters, overlapping its start with the kernel before it.
template <typename... KArgs, typename... Args>
static inline cudaError_t skinny_launch(void (*kernel)(KArgs...), int tiles, int split, int threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaError_t e = scr_smem_limit((const void*)kernel, smem);
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
