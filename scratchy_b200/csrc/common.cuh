// Shared host/device helpers for the sm_100a quantized-linear library.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>
#include <atomic>

#include "../../include/scratchy_cuda.h"

// What a forward call asks of a linear's epilogue, passed down as an argument (never parked in the context: a
// context may serve two streams).
struct LinearEnds {
    int out_f32 = 0;                         // unrounded f32 partial sums instead of bf16 (row-parallel linears)
    const uint16_t* bias = nullptr;          // the linear's own bias [N] (bf16), added in f32 before the one rounding
};

struct scr_ctx {
    int device = 0;
    int sm_count = 0;
    int cc_major = 0, cc_minor = 0;
    std::atomic<long long> launches{0};
    int* dev_status = nullptr;      // device word: first bounded wait that ran out (0 = none)
    char err[256] = {0};
};

static inline int32_t scr_fail(scr_ctx* ctx, int32_t code, const char* fmt, ...) {
    if (ctx) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(ctx->err, sizeof(ctx->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

// Checks the launch that was just issued (configuration errors surface here; execution
// errors surface at the caller's next synchronisation).
static inline int32_t scr_check_launch(scr_ctx* ctx, const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return scr_fail(ctx, SCR_E_CUDA, "%s: %s", what, cudaGetErrorString(e));
    if (ctx) ctx->launches.fetch_add(1, std::memory_order_relaxed);
    return SCR_OK;
}

static inline bool scr_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

#define SCR_REQUIRE_CTX(ctx) do { if (!(ctx)) return SCR_E_ARG; (ctx)->err[0] = 0; } while (0)

static inline int scr_ceil_div(int a, int b) { return (a + b - 1) / b; }

// Lets `kernel` be launched with `bytes` of dynamic shared memory.  The limit is a property of the kernel on the device, which all host threads share:
// it is always set to all that a CTA can have beside the kernel's static arrays, so that no thread lowers it between another's setting and
// launch.  (Those arrays' size is asked for once; the limit itself is set on every call, since a reset of the device takes it back.)
constexpr int SCR_SMEM_BLOCK = 227 * 1024;
static inline cudaError_t scr_smem_limit(const void* kernel, size_t bytes) {
    static std::atomic<const void*> kernels[256];
    static std::atomic<int> rooms[256];
    int room = 0;
    size_t at = (reinterpret_cast<uintptr_t>(kernel) >> 4) % 256, tries = 0;
    for (; tries < 256; ++tries, at = (at + 1) % 256) {
        const void* there = kernels[at].load(std::memory_order_acquire);
        if (there == kernel) room = rooms[at].load(std::memory_order_acquire);
        if (!there || there == kernel) break;
    }
    if (room == 0) {
        cudaFuncAttributes a;
        const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
        if (e != cudaSuccess) return e;
        room = SCR_SMEM_BLOCK - (int)a.sharedSizeBytes;
        const void* none = nullptr;
        if (tries < 256 && (kernels[at].compare_exchange_strong(none, kernel, std::memory_order_acq_rel) || none == kernel))
            rooms[at].store(room, std::memory_order_release);
    }
    if (bytes > (size_t)room) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, room);
}

constexpr int SCR_NORM_MAX_HIDDEN = 200 * 1024 / 4;      // features that scr_rmsnorm_bf16 holds in shared memory

// ---- device-side load helpers -------------------------------------------------------
// Streaming 128-bit / 64-bit loads for weights that are read exactly once per call:
// read-only path, no L1 allocation.
__device__ __forceinline__ uint4 ld_stream_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_stream_v2(const void* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
// Activations: an ordinary (coherent, L1-allocating) 128-bit load.  They are written by the preceding kernel of the
// stream, and under programmatic dependent launch the reading kernel is alive before that kernel has finished, so
// the read-only path (whose contract is data constant for the kernel's lifetime) is not used for them.
__device__ __forceinline__ uint4 ld_act_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
// Cached read-only 128-bit load: load-time constants only (norm gains, tables).
__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
