"""Host threads: a thread's first call, and two threads of one device, a context each, whose calls of the same kernel at sizes that ask for
different shared memory do not disturb one another."""
import ctypes
import os
import subprocess
import threading

import pytest

from scratchy_b200 import synth
from util import bf16_dev, u32_dev

pytestmark = pytest.mark.gpu
ROUNDS = 20000


def problem(ctx, status):
    from scratchy_b200 import _lib
    return status and (status, _lib.lib().scr_last_error(ctx.handle))


def linear(ctx, layer, x, y, stream):
    from scratchy_b200 import _lib
    return _lib.lib().scr_linear_affine_b4(ctx.handle, layer.packed.data_ptr(), x.data_ptr(), x.shape[0], layer.out_features, layer.in_features, 64, None,
                                           y.data_ptr(), None, ctypes.c_size_t(0), stream)


HAMMER = """
#include <atomic>
#include <thread>
#include "scratchy_cuda.h"
typedef int32_t (*linear_fn)(scr_ctx*, const void*, const uint16_t*, int32_t, int32_t, int32_t, int32_t, const uint16_t*, uint16_t*, void*, size_t, void*);
typedef int32_t (*attention_fn)(scr_ctx*, const uint16_t*, int64_t, const uint16_t*, const uint16_t*, int32_t, const uint32_t*, const uint32_t*, uint16_t*,
                                int64_t, int32_t, int32_t, int32_t, int32_t, int32_t, int32_t, float, void*);
typedef int32_t (*init_fn)(int32_t, scr_ctx**);
typedef int32_t (*destroy_fn)(scr_ctx*);
struct Library { init_fn init; destroy_fn destroy; void* call; };
template <typename Call>
static int side_by_side(const Library* lib, int rounds, Call call) {
    std::atomic<int> ready{0}, failed{0};
    auto work = [&](int which) {
        scr_ctx* ctx = nullptr;
        const int32_t made = lib->init(0, &ctx);
        ready++;
        while (ready < 2) {}
        if (made) failed = made;
        for (int i = 0; i < rounds && !failed; ++i) {
            const int32_t status = call(ctx, which);
            if (status) failed = status;
        }
        if (ctx) lib->destroy(ctx);
    };
    std::thread other(work, 1);
    work(0);
    other.join();
    return failed;
}
extern "C" int linears(const Library* lib, int rounds, void** w, void** x, int32_t M, int32_t* N, int32_t* K, void** y, void** stream) {
    const linear_fn f = (linear_fn)lib->call;
    return side_by_side(lib, rounds, [&](scr_ctx* c, int i) { return f(c, w[i], (uint16_t*)x[i], M, N[i], K[i], 64, nullptr, (uint16_t*)y[i], nullptr, 0, stream[i]); });
}
extern "C" int attentions(const Library* lib, int rounds, void** q, void** k, void** v, void** table, void** used, void** y, int32_t* batch, int32_t* blocks,
                          int32_t heads, int32_t kv_heads, int32_t dim, void** stream) {
    const attention_fn f = (attention_fn)lib->call;
    return side_by_side(lib, rounds, [&](scr_ctx* c, int i) {
        return f(c, (uint16_t*)q[i], heads * dim, (uint16_t*)k[i], (uint16_t*)v[i], batch[i] * blocks[i], (uint32_t*)table[i], (uint32_t*)used[i], (uint16_t*)y[i],
                 heads * dim, batch[i], heads, kv_heads, dim, 16, blocks[i], 0.088f, stream[i]);
    });
}
"""


@pytest.fixture(scope="module")
def hammer(tmp_path_factory):
    """Calls from two threads, over and over, without the interpreter between them."""
    folder, include = tmp_path_factory.mktemp("hammer"), os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include")
    (folder / "hammer.cpp").write_text(HAMMER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-I", include, "-o", folder / "hammer.so", folder / "hammer.cpp"], check=True)
    return ctypes.CDLL(str(folder / "hammer.so"))


def pointers(items):
    """Of streams and tensors."""
    return (ctypes.c_void_p * len(items))(*[i.cuda_stream if hasattr(i, "cuda_stream") else i.data_ptr() for i in items])


def library(call):
    from scratchy_b200 import _lib
    return (ctypes.c_void_p * 3)(*[ctypes.cast(getattr(_lib.lib(), n), ctypes.c_void_p) for n in ("scr_cuda_init", "scr_cuda_destroy", call)])


def ints(items):
    return (ctypes.c_int32 * len(items))(*items)


@pytest.mark.parametrize("M", [1, 9, 16, 24])
def test_first_call_of_a_thread(M):
    """A thread that has made no CUDA call of its own yet, on the context that its program made elsewhere."""
    import torch
    from scratchy_b200 import AffineQuantLinear, _lib
    N, K = 3072, 2048
    w, s, b = synth.affine_int4_weights(N, K, 64, 3)
    layer, x = AffineQuantLinear.from_tensors(u32_dev(w), bf16_dev(s), bf16_dev(b), 64, 4), bf16_dev(synth.activations_bf16(M, K, 1)).reshape(M, K)
    want, y, ctx, found = layer.forward(x), torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), _lib.context(0), []
    torch.cuda.synchronize()
    thread = threading.Thread(target=lambda: found.append(problem(ctx, linear(ctx, layer, x, y, None))))
    thread.start()
    thread.join()
    torch.cuda.synchronize()
    assert found == [0] and torch.equal(y, want)


def test_few_token_linears(hammer):
    """A matrix whose clusters all run at once has each CTA alone on its SM, one of more tiles than SMs two to an SM."""
    import torch
    from scratchy_b200 import AffineQuantLinear
    made, M = [], 24
    for N, K in ((3072, 1024), (128 * 300, 256)):
        w, s, b = synth.affine_int4_weights(N, K, 64, synth.seed_for("threads", N, K))
        layer, x = AffineQuantLinear.from_tensors(u32_dev(w), bf16_dev(s), bf16_dev(b), 64, 4), bf16_dev(synth.activations_bf16(M, K, 1)).reshape(M, K)
        made.append((layer.packed, x, N, K, torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), torch.cuda.Stream(), layer.forward(x)))
    w, x, N, K, y, streams, want = zip(*made)
    torch.cuda.synchronize()
    failed = hammer.linears(library("scr_linear_affine_b4"), ROUNDS, pointers(w), pointers(x), M, ints(N), ints(K), pointers(y), pointers(streams))
    torch.cuda.synchronize()
    assert failed == 0
    assert all(torch.equal(a, b) for a, b in zip(y, want))


def test_decode_attention(hammer):
    """One sequence, whose CTAs are alone on their SMs, beside as many as share theirs."""
    import torch
    from scratchy_b200 import decode
    made, H, G, D = [], 16, 8, 128
    for B, length in ((1, 900), (16, 100)):
        blocks, g = (length + 15) // 16, torch.Generator(device="cuda").manual_seed(B)
        q, k, v = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((B, H * D), (B * blocks, G, 16, D), (B * blocks, G, 16, D)))
        table = torch.arange(B * blocks, dtype=torch.int32, device="cuda").reshape(B, blocks)
        used = torch.full((B,), length, dtype=torch.int32, device="cuda")
        want = decode.attention_via_cache(q, k, v, table, used, H, G, D, 16, 0.088)
        made.append((q, k, v, table, used, torch.empty_like(want), torch.cuda.Stream(), want, B, blocks))
    q, k, v, table, used, y, streams, want, batch, blocks = zip(*made)
    torch.cuda.synchronize()
    failed = hammer.attentions(library("scr_attention_via_cache_bf16"), ROUNDS, pointers(q), pointers(k), pointers(v), pointers(table), pointers(used),
                               pointers(y), ints(batch), ints(blocks), H, G, D, pointers(streams))
    torch.cuda.synchronize()
    assert failed == 0
    assert all(torch.equal(a, b) for a, b in zip(y, want))
