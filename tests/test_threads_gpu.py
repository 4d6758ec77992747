"""Host threads: a thread's first call."""
import ctypes
import threading

import pytest

from scratchy_b200 import synth
from util import bf16_dev, u32_dev

pytestmark = pytest.mark.gpu


def problem(ctx, status):
    from scratchy_b200 import _lib
    return status and (status, _lib.lib().scr_last_error(ctx.handle))


def linear(ctx, layer, x, y, stream):
    from scratchy_b200 import _lib
    return _lib.lib().scr_linear_affine_b4(ctx.handle, layer.packed.data_ptr(), x.data_ptr(), x.shape[0], layer.out_features, layer.in_features, 64, None,
                                           y.data_ptr(), None, ctypes.c_size_t(0), stream)


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
