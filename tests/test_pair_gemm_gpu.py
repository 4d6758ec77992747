"""The int4 GEMM on CTA pairs (given every full round of them through the environment, read once per process) in the forms that a whole-tile shape does not
show: ragged tokens and channels, every group size, f32 partial sums, several tiles per pair over rings that go round."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from scratchy_b200 import synth
from util import rel_l2

pytestmark = pytest.mark.gpu
REL_L2_TOL = 1e-3                    # the bar of every int4 output: one bf16 rounding of an f32-accumulated sum

# N, K, M, group: 37 channel tiles (the last one ragged) by 2 or 4 token tiles, one or two full rounds of 74 pairs
CASES = [(9400, 640, 500, 32), (9472, 640, 257, 64), (9400, 1152, 511, 128), (9464, 2176, 1000, 64), (9472, 3072, 900, 32)]


def made(case):
    N, K, M, group = case
    seed = synth.seed_for("pair", *case)
    w, s, b = synth.affine_int4_weights(N, K, group, seed)
    return w, s, b, synth.activations_bf16(M, K, seed + 1), synth.activations_bf16(1, N, seed + 2).reshape(N)


CHILD = """
import os, sys
import numpy as np
root, out = sys.argv[1:]
sys.path[:0] = [root, os.path.join(root, "tests")]
import torch
from scratchy_b200 import AffineQuantLinear, _lib
from test_pair_gemm_gpu import CASES, made
from util import bf16_dev, bits_of, u32_dev
for i, case in enumerate(CASES):
    N, K, M, group = case
    w, s, b, x, bias = made(case)
    layer, xd = AffineQuantLinear.from_tensors(u32_dev(w), bf16_dev(s), bf16_dev(b), group, 4), bf16_dev(x).reshape(M, K)
    y, part = layer.forward(xd), layer.forward_partial(xd)
    layer.linear_bias = bf16_dev(bias)
    np.savez(os.path.join(out, f"{i}.npz"), y=bits_of(y), part=part.cpu().numpy(), biased=bits_of(layer.forward(xd)))
torch.cuda.synchronize()
_lib.context(0).device_status(None)
"""


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    out = tmp_path_factory.mktemp("pairs")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", CHILD, root, str(out)], check=True, env=dict(os.environ, SCR_AFFINE_GEMM_PAIR="1"), timeout=600)
    return [np.load(out / f"{i}.npz") for i in range(len(CASES))]


@pytest.mark.parametrize("i", range(len(CASES)))
def test_forms(results, i):
    N, K, M, group = CASES[i]
    w, s, b, x, bias = made(CASES[i])
    got = results[i]
    rows = np.unique(np.r_[0, 127, 128, 255, 256, np.random.default_rng(i).integers(0, M, 24), M - 1])
    want = oracle.affine_qmm_t_b4(w.view(np.uint8).reshape(-1), s, b, x.reshape(M, K)[rows], len(rows), N, K, group)
    f32 = lambda bits: (bits.astype(np.uint32) << 16).view(np.float32)
    part = got["part"].reshape(M, N)
    assert rel_l2(got["y"].reshape(M, N)[rows], want) <= REL_L2_TOL
    assert np.isfinite(part).all() and np.array_equal(synth.f32_to_bf16_bits(part), got["y"].reshape(M, N))
    assert np.array_equal(synth.f32_to_bf16_bits(part + f32(bias)[None, :]), got["biased"].reshape(M, N))


@pytest.mark.parametrize("N,M", [(14336, 256), (14210, 193)])
def test_where_it_is_chosen(N, M):
    """Without the environment: a second token tile that would start a round of its own, up to its edges (192 tokens are one tile)."""
    from test_few_tokens_gpu import test_int4
    test_int4(N, 3072, M, 64)
