"""Row operators that hold a row in registers, at the widths where their dispatch changes, against plain 64-bit statements."""
import ctypes

import numpy as np
import pytest

from oracle import sequence_plain as plain
from tests import seq_util as su
from tests.test_sequence_ops_gpu import TOL, dev, draw, healthy, host, lib, ptr, stream, torch_

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,vdim,lead,pad", [(3, 8, 8, 0), (2, 248, 0, 8), (5, 256, 8, 0), (1, 264, 0, 0), (2, 512, 8, 8), (2, 520, 0, 0), (2, 256, 4, 0),
                                                 (2, 256, 0, 4)])
def test_memory_readout(heads, vdim, lead, pad):
    """A warp per row and head up to 512 values; a CTA beyond, and where the gate's rows do not start on 16 bytes."""
    from scratchy_b200 import _lib
    from scratchy_b200.dense import dtype_code
    torch = torch_()
    L, c = lib()
    rng = np.random.default_rng(heads * vdim + lead)
    T = 7
    o, w = rng.standard_normal((T, heads * vdim)).astype(np.float32), rng.standard_normal(heads * vdim).astype(np.float32)
    g = draw(rng, (T, lead + heads * vdim + pad), "bfloat16")
    o[0] *= 1e-4
    shape = _lib.MlstmShape(heads, 16, vdim, 1.0, 1e-5)
    od, wd, gd, y = dev(o), dev(w), dev(g, "bfloat16"), torch.full((T, heads * vdim), float("nan"), dtype=torch.bfloat16, device="cuda")
    c.check(L.scr_mlstm_finish(c.handle, dtype_code(y.dtype), ctypes.byref(shape), ptr(od), ptr(wd), ptr(gd, lead), g.shape[1], T, ptr(y), stream()))
    want = plain.unit_rms(o.astype(np.float64).reshape(T, heads, vdim), 1e-5).reshape(T, -1) * w * plain.sigmoid(g[:, lead:lead + heads * vdim].astype(np.float64))
    assert su.rel(host(y), want) < TOL["bfloat16"] and su.rel(host(y)[0], want[0]) < TOL["bfloat16"]
    healthy()


@pytest.mark.parametrize("W", [4, 1020, 1024, 1028, 2052, 4092, 4096, 4100])
def test_norm_widths(W):
    from scratchy_b200.dense import seq_norm
    torch = torch_()
    rng = np.random.default_rng(W)
    T, eps = 3, 0.01
    x, d = rng.standard_normal((T, W)).astype(np.float32), 3 * rng.standard_normal((T, W)).astype(np.float32)
    wd, wo = (0.5 * rng.standard_normal(W).astype(np.float32) for _ in range(2))
    xd, out = dev(x), torch.full((T, W), float("nan"), dtype=torch.bfloat16, device="cuda")
    seq_norm(xd, eps, delta=dev(d), w_delta=dev(wd), out=out, w_out=dev(wo))
    want = x.astype(np.float64) + plain.norm_around_zero(d.astype(np.float64), wd, eps)
    assert su.rel(host(xd), want) < 1e-6 and su.rel(host(out), plain.norm_around_zero(want, wo, eps)) < TOL["bfloat16"]
    healthy()


@pytest.mark.parametrize("width,ld", [(1, 4), (5, 8), (4097, 4100), (128256, 128256), (777, 779)])
def test_greedy_picks_the_first_of_equals_at_any_alignment(width, ld):
    from scratchy_b200.dense import greedy
    torch = torch_()
    g = torch.Generator().manual_seed(width)
    rows = torch.randint(-50, 50, (3, ld), generator=g).float()
    rows[1, :width] = -3.0                                           # all equal: the first
    want = rows[:, :width].numpy().argmax(axis=1)
    assert greedy(rows.cuda()[:, :width]).cpu().numpy().tolist() == want.tolist()


@pytest.mark.parametrize("longest,hq,hkv,d,bs,batch", [(1600, 8, 4, 64, 16, 40), (1600, 6, 2, 128, 32, 80), (700, 8, 4, 128, 16, 40), (300, 8, 4, 128, 16, 40),
                                                       (1700, 4, 4, 64, 64, 12), (2100, 3, 1, 128, 16, 21)])
def test_decode_attention_at_every_cut_and_number_of_warps(longest, hq, hkv, d, bs, batch):
    """Sequences of all lengths up to `longest` in one launch: halved for length alone, four, six and eight warps a CTA."""
    from scratchy_b200 import synth
    from tests.test_decode_gpu import REL_L2_TOL, _attention_case
    from util import rel_l2
    rng = np.random.default_rng(longest + batch)
    lens = [longest, 1, bs, bs + 1] + rng.integers(1, longest + 1, batch - 4).tolist()
    got, want = _attention_case(lens, hq, hkv, d, bs, synth.seed_for("cut", longest, hq, hkv, d, bs))
    assert rel_l2(got, want) <= REL_L2_TOL


@pytest.mark.parametrize("longest,hq,hkv,d,bs,batch", [(1000, 16, 4, 128, 16, 24), (1700, 28, 4, 128, 16, 20), (4500, 16, 2, 128, 16, 9), (1000, 8, 4, 128, 48, 20)])
def test_decode_attention_with_warps_that_do_not_all_fit(longest, hq, hkv, d, bs, batch):
    """Four or two warps where the query heads, the table or the blocks leave no room for six."""
    test_decode_attention_at_every_cut_and_number_of_warps(longest, hq, hkv, d, bs, batch)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,dim,vdim,batch", [(2, 129, 40, 3), (5, 256, 64, 29), (5, 256, 64, 30), (2, 260, 72, 4), (1, 512, 33, 2)])
def test_memory_step_of_large_heads(heads, dim, vdim, batch, dtype):
    """Keys of more than 128 values: in registers while a round of CTAs holds them, in shared memory beyond (and beyond 256)."""
    from tests.test_sequence_ops_gpu import draw_memory, head_rows, plain_memory, run_memory
    m = su.memory_spec(heads, dim, vdim)["mixer"]
    rng = np.random.default_rng(dim + batch)
    seqs = [(draw_memory(rng, 5, m, dtype), (2.0 * rng.standard_normal((5, 2 * heads))).astype(np.float32)) for _ in range(batch)]
    bi, bf = np.zeros(heads, np.float32), np.full(heads, 2.0, np.float32)
    got, _ = run_memory(m, dtype, [p for p, _ in seqs], [g for _, g in seqs], bi, bf, [[3] * batch, [1] * batch, [1] * batch], list(range(batch)))
    for o, (p, g) in zip(got, seqs):
        assert su.rel(head_rows(o, heads), head_rows(plain_memory(m, p, g, bi, bf), heads)) < (2e-5 if dtype == "float32" else 5e-4)


@pytest.mark.parametrize("W,T,delta", [(88, 296, True), (88, 297, True), (1020, 300, True), (1024, 300, True), (3072, 300, True), (3076, 300, True), (1024, 300, False),
                                       (4096, 296, False), (4096, 297, False)])
def test_norm_of_many_rows(W, T, delta):
    """Both kernels on both sides of the rule between them: one round of rows, and widths with a sublayer's output beyond it."""
    from scratchy_b200.dense import seq_norm
    torch = torch_()
    rng = np.random.default_rng(W + T)
    x, d = rng.standard_normal((T, W)).astype(np.float32), 3 * rng.standard_normal((T, W)).astype(np.float32)
    wd, wo = (0.5 * rng.standard_normal(W).astype(np.float32) for _ in range(2))
    xd, out = dev(x), torch.full((T, W), float("nan"), dtype=torch.bfloat16, device="cuda")
    seq_norm(xd, 0.01, **(dict(delta=dev(d), w_delta=dev(wd)) if delta else {}), out=out, w_out=dev(wo))
    want = x.astype(np.float64) + (plain.norm_around_zero(d.astype(np.float64), wd, 0.01) if delta else 0.0)
    assert su.rel(host(xd), want) < 1e-6 and su.rel(host(out), plain.norm_around_zero(want, wo, 0.01)) < TOL["bfloat16"]
    healthy()


@pytest.mark.parametrize("rows,width,ld", [(148, 8192, 8192), (149, 8192, 8192), (5, 8191, 8192), (3, 12289, 12289), (200, 50000, 50000)])
def test_greedy_with_one_and_eight_requests_in_flight(rows, width, ld):
    """Rows and widths on both sides of the rule; the largest value at the ends of a thread's run, and NaN never."""
    from scratchy_b200.dense import greedy
    torch = torch_()
    g = torch.Generator().manual_seed(width + rows)
    x = torch.randint(-50, 50, (rows, ld), generator=g).float()
    for r in range(rows):
        x[r, (0, width - 1, width // 2, 4095, 4096)[r % 5]] = 60.0
    x[-1] = float("nan")
    x[-1, 7] = -1.0
    want = torch.nan_to_num(x[:, :width], nan=-1e9).numpy().argmax(axis=1)
    assert greedy(x.cuda()[:, :width]).cpu().numpy().tolist() == want.tolist()
