"""Calls of the matrix memories that follow each other on one stream without the host between them: each goes on from the state
that the one before it leaves.  The bits are those of the same calls with a synchronisation after each."""
import ctypes

import numpy as np
import pytest

from tests import seq_util as su
from tests.test_side_ops_gpu import Window, per_head, plain_lightning, run_lightning
from tests.test_sequence_ops_gpu import DTYPES, Latents, arena, dev, draw, draw_memory, healthy, head_rows, lib, plain_memory, ptr, run_memory, stream, torch_

pytestmark = pytest.mark.gpu

# one portion per call; the state goes from a step to a step, from a prompt's chunks to a step, from a step to chunks
PORTIONS = [[1] * 12, [70, 1, 1], [3, 64, 1, 1, 130, 2]]


def queued(calls, captured):
    """Issues the prepared calls back to back, as they are or as one captured graph."""
    torch = torch_()
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for call in calls:
                call()
        graph.replay()
    else:
        for call in calls:
            call()
    healthy()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim,vdim", [(2, 16, 24), (3, 48, 72), (12, 128, 256), (1, 256, 64), (2, 300, 40)])
@pytest.mark.parametrize("portions", PORTIONS)
def test_gated_memory(heads, dim, vdim, portions, dtype, captured):
    from scratchy_b200 import _lib
    from scratchy_b200.dense import dtype_code
    torch = torch_()
    L, c = lib()
    m = su.memory_spec(heads, dim, vdim)["mixer"]
    rng = np.random.default_rng(heads * dim + vdim)
    T, sl = sum(portions), (vdim + 31) // 32
    proj, gates = draw_memory(rng, T, m, dtype), (2.0 * rng.standard_normal((T, 2 * heads))).astype(np.float32)
    bi, bf = np.zeros(heads, np.float32), np.full(heads, 2.0, np.float32)
    (want,), _ = run_memory(m, dtype, [proj], [gates], bi, bf, [[n] for n in portions], [1])
    shape = _lib.MlstmShape(heads, dim, vdim, m["gate_cap"], 1e-5)
    state = [torch.full(s, float("nan"), device="cuda") for s in ((2, heads, dim, vdim), (2, heads, sl, dim), (2, heads, sl))]
    pd, gd, bid, bfd = dev(proj, dtype), dev(gates), dev(bi), dev(bf)
    out, code = torch.full((T, heads * vdim), float("nan"), device="cuda"), dtype_code(pd.dtype)
    calls, keep, at = [], [], 0
    for n in portions:
        segs = torch.tensor([[0, n, at, 1]], dtype=torch.int32, device="cuda")
        st, need = _lib.Step(0, 0, segs.data_ptr(), 0, n, 1, n, 0, 2), ctypes.c_size_t(0)
        c.check(L.scr_mlstm_workspace(code, ctypes.byref(shape), ctypes.byref(st), ctypes.byref(need)))
        ws = torch.full((max(16, need.value) // 4,), float("nan"), device="cuda")
        keep.append((segs, st, ws))
        calls.append(lambda n=n, at=at, st=st, ws=ws, need=need: c.check(L.scr_mlstm_run(
            c.handle, code, ctypes.byref(shape), ctypes.byref(st), ptr(pd, at * pd.shape[1]), pd.shape[1], ptr(gd, at * 2 * heads), 2 * heads, ptr(bid),
            ptr(bfd), *[ptr(t) for t in state], ptr(out, at * out.shape[1]), ptr(ws), need, stream())))
        at += n
    queued(calls, captured)
    got = out.cpu().numpy()
    assert np.array_equal(got, want.astype(np.float32))
    err = np.sqrt(((head_rows(got, heads) - head_rows(plain_memory(m, proj, gates, bi, bf), heads)) ** 2).mean(axis=2)).ravel()
    assert np.median(err) < (5e-6 if dtype == "float32" else 5e-5)        # (the bar of the calls with a synchronisation after each)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim,vdim", [(2, 16, 24), (3, 48, 72), (8, 128, 128), (1, 256, 64), (1, 300, 20)])
@pytest.mark.parametrize("portions", PORTIONS)
def test_decaying_memory(heads, dim, vdim, portions, dtype, captured):
    from scratchy_b200 import _lib
    from scratchy_b200.dense import dtype_code
    from scratchy_b200.mixers import decay_powers
    torch = torch_()
    L, c = lib()
    m = {"heads": heads, "dim": dim, "vdim": vdim, "decay": ([0.999, 0.6, 0.97] * 3)[:heads]}
    rng = np.random.default_rng(heads * dim + vdim)
    T = sum(portions)
    proj = rng.standard_normal((T, heads * (2 * dim + vdim))).astype(np.float32)
    proj = su.round_bf16(proj) if dtype == "bfloat16" else proj
    (want,), _ = run_lightning(m, dtype, [proj], [[n] for n in portions], [1])
    shape, powers = _lib.LightningShape(heads, dim, vdim, 1e-5, 1.0), decay_powers(np.asarray(m["decay"], np.float64)).cuda()
    state, pd, out = torch.full((2, heads, dim, vdim), float("nan"), device="cuda"), dev(proj, dtype), torch.full((T, heads * vdim), float("nan"), device="cuda")
    code, calls, keep, at = dtype_code(pd.dtype), [], [], 0
    for n in portions:
        segs = torch.tensor([[0, n, at, 1]], dtype=torch.int32, device="cuda")
        st, need = _lib.Step(0, 0, segs.data_ptr(), 0, n, 1, n, 0, 2), ctypes.c_size_t(0)
        c.check(L.scr_lightning_workspace(code, ctypes.byref(shape), ctypes.byref(st), ctypes.byref(need)))
        ws = torch.full((max(16, need.value) // 4,), float("nan"), device="cuda")
        keep.append((segs, st, ws))
        calls.append(lambda n=n, at=at, st=st, ws=ws, need=need: c.check(L.scr_lightning_run(
            c.handle, code, ctypes.byref(shape), ctypes.byref(st), ptr(pd, at * pd.shape[1]), pd.shape[1], ptr(powers), ptr(state),
            ptr(out, at * out.shape[1]), ptr(ws), need, stream())))
        at += n
    queued(calls, captured)
    got = out.cpu().numpy()
    assert np.array_equal(got, want.astype(np.float32))
    assert per_head(got, plain_lightning(m, proj), heads) < (4e-6 if dtype == "float32" else 1e-4)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim,vdim", [(3, 48, 72), (8, 128, 128), (1, 300, 20)])
@pytest.mark.parametrize("rows,attention", [(1, (4, 2, 64)), (1, (5, 1, 10)), (3, (40, 8, 128)), (70, (2, 1, 128)), (300, (2, 1, 64))])
@pytest.mark.parametrize("order", ["attention", "preparation"])
def test_decaying_memory_beside_an_attention(order, rows, attention, heads, dim, vdim, dtype, captured):
    """The memory beside each kernel of the window attention or of its preparation and, after the latter, the readout norm beside the attention; the
    inputs by the linear before them, in the buffers that the step before has read."""
    from scratchy_b200 import _lib
    from scratchy_b200.dense import DenseLinear, dtype_code
    from scratchy_b200.mixers import decay_powers
    torch = torch_()
    L, c = lib()
    steps, W, past, C = 8, heads * (2 * dim + vdim), 200, (attention[0] + attention[1]) * attention[2]
    rng = np.random.default_rng(rows + dim)
    w = Window(*attention, 90, 5, 40, [past + rows], dtype, seed=rows)
    cache, taps, ones = dev(draw(rng, tuple(w.cache.shape), dtype), dtype), dev(rng.standard_normal((3, C))), torch.ones(C, device="cuda")
    st, sh, nq, bias = w.step([rows], [past], [1]), w.shape(), attention[0] * attention[2], w.padded_bias()
    q, gate = dev(draw(rng, (rows, nq), dtype), dtype), dev(rng.standard_normal((rows, attention[0])))
    x, a, lin = dev(draw(rng, (steps, rows, 64), dtype), dtype), arena(), DenseLinear(dev(draw(rng, (W + C + heads * vdim, 64), dtype, 0.125), dtype))
    shape, powers, code = _lib.LightningShape(heads, dim, vdim, 1e-5, 1.0), decay_powers(np.asarray(([0.999, 0.6, 0.97] * 3)[:heads], np.float64)).cuda(), dtype_code(q.dtype)
    need = ctypes.c_size_t(0)
    c.check(L.scr_lightning_workspace(code, ctypes.byref(shape), ctypes.byref(st), ctypes.byref(need)))
    ws, results = torch.empty(max(16, need.value), dtype=torch.uint8, device="cuda"), []
    ones_v = torch.ones(heads * vdim, device="cuda")
    for beside in (False, True):
        nan = lambda *n, t=torch.float32: torch.full(n, float("nan"), dtype=t, device="cuda")
        proj, state, out, y = nan(rows, W + C + heads * vdim, t=q.dtype), torch.zeros((2, heads, dim, vdim), device="cuda"), nan(rows, heads * vdim), nan(steps, rows, nq + 8, t=q.dtype)
        z, kept, inv, last = nan(steps, rows, heads * vdim, t=q.dtype), cache.clone(), torch.full_like(w.key_scale, 0.1), torch.zeros((2, 2, C), dtype=q.dtype, device="cuda")
        ld, qs = proj.shape[1], q.clone()
        common = (c.handle, code, ctypes.byref(sh), ctypes.byref(st))

        def step(t, beside=beside, proj=proj, state=state, out=out, y=y, z=z, kept=kept, inv=inv, last=last, ld=ld, qs=qs, common=common):
            lin(a, x[t], proj)
            prepare = lambda: c.check(L.scr_window_prepare(*common, ptr(proj, W), ld, ptr(taps), ptr(ones), ptr(last), ptr(qs), ptr(kept), ptr(inv), stream()))
            attend = lambda: c.check(L.scr_window_attention(*common, ptr(qs), ptr(kept), ptr(inv), ptr(bias), ptr(gate), attention[0], ptr(y[t]), nq + 8, stream()))
            remember = lambda: c.check((L.scr_lightning_beside if beside else L.scr_lightning_run)(
                c.handle, code, ctypes.byref(shape), ctypes.byref(st), ptr(proj), ld, ptr(powers), ptr(state), ptr(out), ptr(ws), need, stream()))
            read = lambda finish: c.check(finish(c.handle, code, ctypes.byref(shape), ptr(out), ptr(ones_v), ptr(proj, W + C), ld, rows, ptr(z[t]), heads * vdim, stream()))
            prepare()
            if order == "attention":
                attend()
                remember()
                read(L.scr_lightning_finish)
            else:
                remember()
                attend()
                read(L.scr_lightning_finish_beside if beside else L.scr_lightning_finish)

        if beside:
            queued([lambda t=t: step(t) for t in range(steps)], captured)
        else:
            for t in range(steps):
                step(t)
                healthy()
        results.append((z, state[1], y[:, :, :nq], last, kept))
    for one, other in zip(*results):
        assert torch.equal(one, other) and torch.isfinite(one).all()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("heads,kv_rank,rot_dim", [(3, 48, 8), (24, 512, 64)])
@pytest.mark.parametrize("start,tokens", [(0, 3), (58, 12), (126, 6), (700, 8)])
def test_latent_cache(start, tokens, heads, kv_rank, rot_dim, captured):
    """A token's cache row stored by one call and read by the next ones, on both sides of a key tile's end."""
    torch = torch_()
    L, c = lib()
    m = su.attention_spec(heads=heads, kv_rank=kv_rank, rot_dim=rot_dim, q_rank=32, scale=(kv_rank + rot_dim) ** -0.5)["mixer"]
    from scratchy_b200 import _lib
    results = []
    for synchronised in (True, False):
        lt = Latents(m, [start], [tokens], "bfloat16", seed=start + heads)          # (the same seed: the same cache, blocks and rows)
        rng = np.random.default_rng(start)
        lt.cache[lt.slots[0][start:]] = float("nan")                                # the calls below store these rows
        d, q = dev(rng.standard_normal((tokens, 32 + lt.D))), dev(rng.standard_normal((tokens, heads, lt.D)), "bfloat16")
        wq, wkv = dev(np.ones(32)), dev(np.ones(kv_rank))
        cq, out = (torch.full((tokens, n), float("nan"), dtype=torch.bfloat16, device="cuda") for n in (32, heads * kv_rank))
        calls, keep = [], []
        for t in range(tokens):
            i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
            arrays = [i32(0), i32(start + t), i32(0, 1, start + t, 0)]
            st = _lib.Step(*[a.data_ptr() for a in arrays], lt.dev_arrays[3].data_ptr(), 1, 1, 1, start + t + 1, 1)
            need = ctypes.c_size_t(0)
            c.check(L.scr_latent_attention_workspace(lt.code(), ctypes.byref(lt.shape), ctypes.byref(st), ctypes.byref(need)))
            ws = torch.empty(max(16, need.value), dtype=torch.uint8, device="cuda")
            keep.append((arrays, st, ws))

            def call(t=t, st=st, ws=ws, need=need):
                c.check(L.scr_latent_prepare(c.handle, lt.code(), ctypes.byref(lt.shape), ctypes.byref(st), ptr(d, t * d.shape[1]), d.shape[1], ptr(wq), ptr(wkv),
                                             ptr(lt.cos), ptr(lt.sin), ptr(cq, t * 32), ptr(lt.cache), stream()))
                c.check(L.scr_latent_attention(c.handle, lt.code(), ctypes.byref(lt.shape), ctypes.byref(st), ptr(q, t * heads * lt.D), ptr(lt.cache),
                                               ptr(out, t * heads * kv_rank), ptr(ws), need, stream()))
                if synchronised:
                    torch.cuda.synchronize()
            calls.append(call)
        queued(calls, captured and not synchronised)
        results.append(out.float().cpu().numpy())
    assert np.isfinite(results[0]).all() and np.array_equal(*results)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("M,N,K", [(5, 200, 512), (16, 18952, 1032), (120, 1024, 512), (40, 3072, 3072), (200, 512, 512)])
def test_a_linear_whose_matrix_the_call_before_it_writes(M, N, K, captured):
    """`w_fresh`: the latents of a prompt are the matrix of the linear that expands its values, at row counts of every kernel."""
    from scratchy_b200.dense import Arena, DenseLinear
    torch = torch_()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    draw = lambda *s: torch.randn(s, device="cuda", generator=g).bfloat16()
    a, b, x = draw(N, 2048), draw(K, 2048), draw(M, K)
    arena, results = Arena("cuda"), []
    for synchronised in (True, False):
        w, y = torch.zeros((N, K), dtype=torch.bfloat16, device="cuda"), torch.full((M, N), float("nan"), device="cuda")
        first, second = DenseLinear(b), DenseLinear(w, fresh=True)
        calls = [lambda: first(arena, a, w), lambda: second(arena, x, y)]
        for _ in range(2):                                                   # (the buffers have their sizes before a capture)
            w.zero_()
            if synchronised:
                for call in calls:
                    call()
                    torch.cuda.synchronize()
            else:
                queued(calls, captured)
        results.append(y)
    assert torch.equal(*results)
