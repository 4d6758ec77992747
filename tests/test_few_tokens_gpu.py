"""The GEMMs for few tokens (weights as the rows of the MMA, k shared by a cluster) at the edges of their tiles and splits,
against the oracle with the bars of the paths they stand beside."""
import numpy as np
import pytest

import oracle
from scratchy_b200 import synth
from util import bf16_dev, bits_of, rel_l2, u32_dev

pytestmark = pytest.mark.gpu
REL_L2_TOL = 1e-3                    # the bar of every int4 and fp8 output: one bf16 rounding of an f32-accumulated sum


@pytest.mark.parametrize("group", [32, 64, 128])
@pytest.mark.parametrize("N,K,M", [(8, 128, 17), (130, 384, 32), (136, 640, 33), (128, 1152, 48), (3072, 3072, 64), (264, 2176, 65), (1000, 8192, 127),
                                   (5120, 3072, 128)])
def test_int4(N, K, M, group):
    """Token counts on both sides of 32, 64 and 128; one k chunk and rings that go round; 1 to 8 CTAs per tile; ragged channels;
    with a bias, and as unrounded partial sums."""
    import torch
    from scratchy_b200 import AffineQuantLinear
    seed = synth.seed_for("few", N, K, M, group)
    w, s, b = synth.affine_int4_weights(N, K, group, seed)
    x = synth.activations_bf16(M, K, seed + 1)
    bias = synth.activations_bf16(1, N, seed + 2).reshape(N)
    want = oracle.affine_qmm_t_b4(w.view(np.uint8).reshape(-1), s, b, x, M, N, K, group)
    layer = AffineQuantLinear.from_tensors(u32_dev(w), bf16_dev(s), bf16_dev(b), group, 4)
    xd = bf16_dev(x).reshape(M, K)
    y, part = layer.forward(xd), layer.forward_partial(xd)
    layer.linear_bias = bf16_dev(bias)
    yb = layer.forward(xd)
    torch.cuda.synchronize()
    assert rel_l2(bits_of(y).reshape(M, N), want) <= REL_L2_TOL
    assert torch.equal(part.bfloat16().view(torch.int16), y.view(torch.int16))
    assert torch.equal((part + layer.linear_bias.float()).bfloat16().view(torch.int16), yb.view(torch.int16))


@pytest.mark.parametrize("N,K,M", [(8, 8, 17), (130, 200, 32), (136, 64, 33), (520, 1032, 64), (300, 4104, 65), (3072, 3072, 128), (18952, 1032, 1),
                                   (9480, 2056, 16)])
def test_dense(N, K, M):
    """The same edges of the bf16 linear: plain and f32 outputs against 64-bit sums, and the residual end."""
    import torch
    from scratchy_b200.dense import Arena, DenseLinear
    rng = np.random.default_rng(N + K + M)
    draw = lambda *shape: torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda().bfloat16()
    x, w, a = draw(M, K), draw(N, K), Arena("cuda")
    want = (x.double() @ w.double().T).cpu()
    lin, rel = DenseLinear(w), lambda t: float((t.double().cpu() - want).norm() / want.norm())
    y, y16 = torch.full((M, N), float("nan"), device="cuda"), torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    lin(a, x, y)
    lin(a, x, y16)
    res = torch.ones((M, N), device="cuda")
    lin.add_to(a, x, res)
    torch.cuda.synchronize()
    assert rel(y) < 1e-5                                          # f32 sums of at most 4104 products
    assert torch.equal(y.bfloat16().view(torch.int16), y16.view(torch.int16))
    assert torch.equal(res, y + 1.0)


@pytest.mark.parametrize("N,K,M", [(256, 64, 256), (2560, 200, 1300), (264, 712, 260), (3072, 1096, 2000)])
def test_dense_on_cta_pairs(N, K, M):
    """256 x 256 tiles on pairs of SMs: odd numbers of k slices, rows and columns that end inside a CTA's half, rounds that are
    cut along k and rounds that are not."""
    test_dense(N, K, M)


@pytest.mark.parametrize("group", [32, 64])
@pytest.mark.parametrize("N,K,M", [(8, 128, 129), (130, 384, 192), (264, 640, 193), (1000, 1152, 400), (4096, 2176, 1030), (8192, 3072, 770)])
def test_int4_prompts(N, K, M, group):
    """The same checks on tiles of 128 to 192 tokens: counts on both sides of a tile, whole rounds, cut tails, one chunk."""
    test_int4(N, K, M, group)


@pytest.mark.parametrize("N,K,M", [(8, 64, 17), (130, 328, 32), (264, 1160, 33), (512, 3584, 65), (300, 18944, 128), (384, 256, 129), (3584, 2184, 250)])
def test_fp8(N, K, M):
    """Token counts on both sides of 32, 64 and 128, and up to the 256 of one accumulator; ragged channels and k."""
    import torch
    from scratchy_b200 import Fp8Linear
    from util import to_dev
    seed = synth.seed_for("few8", N, K, M)
    wq, ws = oracle.fp8_quantize_weight_per_channel(synth.fp8_weights_f32(N, K, seed))
    x = synth.activations_bf16(M, K, seed + 1)
    layer, xd = Fp8Linear.from_tensors(to_dev(wq), to_dev(ws)), bf16_dev(x).reshape(M, K)
    layer.linear_bias = bf16_dev(synth.activations_bf16(1, N, seed + 2).reshape(N))
    yb, part = layer.forward(xd), layer.forward_partial(xd)
    layer.linear_bias, bias = None, layer.linear_bias
    y = layer.forward(xd)
    torch.cuda.synchronize()
    assert rel_l2(bits_of(y).reshape(M, N), oracle.fp8_dynamic_linear(x, wq, ws, M, N, K)) <= REL_L2_TOL
    assert torch.equal(part.bfloat16().view(torch.int16), y.view(torch.int16))
    assert torch.equal((part + bias.float()).bfloat16().view(torch.int16), yb.view(torch.int16))


@pytest.mark.parametrize("M", [5, 8, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K,group", [(2064, 2048, 64), (4160, 1024, 32), (16400, 2560, 128), (4736, 1024, 64), (3600, 1536, 64)])
def test_int4_ends_of_few_tokens(N, K, group, M):
    """The ends of the GEMM for few tokens on both sides of the matvec's sizes: bias and scale, the residual add and the gate/up pairing
    give the bits of the plain linear followed by the operator; the plain linear is held to the oracle."""
    import torch
    from scratchy_b200 import AffineQuantLinear, _lib
    seed = synth.seed_for("few-ends", N, K, M, group)
    w, s, b = synth.affine_int4_weights(N, K, group, seed)
    x = synth.activations_bf16(M, K, seed + 1)
    layer = AffineQuantLinear.from_tensors(u32_dev(w), bf16_dev(s), bf16_dev(b), group, 4)
    xd, new = bf16_dev(x).reshape(M, K), lambda n=N: torch.full((M, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    y = layer.forward(xd, out=new())
    rows = np.unique(np.random.default_rng(M).integers(0, M, 8))
    want = oracle.affine_qmm_t_b4(w.view(np.uint8).reshape(-1), s, b, x[rows], len(rows), N, K, group)
    assert rel_l2(bits_of(y).reshape(M, N)[rows], want) <= REL_L2_TOL
    res = bf16_dev(synth.activations_bf16(M, N, seed + 2)).reshape(M, N)
    added = layer.forward_add(xd, res.clone())
    assert torch.equal(added.view(torch.int16), (res.float() + y.float()).bfloat16().view(torch.int16))
    layer.pairs8 = True
    act, two = layer.forward_silu_mul(xd, out=new(N // 2)), new(N // 2)
    ctx = _lib.context(0)
    ctx.check(_lib.lib().scr_silu_mul_pairs8_bf16(ctx.handle, y.data_ptr(), N, two.data_ptr(), M, N // 2, None))
    assert torch.equal(act.view(torch.int16), two.view(torch.int16))
    layer.linear_bias = bf16_dev(synth.activations_bf16(1, N, seed + 3)).reshape(N)
    part = layer.forward_partial(xd)
    assert torch.equal(part.bfloat16().view(torch.int16), y.view(torch.int16))
    biased = (part + layer.linear_bias.float()).bfloat16()
    assert torch.equal(layer.forward(xd).view(torch.int16), biased.view(torch.int16))
    added = layer.forward_add(xd, res.clone())
    assert torch.equal(added.view(torch.int16), (res.float() + biased.float()).bfloat16().view(torch.int16))
    if M <= 16:
        scaled = layer.forward_ends(xd, new(), scale=0.125)
        assert torch.equal(scaled.view(torch.int16), ((part + layer.linear_bias.float()) * 0.125).bfloat16().view(torch.int16))
    torch.cuda.synchronize()


@pytest.mark.parametrize("N", [51200, 51208])
def test_residual_and_norm_of_rows_wider_than_a_norm_takes(N):
    """The residual end with the norm behind it: rows up to what the stand-alone norm holds, whose launch follows the GEMM, and wider ones, which
    only the matvec's epilogue normalises."""
    import torch
    from scratchy_b200 import AffineQuantLinear
    K, M = 128, 9
    w, s, b = synth.affine_int4_weights(N, K, 64, synth.seed_for("wide-norm", N))
    layer = AffineQuantLinear.from_tensors(u32_dev(w), bf16_dev(s), bf16_dev(b), 64, 4)
    x, res0 = bf16_dev(synth.activations_bf16(M, K, 1)).reshape(M, K), bf16_dev(synth.activations_bf16(M, N, 2)).reshape(M, N)
    gain, res, normed = bf16_dev(synth.activations_bf16(1, N, 3)).reshape(N), res0.clone(), torch.full_like(res0, float("nan"))
    layer.forward_residual_rmsnorm(x, res, gain, 1e-5, normed, torch.zeros(AffineQuantLinear.ENDS_SCRATCH_BYTES, dtype=torch.uint8, device="cuda"))
    want = res0.double() + (x.double() @ layer.dequantize().double().T).bfloat16().double()
    assert float((res.double() - want).norm() / want.norm()) < 4e-3                       # one bf16 rounding, a few of the product's the other way
    r = res.double()
    want = r / torch.sqrt((r * r).mean(dim=1, keepdim=True) + 1e-5) * gain.double()
    assert float((normed.double() - want).norm() / want.norm()) < 4e-3


@pytest.mark.parametrize("tiles", [147, 148, 149, 300])
def test_calls_whose_clusters_do_not_all_run_at_once(tiles):
    """As many tiles of 128 channels as SMs, where every CTA has its SM and memory for the sums to itself, and more, where two share an
    SM and the sums lie over the rings; runs of tokens that are added four at a time and one at a time."""
    N = 128 * tiles - 8
    test_int4(N, 384, 33, 64)
    test_fp8(N, 200, 45)
    test_dense(N, 200, 16)
    test_dense(128 * tiles // 8 + 8, 1096, 33)


@pytest.mark.parametrize("K", [1024, 4096, 8200, 12296, 20480, 20488])
def test_quantisation_of_every_code_and_tie(K):
    """Every bf16 value in [-448, 448] at a scale of one (half-way cases of every binade and of the subnormal grid among them),
    at row lengths on both sides of every count of pieces a thread holds: the oracle's bytes."""
    from scratchy_b200 import Fp8Linear
    every = np.arange(0x43E0 + 1, dtype=np.uint16)                 # 0 .. 448
    every = np.concatenate([every, every | np.uint16(0x8000)])
    M = max(17, -(-every.size // (K - 1)))
    x = np.zeros((M, K), np.uint16)
    x[:, 0] = 0x43E0                                               # the row's largest: scale 448 * (1 / 448) = 1
    flat = np.resize(every, M * (K - 1)).reshape(M, K - 1)
    x[:, 1:] = flat
    xq, a = Fp8Linear.quantize_activation(bf16_dev(x.reshape(-1)).reshape(M, K)).unpack()
    want_q, want_a = oracle.fp8_quant_per_token(x.reshape(-1), M, K)
    assert (want_a == 1.0).all()
    assert np.array_equal(a.cpu().numpy(), want_a) and np.array_equal(xq.cpu().numpy().reshape(want_q.shape), want_q)


@pytest.mark.parametrize("K", [3200, 4224, 5248])
def test_no_unit_of_a_cut_is_left_without_steps(K):
    """Contractions of 25, 33 and 41 steps of 128 (50, 66 and 82 of 64), cut into up to 8 units in every prefill GEMM."""
    test_int4(256, K, 200, 64)
    test_fp8(256, K, 300)
    test_dense(300, K, 200)
    test_dense(300, K // 2 + 32, 200)


@pytest.mark.parametrize("N,K,M", [(12296, 1032, 32), (12296, 1032, 33), (12160, 1032, 64), (10250, 520, 65), (10100, 520, 65), (300, 512, 70), (300, 520, 70), (24584, 4104, 17)])
def test_dense_on_both_sides_of_the_wide_tiles(N, K, M):
    """17 to 128 rows where W's width or a short k decides for the tiles of 128 rows, and just before."""
    test_dense(N, K, M)


@pytest.mark.parametrize("form", ["one row for all", "rows that overlap", "one x for all groups", "a row of any stride"])
def test_rows_of_x_that_are_not_apart(form):
    """Up to 16 rows at a size that goes to the GEMM where x is an ordinary matrix: what has no tensor map runs all the same."""
    import torch
    from scratchy_b200.dense import Arena, DenseLinear
    rng = np.random.default_rng(len(form))
    draw = lambda *shape: torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda().bfloat16()
    N, K, M, groups = (6400, 1032, 5, 3) if "groups" in form else (18952, 1032, 1 if "any stride" in form else 5, 1)
    w, a = draw(groups * N, K), Arena("cuda")
    flat = draw(M * K)
    x = {"one row for all": lambda: flat[:K].expand(M, K), "rows that overlap": lambda: flat.as_strided((M, K), (8, 1)),
         "one x for all groups": lambda: flat.view(M, K), "a row of any stride": lambda: flat.as_strided((1, K), (0, 1))}[form]()
    y = torch.full((M, groups * N), float("nan"), device="cuda")
    DenseLinear(w, groups)(a, x, y, y_group=N)
    torch.cuda.synchronize()
    want = x.double() @ w.double().T
    assert float((y.double() - want).norm() / want.norm()) < 1e-5


@pytest.mark.parametrize("N,K,M", [(512, 512, 90), (512, 512, 128), (1000, 1000, 129), (1000, 1000, 200), (2056, 2048, 250), (8200, 1024, 140), (9480, 1536, 256)])
def test_fp8_on_both_sides_of_the_tiles(N, K, M):
    """65 to 256 tokens where k, the channels and the tokens decide between the GEMM for few tokens and the tiles of 128."""
    test_fp8(N, K, M)


@pytest.mark.parametrize("N,K,M", [(8200, 512, 96), (8200, 512, 97), (136, 128, 128), (1000, 1536, 128), (1000, 1600, 128)])
def test_int4_of_a_short_k_on_both_sides_of_the_prompt_tiles(N, K, M):
    """97 to 128 tokens: the prompt kernel up to a k of 1536 (tiles that are not full, cut or whole), and just beyond it."""
    test_int4(N, K, M, 64)
