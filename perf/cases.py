"""What this framework is timed at: the quantized linears alone, the Llama decode step, and prompts and decode steps of the
two sequence models, each through the calls that a program makes.

The sizes are those of the repository's own benchmark (Llama-3.2-3B and Qwen2.5-7B linears, the 3B and 1B sequence models,
contexts around 2048, batches 1 to 32) and odd ones between them.  Weights are random with magnitudes that keep activations
of order one through the depth of a model, as a trained checkpoint does."""
import math

import torch

from scratchy_b200.decode import LlamaConfig, LlamaDecoder, PagedKvCache
from scratchy_b200.engine import Engine
from scratchy_b200.layers import AffineQuantLinear, Fp8Linear, GpuWeights
from scratchy_b200.vekurax import Vekurax, VekuraxConfig
from scratchy_b200.vumipel import Vumipel, VumipelConfig

DEV = "cuda"
BF16, F64 = torch.bfloat16, torch.float64
VOCAB = 128256


def listed():
    return [
        # a linear called on its own, one token: launches and host calls count
        {"name": "int4 1 row", "kind": "int4", "rows": 1, "K": 3072, "N": 8192, "group": 64, "scales": "bf16", "bias": False},
        # a batch of sequences, or drafted tokens to verify, between the matvec's sizes and a prompt's; an odd count
        {"name": "int4 45 rows", "kind": "int4", "rows": 45, "K": 8192, "N": 3072, "group": 64, "scales": "f16", "bias": False},
        # a prompt's portion
        {"name": "int4 2048 rows", "kind": "int4", "rows": 2048, "K": 3072, "N": 8192, "group": 64, "scales": "bf16", "bias": False},
        {"name": "fp8 1 row", "kind": "fp8", "rows": 1, "K": 3584, "N": 18944, "bias": False},
        # a short prompt, with a contraction that is long for its few outputs
        {"name": "fp8 250 rows", "kind": "fp8", "rows": 250, "K": 18944, "N": 3584, "bias": False},
        # the largest portion of a prompt
        {"name": "fp8 8192 rows", "kind": "fp8", "rows": 8192, "K": 3584, "N": 18944, "bias": False},
        # chat with one user; a full batch of a server, contexts of all lengths
        {"name": "llama decode 1", "kind": "llama", "batch": 1, "context": 2048, "group": 64},
        {"name": "llama decode 32", "kind": "llama", "batch": 32, "context": 2048, "group": 64},
        {"name": "vekurax decode 8", "kind": "decode", "model": "vekurax 3b", "batch": 8, "context": 2048},
        {"name": "vekurax prompt 2000", "kind": "prompt", "model": "vekurax 3b", "batch": 1, "tokens": 2000},
        {"name": "vumipel decode 32", "kind": "decode", "model": "vumipel 3b", "batch": 32, "context": 1024},
        # the longest prompt that a step takes
        {"name": "vumipel prompt 8192", "kind": "prompt", "model": "vumipel 3b", "batch": 1, "tokens": 8192},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    kind = rng.choice(["int4", "int4", "fp8", "fp8", "llama", "decode", "prompt"])
    if kind == "int4":
        group = rng.choice([32, 64, 64, 64, 128])
        K, N = rng.choice([(3072, 3072), (3072, 1024), (3072, 8192), (8192, 3072), (128 * rng.randint(8, 80), 8 * rng.randint(64, 1200))])
        return {"kind": "int4", "rows": _log(rng, 1, 4096), "K": K, "N": N, "group": group, "scales": rng.choice(["bf16", "f16"]), "bias": rng.random() < 0.2}
    if kind == "fp8":
        K, N = rng.choice([(3584, 3584), (3584, 512), (3584, 18944), (18944, 3584), (64 * rng.randint(16, 256), 16 * rng.randint(32, 1100))])
        return {"kind": "fp8", "rows": _log(rng, 1, 8192), "K": K, "N": N, "bias": rng.random() < 0.3}
    if kind == "llama":
        return {"kind": "llama", "batch": _log(rng, 1, 32), "context": _log(rng, 100, 3000), "group": rng.choice([64, 64, 128])}
    model = rng.choice(["vekurax 3b", "vekurax 1b", "vumipel 3b"])
    if kind == "decode":
        batch = _log(rng, 1, 32)
        return {"kind": "decode", "model": model, "batch": batch, "context": _log(rng, 70, min(3000, 32768 // batch))}
    return {"kind": "prompt", "model": model, "batch": rng.choice([1, 1, 2, 3]), "tokens": _log(rng, 100, 8000)}


# ------------------------------------------------------------------------------------ inputs
def _generator(seed, *what):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + sum((i + 1) * 7919 * int(w) for i, w in enumerate(what))) & 0x7FFFFFFF)
    return g


def _randn(g, shape, mean=0.0, std=1.0, dtype=BF16):
    return torch.randn(shape, device=DEV, generator=g).mul_(std).add_(mean).to(dtype)


def _int4(g, N, K, group, dtype=BF16, std=0.02, middle=8.0):
    """Codes of eight to a word, scales and offsets per group: |N(0, std)| and -`middle` times that, the checkpoint format's
    spread.  A middle of 7.5 gives weights of mean zero, as a trained layer's are; with a mean, the depth of a model amplifies it."""
    w = torch.randint(-2 ** 31, 2 ** 31 - 1, (N, K // 8), dtype=torch.int32, device=DEV, generator=g)
    s = torch.randn((N, K // group), device=DEV, generator=g).mul_(std).abs_().add_(std / 20).to(dtype)
    b = (-middle * s.float() + torch.randn((N, K // group), device=DEV, generator=g).mul_(std / 20)).to(dtype)
    return w, s, b


def _int4_values(w, s, b, group):
    """The bf16 weights that codes, scales and offsets stand for, in 64 bits."""
    codes = torch.stack([(w >> (4 * j)) & 15 for j in range(8)], dim=-1).reshape(w.shape[0], -1).float()
    s, b = (t.to(BF16).float().repeat_interleave(group, dim=1) for t in (s, b))
    return (codes * s + b).to(BF16).to(F64)


def _int4_inputs(case, seed):
    g = _generator(seed, 1, case["rows"], case["K"], case["N"])
    parts = _int4(g, case["N"], case["K"], case["group"], BF16 if case["scales"] == "bf16" else torch.float16)
    bias = _randn(g, (case["N"],)) if case["bias"] else None
    return parts, bias, _randn(g, (case["rows"], case["K"]))


def _fp8_inputs(case, seed):
    g = _generator(seed, 2, case["rows"], case["K"], case["N"])
    w = torch.randn((case["N"], case["K"]), device=DEV, generator=g).mul_(0.02)
    scale = w.abs().amax(dim=1) / 448.0
    codes = (w / scale[:, None]).to(torch.float8_e4m3fn)
    bias = _randn(g, (case["N"],)) if case["bias"] else None
    return codes, scale, bias, _randn(g, (case["rows"], case["K"]))


def _spread(seed, batch, most):
    """Lengths of a batch: one of `most`, the others anywhere from a quarter of it up."""
    r = torch.Generator().manual_seed(1000 + int(seed))
    return [most] + torch.randint(max(1, most // 4), most + 1, (batch - 1,), generator=r).tolist()


LLAMA = dict(hidden=3072, n_layers=28, n_q_heads=24, n_kv_heads=8, head_dim=128, intermediate=8192, vocab=VOCAB)


def _llama_weights(seed, group):
    g, h = _generator(seed, 3, group), LLAMA["hidden"]
    qd, kd, ff = LLAMA["n_q_heads"] * 128, LLAMA["n_kv_heads"] * 128, LLAMA["intermediate"]
    ck = {}

    def put(name, N, K):
        # what joins the residual is scaled down with the depth, as initialisations do
        gain = 0.3 if name.endswith(("o_proj", "down_proj")) else 1.0
        ck[f"{name}.weight"], ck[f"{name}.scales"], ck[f"{name}.biases"] = _int4(g, N, K, group, std=0.2 * gain * K ** -0.5, middle=7.5)
    for i in range(LLAMA["n_layers"]):
        root = f"model.layers.{i}"
        for part, N, K in (("self_attn.q_proj", qd, h), ("self_attn.k_proj", kd, h), ("self_attn.v_proj", kd, h), ("self_attn.o_proj", h, qd),
                           ("mlp.gate_proj", ff, h), ("mlp.up_proj", ff, h), ("mlp.down_proj", h, ff)):
            put(f"{root}.{part}", N, K)
        for part in ("input_layernorm", "post_attention_layernorm"):
            ck[f"{root}.{part}.weight"] = _randn(g, (h,), 1.0, 0.1)
    ck["model.norm.weight"] = _randn(g, (h,), 1.0, 0.1)
    ck["model.embed_tokens.weight"] = _randn(g, (VOCAB, h))
    put("lm_head", VOCAB, h)
    return ck


def _llama_state(case, seed):
    """(token ids, contexts, block table, caches per layer): keys and values of the tokens before this one."""
    B, ctx, n = case["batch"], _spread(seed, case["batch"], case["context"]), LLAMA["n_layers"]
    need = [c // 16 + 1 for c in ctx]
    r = torch.Generator().manual_seed(int(seed) + 17)
    ids = torch.randint(0, VOCAB, (B,), generator=r)
    free = (B + torch.randperm(sum(need) - B, generator=r)).tolist()
    table = torch.zeros((B, max(need)), dtype=torch.int32)
    for b in range(B):                                   # a sequence's newest block is block b, the others lie anywhere
        blocks = [free.pop() for _ in range(need[b] - 1)] + [b]
        table[b] = torch.tensor(blocks + [b] * (max(need) - need[b]))
    g = _generator(seed, 4)
    caches = [[_randn(g, (sum(need), LLAMA["n_kv_heads"], 16, 128)) for _ in range(n)] for _ in range(2)]
    return ids, ctx, table, caches


def _vumipel_config():
    """Llama-3.2-3B's width, feed-forward, vocabulary and number of layer runs; one latent attention to three matrix memories."""
    mem = {"type": "mlstm", "mixer": {"heads": 12, "dim": 128, "vdim": 256, "gate_cap": 15.0}}
    att = {"type": "latent_attention", "mixer": {"heads": 24, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 1536,
                                                 "rot": {"base": 5e5, "dims": 64}, "scale": 192 ** -0.5}}
    layers = [{**(att if i % 4 == 3 else mem), "mlp": {"kind": "dense", "ff": 8192, "limit": 7.0}} for i in range(24)]
    return {"architecture": "Vumipel", "layers": layers, "loop": {"start": 8, "stop": 12, "times": 2}, "norm": {"eps": 1e-5}, "vocab": VOCAB, "width": 3072}


def _vekurax_config(size):
    """Llama-3.2-3B's or 1B's width, feed-forward, vocabulary, attention heads and layer runs; the 3B runs four layers twice."""
    width, heads, dim, rheads, runs, own = {"3b": (3072, 24, 128, 12, 28, 24), "1b": (2048, 32, 64, 8, 16, 16)}[size]
    layer = {"type": "parallel", "mlp": {"kind": "dense", "ff": 8192}, "mixer": {
        "left": {"heads": heads, "kv_heads": 8, "dim": dim, "vdim": dim, "conv": 4, "bias_max": 1024, "scale": dim ** -0.5, "mask": {"size": 4096, "keep_first": 64}},
        "left_scale": 0.8, "right": {"heads": rheads, "dim": 128, "vdim": 256, "decay": [math.exp(-2.0 ** (-8.0 * (i + 1) / rheads)) for i in range(rheads)]},
        "right_scale": 0.8}}
    layers = [layer if i < own else {**layer, "weights_of": i - own + 8} for i in range(runs)]
    return {"architecture": "Vekurax", "layers": layers, "norm": {"eps": 1e-5}, "vocab": VOCAB, "width": width}


def _sequence_config(name):
    design, size = name.split()
    return _vumipel_config() if design == "vumipel" else _vekurax_config(size)


def _sequence_weights(cfg, seed):
    g, W, out = _generator(seed, 5), cfg["width"], {}

    def mat(name, rows, cols, gain=1.0):
        out[name] = _randn(g, (rows, cols), 0.0, gain * cols ** -0.5)

    def vec(name, n, mean=0.0, std=0.1):
        out[name] = _randn(g, (n,), mean, std)

    def tanh(name, alpha):
        vec(name, W, 1.0)
        vec(name + ".b", W)
        out[name + ".alpha"] = torch.tensor(alpha, device=DEV, dtype=BF16)
    vekurax = cfg["architecture"] == "Vekurax"
    out["embed"] = _randn(g, (cfg["vocab"], W), 0.0, 1.0 if vekurax else 0.1)
    if cfg.get("loop"):
        mat("loop.in", W, 2 * W)
        out["loop.step"] = _randn(g, (cfg["loop"]["times"], W), 0.0, 0.1)
    for i, spec in enumerate(cfg["layers"]):
        if "weights_of" in spec:
            continue
        ff = spec["mlp"]["ff"]
        mat(f"l{i}.mlp.gate", ff, W)
        mat(f"l{i}.mlp.up", ff, W)
        mat(f"l{i}.mlp.down", W, ff)
        if vekurax:
            tanh(f"l{i}.norm1", 0.5)
            m, p = spec["mixer"]["left"], f"l{i}.mix.left."
            H, dim = m["heads"], m["dim"]
            for part, n in (("q", H * dim), ("k", m["kv_heads"] * dim)):
                mat(p + part, n, W)
                vec(p + part + ".norm", n, 1.0)
                out[p + part + ".conv"] = _randn(g, (n, m["conv"]), 0.25, 0.2)
            out[p + "rel"] = _randn(g, (32, H), 0.0, 0.5)
            mat(p + "g", H, W)
            mat(p + "o", W, H * dim)
            m, p = spec["mixer"]["right"], f"l{i}.mix.right."
            H = m["heads"]
            for part, n in (("q", H * m["dim"]), ("k", H * m["dim"]), ("v", H * m["vdim"]), ("g", H * m["vdim"])):
                mat(p + part, n, W)
            vec(p + "norm", H * m["vdim"], 1.0)
            mat(p + "o", W, H * m["vdim"])
            continue
        for part in ("norm1", "norm1b", "norm2", "norm2b"):
            vec(f"l{i}.{part}", W)
        m, p = spec["mixer"], f"l{i}.mix."
        H = m["heads"]
        if spec["type"] == "mlstm":
            for part, n in (("q", H * m["dim"]), ("k", H * m["dim"]), ("v", H * m["vdim"]), ("g", H * m["vdim"])):
                mat(p + part, n, W)
            # keys that lean towards the queries, as trained ones do: the readout is divided by what the two have in common
            out[p + "k"] = (0.8 * out[p + "q"].float() + 0.6 * out[p + "k"].float()).to(BF16)
            mat(p + "i", H, W)
            mat(p + "f", H, W)
            vec(p + "i.b", H, -1.0, 0.5)
            vec(p + "f.b", H, 3.0, 1.0)
            vec(p + "norm", H * m["vdim"], 1.0)
            mat(p + "o", W, H * m["vdim"])
        else:
            mat(p + "dq", m["q_rank"], W)
            vec(p + "dq.norm", m["q_rank"], 1.0)
            mat(p + "uq", H * (m["dim"] + m["rot_dim"]), m["q_rank"])
            mat(p + "dkv", m["kv_rank"] + m["rot_dim"], W)
            vec(p + "dkv.norm", m["kv_rank"], 1.0)
            mat(p + "uk", H * m["dim"], m["kv_rank"])
            mat(p + "uv", H * m["vdim"], m["kv_rank"])
            mat(p + "g", H * m["vdim"], W)
            mat(p + "o", W, H * m["vdim"])
    if vekurax:
        tanh("final.norm", 0.5)
    else:
        vec("final.norm", W)
    return out


def _sequence_tokens(case, seed):
    """Token ids of every sequence: the prompts, or the contexts and one token more."""
    r = torch.Generator().manual_seed(int(seed) + 29)
    if case["kind"] == "decode":
        lengths = [c + 1 for c in _spread(seed, case["batch"], case["context"])]
    else:                                                # prompts that fill a step together, of unequal lengths
        n, b = case["tokens"], case["batch"]
        lengths = [n // b + (i - b // 2) * (n // (4 * b)) for i in range(b)]
        lengths[-1] += n - sum(lengths)
    return [torch.randint(0, VOCAB, (n,), generator=r).tolist() for n in lengths]


def _sequence_model(case, seed, max_tokens):
    cfg = _sequence_config(case["model"])
    cls, config = (Vekurax, VekuraxConfig) if cfg["architecture"] == "Vekurax" else (Vumipel, VumipelConfig)
    return cls(config.from_dict(cfg), GpuWeights(_sequence_weights(cfg, seed)), DEV, "bfloat16", max_tokens=max_tokens, max_sequences=case["batch"])


# ------------------------------------------------------------------------------------ the calls
def prepare(case, seed):
    kind = case["kind"]
    if kind == "int4":
        (w, s, b), bias, x = _int4_inputs(case, seed)
        lin = AffineQuantLinear.from_tensors(w, s, b, case["group"], 4, bias)
    elif kind == "fp8":
        codes, scale, bias, x = _fp8_inputs(case, seed)
        lin = Fp8Linear.from_tensors(codes, scale, bias)
    if kind in ("int4", "fp8"):
        out = torch.empty((case["rows"], case["N"]), dtype=BF16, device=DEV)
        return {"kind": kind, "lin": lin, "x": x, "out": out, "ws": torch.empty(max(16, lin.workspace_bytes(case["rows"])), dtype=torch.uint8, device=DEV)}
    if kind == "llama":
        ids, ctx, table, (k, v) = _llama_state(case, seed)
        cfg = LlamaConfig(**LLAMA, group_size=case["group"])
        model = LlamaDecoder(cfg, _llama_weights(seed, case["group"]), DEV, max_pos=4096)
        cache = PagedKvCache(cfg, int(k[0].shape[0]), 16, DEV)
        buf = model.buffers(case["batch"], int(table.shape[1]))
        c = torch.tensor(ctx, dtype=torch.int32)
        buf.ids.copy_(ids.to(torch.int32))
        buf.positions.copy_(c)
        buf.seq_used_k.copy_(c + 1)
        buf.slot_mapping.copy_(torch.arange(case["batch"], dtype=torch.int32) * 16 + c % 16)
        buf.block_table.copy_(table)
        graph = model.capture(buf, cache)
        for mine, theirs in zip(cache.k + cache.v, k + v):
            mine.copy_(theirs)
        newest = [t[:case["batch"]] for t in cache.k + cache.v]
        return {"kind": kind, "graph": graph, "out": [buf.logits] + newest, "keep": (model, cache, buf)}
    tokens = _sequence_tokens(case, seed)
    if kind == "prompt":
        model = _sequence_model(case, seed, sum(len(t) for t in tokens))
        entries = [(f"prompt {i}", t, [len(t) - 1]) for i, t in enumerate(tokens)]
        return {"kind": kind, "engine": Engine(model, step_tokens=8192, max_batch=case["batch"]), "entries": entries}
    model = _sequence_model(case, seed, sum(len(t) for t in tokens) + 64 * case["batch"])
    seqs = [model.table.open(i) for i in range(case["batch"])]
    for seq, t in zip(seqs, tokens):
        model.forward([(seq, t[:-1])], [[]])
        model.table.extend(seq, 1)
    step = model.decode_graph(case["batch"], max(len(t) for t in tokens))
    step.inputs.fill([(seq, t[-1:]) for seq, t in zip(seqs, tokens)], list(range(case["batch"])))
    return {"kind": kind, "step": step, "keep": model}


def run(state):
    kind = state["kind"]
    if kind in ("int4", "fp8"):
        return state["lin"].forward(state["x"], out=state["out"], workspace=state["ws"])
    if kind == "llama":
        state["graph"].replay()
        return state["out"]
    if kind == "decode":
        state["step"].graph.replay()
        return state["step"].logits
    return state["engine"].run_step(state["entries"], end=[name for name, _, _ in state["entries"]])


# ------------------------------------------------------------------------------------ what a pass cannot do without
def _sequence_work(case):
    cfg = _sequence_config(case["model"])
    W, embed = cfg["width"], VOCAB * cfg["width"]
    decode = case["kind"] == "decode"
    # (new tokens, tokens in all) of every sequence; the lengths of a seed differ little in their sum
    if decode:
        seqs = [(1, case["context"])] + [(1, 0.625 * case["context"])] * (case["batch"] - 1)
    else:
        seqs = [(case["tokens"] / case["batch"],) * 2] * case["batch"]
    rows = sum(n for n, _ in seqs)
    pairs = sum(n * (t - n) + n * (n + 1) / 2 for n, t in seqs)
    weights, flops, state = embed, 2.0 * embed * case["batch"], 0.0
    loop = cfg.get("loop") or {"start": 0, "stop": 0, "times": 1}
    if cfg.get("loop"):
        weights += 2 * W * W
        flops += 2.0 * rows * 2 * W * W * loop["times"]
    for i, spec in enumerate(cfg["layers"]):
        m, times = spec["mixer"], loop["times"] if loop["start"] <= i < loop["stop"] else 1
        n, mixing, kept = 3 * W * spec["mlp"]["ff"], 0.0, 0.0
        if cfg["architecture"] == "Vekurax":
            left, right = m["left"], m["right"]
            n += W * (left["dim"] * (2 * left["heads"] + left["kv_heads"]) + left["heads"])
            mixing += 4.0 * left["heads"] * left["dim"] * pairs
            kept += left["kv_heads"] * left["dim"] * 2 * sum(t for _, t in seqs)
            mem = right
            n += W * mem["heads"] * (2 * mem["dim"] + 3 * mem["vdim"])
        elif spec["type"] == "mlstm":
            mem = m
            n += W * mem["heads"] * (2 * mem["dim"] + 3 * mem["vdim"] + 2)
        else:
            mem, H = None, m["heads"]
            per = m["dim"] + m["rot_dim"]
            n += W * (m["q_rank"] + m["kv_rank"] + m["rot_dim"] + 2 * H * m["vdim"]) + m["q_rank"] * H * per + m["kv_rank"] * H * (m["dim"] + m["vdim"])
            mixing += 2.0 * H * (per + m["vdim"] if not decode else 2 * m["kv_rank"] + m["rot_dim"]) * pairs
            kept += (m["kv_rank"] + m["rot_dim"]) * 2 * sum(t for _, t in seqs)
        if mem is not None:
            mixing += 4.0 * rows * mem["heads"] * mem["dim"] * mem["vdim"]
            kept += mem["heads"] * mem["dim"] * mem["vdim"] * 4 * len(seqs) * (2 if decode else 1)
        if "weights_of" not in spec:
            weights += n
        flops += times * (2.0 * rows * n + mixing)
        state += times * kept
    return {"bytes": 2.0 * weights + state + 4.0 * VOCAB * case["batch"], "flops": flops}


def work(case):
    kind = case["kind"]
    if kind == "int4":
        M, K, N = case["rows"], case["K"], case["N"]
        return {"bytes": N * K / 2 + 4 * N * K / case["group"] + 2 * M * (K + N), "flops": 2.0 * M * N * K}
    if kind == "fp8":
        M, K, N = case["rows"], case["K"], case["N"]
        return {"bytes": N * K + 4 * N + 2 * M * (K + N), "flops": 2.0 * M * N * K}
    if kind == "llama":
        h, qd, kd, ff = 3072, 3072, 1024, 8192
        weights = 28 * (h * (2 * qd + 2 * kd) + 3 * h * ff) + VOCAB * h
        tokens = case["context"] + (case["batch"] - 1) * 0.625 * case["context"]
        return {"bytes": weights * (0.5 + 4 / case["group"]) + 28 * tokens * 2 * kd * 2 + case["batch"] * 2 * VOCAB,
                "flops": 2.0 * weights * case["batch"] + 28 * 4.0 * qd * tokens}
    return _sequence_work(case)


def tolerance(case):
    return {"int4": {"rel": 4e-3}, "fp8": {"rel": 4e-3}, "llama": {"rel": 0.03, "max": 0.5}, "decode": {"rel": 0.03, "max": 0.5}, "prompt": {"rel": 0.03, "max": 0.5}}[case["kind"]]


# ------------------------------------------------------------------------------------ the same in 64 bits
def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _e4m3(v):
    """Nearest e4m3 value, halves away from zero; |v| <= 448."""
    a = v.abs()
    step = torch.exp2(torch.floor(torch.log2(a.clamp_min(2.0 ** -6))) - 3)
    return torch.sign(v) * (torch.floor(a / step + 0.5) * step).clamp_max(448.0)


def _rows_of(pieces):
    at = 0
    for n in pieces:
        yield slice(at, at + n)
        at += n


def _softmax_rows(q, k, v, scale, seen, bias=None, block=1024):
    """Attention of the queries at the last len(q) places of the keys' sequence, a block of queries at a time."""
    T, n = k.shape[0], q.shape[0]
    out = []
    for lo in range(0, n, block):
        i = torch.arange(T - n + lo, T - n + min(n, lo + block), device=DEV)[:, None]
        j = torch.arange(T, device=DEV)[None, :]
        s = q[lo:lo + block] @ k.T * scale
        if bias is not None:
            s = s + bias[(i - j).clamp_min(0)]
        out.append(torch.softmax(s.masked_fill(~seen(i, j), -math.inf), dim=1) @ v)
    return torch.cat(out)


def _memory_rows(q, k, v, f, i=None, last=0, block=1024):
    """One head's matrix memory in closed form.  f, i: log gates per token (i None: one, without a normaliser)."""
    T, F, out = q.shape[0], torch.cumsum(f, 0), []
    for lo in range(last, T, block):
        hi = min(T, lo + block)
        t, s = torch.arange(lo, hi, device=DEV)[:, None], torch.arange(hi, device=DEV)[None, :]
        D = F[lo:hi, None] - F[None, :hi] + (0.0 if i is None else i[None, :hi])
        D = D.masked_fill(s > t, -math.inf)
        dots = q[lo:hi] @ k[:hi].T
        if i is None:
            out.append((torch.exp(D) * dots) @ v[:hi])
            continue
        top = torch.maximum(F[lo:hi], D.amax(dim=1))
        P = torch.exp(D - top[:, None]) * dots
        out.append(P @ v[:hi] / (torch.maximum(P.sum(dim=1).abs(), torch.exp(-top)) + 1e-6)[:, None])
    return torch.cat(out)


def _exact_llama(case, seed):
    ids, ctx, table, (ck, cv) = _llama_state(case, seed)
    w, group, B, eps = _llama_weights(seed, case["group"]), case["group"], case["batch"], 1e-5
    get = lambda name: _int4_values(w[f"{name}.weight"], w[f"{name}.scales"], w[f"{name}.biases"], group)
    norm = lambda x, name: _unit(x, eps) * w[name].to(F64)
    pos = torch.tensor(ctx, device=DEV, dtype=F64)
    ang = pos[:, None] * 500000.0 ** (-torch.arange(64, device=DEV, dtype=F64) / 64)[None, :]
    cos, sin = ang.cos()[:, None, :], ang.sin()[:, None, :]

    def rope(z):
        a, b = z[..., :64], z[..., 64:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)
    x = w["model.embed_tokens.weight"][ids.to(DEV)].to(F64)
    newest = [[], []]
    for i in range(LLAMA["n_layers"]):
        root = f"model.layers.{i}"
        h = norm(x, f"{root}.input_layernorm.weight")
        q = rope((h @ get(f"{root}.self_attn.q_proj").T).view(B, 24, 128))
        k = rope((h @ get(f"{root}.self_attn.k_proj").T).view(B, 8, 128))
        v = (h @ get(f"{root}.self_attn.v_proj").T).view(B, 8, 128)
        heads = []
        for b in range(B):
            blocks = table[b, :ctx[b] // 16 + 1].long().to(DEV)
            K, V = (torch.cat([c[blocks].transpose(0, 1).reshape(8, -1, 128)[:, :ctx[b]].to(F64), n[b][:, None]], dim=1) for c, n in ((ck[i], k), (cv[i], v)))
            p = torch.softmax(q[b].view(8, 3, 128) @ K.transpose(1, 2) / math.sqrt(128.0), dim=-1)
            heads.append((p @ V).reshape(-1))
        for to, c, n in ((newest[0], ck[i], k), (newest[1], cv[i], v)):
            c = c[:B].to(F64)
            for b in range(B):
                c[b, :, ctx[b] % 16] = n[b]
            to.append(c)
        x = x + torch.stack(heads) @ get(f"{root}.self_attn.o_proj").T
        h = norm(x, f"{root}.post_attention_layernorm.weight")
        act = torch.nn.functional.silu(h @ get(f"{root}.mlp.gate_proj").T) * (h @ get(f"{root}.mlp.up_proj").T)
        x = x + act @ get(f"{root}.mlp.down_proj").T
    return [norm(x, "model.norm.weight") @ get("lm_head").T] + newest[0] + newest[1]


def _exact_sequences(case, seed):
    cfg, tokens = _sequence_config(case["model"]), _sequence_tokens(case, seed)
    w, eps, lengths = _sequence_weights(cfg, seed), cfg["norm"]["eps"], [len(t) for t in tokens]
    get = lambda name: w[name].to(F64)
    pieces = list(_rows_of(lengths))
    x = get("embed")[torch.tensor([t for seq in tokens for t in seq], device=DEV)]

    def window(h, p, m):
        H, G, dim, taps, out = m["heads"], m["kv_heads"], m["dim"], m["conv"], torch.empty((h.shape[0], m["heads"] * m["dim"]), dtype=F64, device=DEV)
        q, k, gate = h @ get(p + "q").T, h @ get(p + "k").T, torch.sigmoid(h @ get(p + "g").T)
        size, first = m["mask"]["size"], m["mask"]["keep_first"]
        rows = 32
        n = torch.arange(max(lengths), device=DEV, dtype=F64)
        far = 16 + torch.floor(torch.log(n.clamp_min(16) / 16) / math.log(m["bias_max"] / 16) * (rows - 16) + 1e-12)
        bias = get(p + "rel")[torch.where(n < 16, n, far.clamp_max(rows - 1)).long()]

        def conv(u, c):
            u = torch.cat([torch.zeros((taps - 1, u.shape[1]), dtype=F64, device=DEV), u])
            return sum(c[:, j] * u[j:j + u.shape[0] - taps + 1] for j in range(taps))
        for rows in pieces:
            a, b = conv(q[rows], get(p + "q.conv")), conv(k[rows], get(p + "k.conv"))
            qn, kn = _unit(a, eps) * get(p + "q.norm"), _unit(b, eps) * get(p + "k.norm")
            for i in range(H):
                c, d = slice(i * dim, (i + 1) * dim), slice(i // (H // G) * dim, (i // (H // G) + 1) * dim)
                out[rows, c] = _softmax_rows(qn[:, c], kn[:, d], b[:, d], m["scale"], lambda i, j: (j <= i) & ((i - j < size) | (j < first)), bias[:, i]) * gate[rows, i:i + 1]
        return out @ get(p + "o").T

    def lightning(h, p, m):
        H, dim, vdim, out = m["heads"], m["dim"], m["vdim"], torch.empty((h.shape[0], m["heads"] * m["vdim"]), dtype=F64, device=DEV)
        q, k, v = (torch.nn.functional.silu(h @ get(p + n).T) for n in "qkv")
        for rows in pieces:
            for a in range(H):
                c, d = slice(a * dim, (a + 1) * dim), slice(a * vdim, (a + 1) * vdim)
                f = torch.full((rows.stop - rows.start,), math.log(m["decay"][a]), dtype=F64, device=DEV)
                out[rows, d] = _memory_rows(q[rows, c], k[rows, c], v[rows, d], f)
        return (_unit(out, eps) * get(p + "norm") * torch.sigmoid(h @ get(p + "g").T)) @ get(p + "o").T

    def mlstm(h, p, m):
        H, dim, vdim, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = (h @ get(p + n).T for n in "qkv")
        i = cap * torch.tanh((h @ get(p + "i").T + get(p + "i.b")) / cap)
        f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ get(p + "f").T + get(p + "f.b")) / cap))
        out = torch.empty((h.shape[0], H, vdim), dtype=F64, device=DEV)
        for rows in pieces:
            for a in range(H):
                c, d = slice(a * dim, (a + 1) * dim), slice(a * vdim, (a + 1) * vdim)
                out[rows, a] = _memory_rows(q[rows, c] * dim ** -0.5, k[rows, c], v[rows, d], f[rows, a], i[rows, a])
        out = _unit(out, eps).reshape(h.shape[0], -1) * get(p + "norm")
        return (out * torch.sigmoid(h @ get(p + "g").T)) @ get(p + "o").T

    def rotate(z, dims, base):
        """z [T, ..., D]: dimension 2i goes with 2i + 1."""
        pos = torch.arange(z.shape[0], device=DEV, dtype=F64)
        ang = (pos[:, None] * base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=F64) / dims)).view((z.shape[0],) + (1,) * (z.dim() - 2) + (-1,))
        u, v = z[..., 0:dims:2], z[..., 1:dims:2]
        return torch.cat([torch.stack([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()], dim=-1).flatten(-2), z[..., dims:]], dim=-1)

    def latent(h, p, m):
        H, dim, kvr, vdim, rot = m["heads"], m["dim"], m["kv_rank"], m["vdim"], m["rot"]
        q = (_unit(h @ get(p + "dq").T, eps) * get(p + "dq.norm")) @ get(p + "uq").T
        dkv = h @ get(p + "dkv").T
        c = _unit(dkv[:, :kvr], eps) * get(p + "dkv.norm")
        k, v = c @ get(p + "uk").T, c @ get(p + "uv").T
        out = torch.empty((h.shape[0], H * vdim), dtype=F64, device=DEV)
        for rows in pieces:
            qs = q[rows].view(-1, H, dim + m["rot_dim"])
            q_rot, k_rot = rotate(qs[:, :, dim:], rot["dims"], rot["base"]), rotate(dkv[rows, kvr:], rot["dims"], rot["base"])
            for a in range(H):
                qa, ka = torch.cat([qs[:, a, :dim], q_rot[:, a]], 1), torch.cat([k[rows, a * dim:(a + 1) * dim], k_rot], 1)
                out[rows, a * vdim:(a + 1) * vdim] = _softmax_rows(qa, ka, v[rows, a * vdim:(a + 1) * vdim], m["scale"], lambda i, j: j <= i)
        return (out * torch.sigmoid(h @ get(p + "g").T)) @ get(p + "o").T

    def squash(x, name):
        return torch.tanh(float(w[name + ".alpha"]) * x) * get(name) + get(name + ".b")
    wanted = [rows.stop - 1 for rows in pieces]
    if cfg["architecture"] == "Vekurax":
        for i, spec in enumerate(cfg["layers"]):
            j, m = spec.get("weights_of", i), spec["mixer"]
            h = squash(x, f"l{j}.norm1")
            y = m["left_scale"] * window(h, f"l{j}.mix.left.", m["left"])
            y += m["right_scale"] * lightning(h, f"l{j}.mix.right.", m["right"])
            y += (torch.nn.functional.gelu(h @ get(f"l{j}.mlp.gate").T, approximate="tanh") * (h @ get(f"l{j}.mlp.up").T)) @ get(f"l{j}.mlp.down").T
            x = x + y
        return squash(x[wanted], "final.norm") @ get("embed").T
    around = lambda x, name: _unit(x, eps) * (1.0 + get(name))
    loop, x0 = cfg["loop"], x
    order = [(i, None) for i in range(loop["start"])]
    order += [(i, t if i == loop["start"] else None) for t in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
    order += [(i, None) for i in range(loop["stop"], len(cfg["layers"]))]
    for i, t in order:
        spec = cfg["layers"][i]
        if t is not None:
            x = torch.cat([x, x0], dim=1) @ get("loop.in").T + get("loop.step")[t]
        mixer = mlstm if spec["type"] == "mlstm" else latent
        x = x + around(mixer(around(x, f"l{i}.norm1"), f"l{i}.mix.", spec["mixer"]), f"l{i}.norm1b")
        h, limit = around(x, f"l{i}.norm2"), spec["mlp"]["limit"]
        g = (h @ get(f"l{i}.mlp.gate").T).clamp_max(limit)
        u = (h @ get(f"l{i}.mlp.up").T).clamp(-limit, limit)
        x = x + around((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ get(f"l{i}.mlp.down").T, f"l{i}.norm2b")
    return around(x[wanted], "final.norm") @ get("embed").T


def exact(case, seed):
    kind = case["kind"]
    if kind == "int4":
        (w, s, b), bias, x = _int4_inputs(case, seed)
        y = x.to(F64) @ _int4_values(w, s, b, case["group"]).T
        return y if bias is None else y + bias.to(F64)
    if kind == "fp8":
        codes, scale, bias, x = _fp8_inputs(case, seed)
        # the format's own rule for activations: one f32 scale per token, the quotient rounded to e4m3
        a = (x.float().abs().amax(dim=1) * (1.0 / 448.0)).clamp(1.0 / 448.0 ** 2, 448.0)
        xq = _e4m3((x.float() * (1.0 / a)[:, None]).clamp(-448.0, 448.0).to(F64))
        y = xq @ codes.float().to(F64).T * a.to(F64)[:, None] * scale.to(F64)
        return y if bias is None else y + bias.to(F64)
    return _exact_llama(case, seed) if kind == "llama" else _exact_sequences(case, seed)
