"""The workloads that this framework's speed is judged by, through its public entry points.

A case is a dict of plain values; its "family" says which entry points it goes through:

  generate   QWen3AWQInfer.generateResponse: a prompt in host memory in, greedy ids in host memory out
  step       one token through a stack of decoder layers by the per-operator entry points, as a host that schedules
             the operators itself runs it: embedding, RMSNorm + Wqkv + RoPE + KV append, attention over the cache,
             Wo + residual, RMSNorm + W1 + GeLU, W2 + residual, final norm + unembedding + arg-max
  linear     the dequantising matrix-vector product of single AWQ linears, one after the other (one per layer)
  rows       the W4A16 contraction of a block of activation rows (prompt blocks, batched rows)
  attention  causal attention of a block of prompt rows over the KV cache

Sizes are those of the repository's configurations: the Qwen3-8B-shape decoder (hidden 4096, 32 heads, inter 12288,
vocabulary 151936, 36 layers), the four-layer model of the tests, the row sweep 16 .. 2048 of the benchmark, and generic
multiples of 128, which is what the operators take.
"""
import importlib
import math
import os
import tempfile

import numpy as np
import torch

PACKAGE = "cuda-kernel-qwen3-8b-awq_b200"

MODELS = {
    "full": dict(hidden=4096, inter=12288, heads=32, head_dim=128, layers=36, vocab=151936, max_pos=8192, rope_base=1e6),
    "small": dict(hidden=512, inter=1536, heads=4, head_dim=128, layers=4, vocab=2176, max_pos=512, rope_base=1e4),
}
H, HEADS, INTER, VOCAB = 4096, 32, 12288, 151936
CODE_RMS = 4.72   # root mean square of code - zero point: codes uniform in 0..15, zero points in 6..9


def _pkg():
    return importlib.import_module(PACKAGE)


def _ops():
    return importlib.import_module(PACKAGE + ".ops")


# ---- what is measured ----------------------------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest model and a handful of tokens: launches, host work and the latency of one pass
        {"name": "generate small 6+8", "family": "generate", "model": "small", "prompt": 6, "new": 8, "cluster": 0},
        # the reference's own use: a chat-sized prompt and a short answer
        {"name": "generate 128+20", "family": "generate", "model": "full", "prompt": 128, "new": 20, "cluster": 0},
        # a document with a ragged length and a short answer: the prompt phase dominates
        {"name": "generate 4001+32", "family": "generate", "model": "full", "prompt": 4001, "new": 32, "cluster": 0},
        # a few words and a long answer: the decode loop dominates; head groups as clusters, as the benchmark sets it
        {"name": "generate 11+112", "family": "generate", "model": "full", "prompt": 11, "new": 112, "cluster": 1},
        # a host that calls the operators itself: six layers and the unembedding at position 511, dependent launch on
        {"name": "step 6 layers at 511", "family": "step", "layers": 6, "pos": 511, "pdl": True},
        # one small linear: what a single call costs
        {"name": "linear 1536x512", "family": "linear", "out": 1536, "in": 512, "count": 1, "epilogue": "gelu", "integral": True,
         "noalloc": False},
        # the single-linear configuration, one matrix per layer so that they come from HBM as in a model
        {"name": "linear 4096x4096", "family": "linear", "out": 4096, "in": 4096, "count": 36, "epilogue": "store", "integral": True,
         "noalloc": False},
        # batched rows: a handful of sequences, a batch through the unembedding, a ragged block with fractional zero
        # points (what a checkpoint converted from another scheme has), and a full prompt block
        {"name": "rows 16 12288x4096", "family": "rows", "rows": 16, "out": 12288, "in": 4096, "count": 8, "integral": True},
        {"name": "rows 64 151936x4096", "family": "rows", "rows": 64, "out": 151936, "in": 4096, "count": 1, "integral": True},
        {"name": "rows 300 4096x12288", "family": "rows", "rows": 300, "out": 4096, "in": 12288, "count": 4, "integral": False},
        {"name": "rows 2048 12288x4096", "family": "rows", "rows": 2048, "out": 12288, "in": 4096, "count": 1, "integral": True},
        # the second block of a 4001-token prompt
        {"name": "attention 1953 at 2048", "family": "attention", "heads": 32, "pos0": 2048, "rows": 1953},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng):
    """A linear of the model, a row-split share of one, or a generic one."""
    kind = rng.random()
    if kind < 0.45:
        return rng.choice([(3 * H, H), (H, H), (INTER, H), (H, INTER)])
    if kind < 0.6:
        n = rng.choice([2, 4, 8])
        return rng.choice([(3 * H // n, H), (H, H // n), (INTER // n, H), (H, INTER // n)])
    if kind < 0.7:
        return VOCAB, H
    return 128 * _log_int(rng, 1, 128), 128 * _log_int(rng, 1, 96)


def _count(rng, out, inp, most):
    """How many matrices of a shape one pass goes through: one to `most`, 300 MB of packed weights at the largest."""
    return max(1, min(rng.randint(1, most), int(300e6 / (out * inp / 2))))


def draw(rng):
    family = rng.choices(["generate", "step", "linear", "rows", "attention"], [4, 1, 2, 4, 1])[0]
    if family == "generate":
        model = "small" if rng.random() < 0.25 else "full"
        prompt = _log_int(rng, 1, 300 if model == "small" else 4000)
        new = _log_int(rng, 1, 96 if prompt < 600 else 24)
        return {"family": family, "model": model, "prompt": prompt, "new": new, "cluster": rng.choice([0, 1])}
    if family == "step":
        return {"family": family, "layers": rng.randint(1, 6), "pos": _log_int(rng, 1, 8192) - 1, "pdl": rng.random() < 0.5}
    if family == "linear":
        out, inp = _shape(rng)
        noalloc = out <= 16384 and rng.random() < 0.25
        epilogue = "store" if noalloc else rng.choice(["store", "gelu", "argmax"])
        return {"family": family, "out": out, "in": inp, "count": _count(rng, out, inp, 36), "epilogue": epilogue,
                "integral": rng.random() < 0.75, "noalloc": noalloc}
    if family == "rows":
        out, inp = _shape(rng)
        rows = _log_int(rng, 2, 200 if out == VOCAB else 2500)
        return {"family": family, "rows": rows, "out": out, "in": inp, "count": _count(rng, out, inp, 1 if rows > 256 else 8),
                "integral": rng.random() < 0.75}
    return {"family": family, "heads": rng.choice([4, 8, 16, 32]), "pos0": rng.choice([0, 2048, rng.randint(1, 4096)]),
            "rows": _log_int(rng, 2, 2048)}


# ---- inputs --------------------------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _codes(g, out, inp):
    return torch.randint(0, 256, (out * inp // 2,), dtype=torch.uint8, device="cuda", generator=g)


def _scales(g, n, rms):
    """Group scales for weights of the given root mean square, spread by a factor of two as a trained model's are."""
    return ((0.67 + 0.66 * torch.rand(n, device="cuda", generator=g)) * (rms / CODE_RMS)).half()


def _zeros(g, n, integral=True):
    if integral:
        return torch.randint(6, 10, (n,), device="cuda", generator=g).half()
    return (7.5 + torch.randn(n, device="cuda", generator=g)).half()


def _normal(g, *shape, mean=0.0, std=1.0):
    return (mean + std * torch.randn(*shape, device="cuda", generator=g)).half()


# Weights of a stack of layers keep activations near one and let a layer add a tenth to the residual stream; the unembedding is
# the embedding with its vocabulary turned by some places.  The next-token distribution is then peaked, as a trained
# model's is, and the greedy ids do not hang on the last bit of a logit, which they do with unrelated random matrices.
def _layer_matrices(g, hidden, inter):
    for stem, out, inp, gain in (("wqkv", 3 * hidden, hidden, 1.0), ("wo", hidden, hidden, 0.1), ("w1", inter, hidden, 1.0),
                                 ("w2", hidden, inter, 0.1)):
        yield stem, out, inp, _codes(g, out, inp), _scales(g, out // 128, gain / math.sqrt(inp)), _zeros(g, out // 128)


def _embeddings(g, hidden, vocab):
    emb = _codes(g, hidden, vocab)
    unemb = torch.roll(emb.view(hidden, vocab // 2), 501, 1).reshape(-1)
    return ((emb, _scales(g, hidden // 128, 1.0), _zeros(g, hidden // 128)),
            (unemb, _scales(g, vocab // 128, 1.0 / math.sqrt(hidden)), _zeros(g, vocab // 128)))


_ENGINES = {}


def _engine(model, cluster):
    """A program loads its model once and keeps it for all prompts: one handle for a configuration and process."""
    if (model, cluster) not in _ENGINES:
        cfg = MODELS[model]
        g = _generator(1)
        with tempfile.TemporaryDirectory() as d:
            def write(name, t):
                t.cpu().numpy().tofile(os.path.join(d, name + ".bin"))

            for i in range(cfg["layers"]):
                for stem, _, _, packed, scale, zp in _layer_matrices(g, cfg["hidden"], cfg["inter"]):
                    write("layer_%d_%s" % (i, stem), packed)
                    stem = "bqkv" if stem == "wqkv" else stem
                    write("layer_%d_%s_scale" % (i, stem), scale)
                    write("layer_%d_%s_zp" % (i, stem), zp)
                write("rms_norm_gamma_%d" % i, _normal(g, cfg["hidden"], mean=1.0, std=0.02))
            emb, unemb = _embeddings(g, cfg["hidden"], cfg["vocab"])
            for stem, short, (packed, scale, zp) in (("word_embedding", "word_embed", emb), ("unembed", "unembed", unemb)):
                write(stem, packed)
                write(short + "_scale", scale)
                write(short + "_zp", zp)
            del emb, unemb, packed
            torch.cuda.empty_cache()
            _ENGINES[model, cluster] = _pkg().QWen3AWQInfer(d, keep_logits=1, cluster=cluster, **cfg)
    return _ENGINES[model, cluster]


def _rope_tables(max_pos, base):
    inv = base ** (-torch.arange(0, 64, device="cuda", dtype=torch.float64) / 64.0)
    angle = torch.arange(max_pos, device="cuda", dtype=torch.float64)[:, None] * inv[None, :]
    return angle.cos().half(), angle.sin().half()


def _prepare_step(case, g):
    ops = _ops()
    cabi = ops.cabi
    max_pos = max(512, -(-(case["pos"] + 1) // 512) * 512)
    cos, sin = _rope_tables(max_pos, 1e6)
    s = {"ops": ops, "ws": ops.Workspace(pdl=case["pdl"]), "layers": [], "keep": [cos, sin], "pos": case["pos"], "max_pos": max_pos}
    hidden = s["hidden"] = torch.zeros(H, dtype=torch.float16, device="cuda")
    q = torch.zeros(H, dtype=torch.float16, device="cuda")
    mlp = torch.zeros(INTER, dtype=torch.float16, device="cuda")
    s["q"] = q
    s["keep"] += [mlp]
    for _ in range(case["layers"]):
        w = {stem: ops.W4Linear(packed, scale, zp, out, inp) for stem, out, inp, packed, scale, zp in _layer_matrices(g, H, INTER)}
        gamma = _normal(g, H, mean=1.0, std=0.02)
        kc, vc = _normal(g, HEADS, max_pos, 128), _normal(g, HEADS, max_pos, 128)
        s["keep"].append(gamma)
        s["layers"].append((
            w, kc, vc,
            ops.gemv_args(hidden, epilogue=cabi.EPI_ROPE_KV, y=q, gamma=gamma, k_cache=kc, v_cache=vc, cos=cos, sin=sin, heads=HEADS,
                          max_pos=max_pos, pos=case["pos"]),
            ops.gemv_args(hidden, epilogue=cabi.EPI_GELU, y=mlp, gamma=gamma),
            ops.gemv_args(mlp, epilogue=cabi.EPI_RESIDUAL, y=hidden)))
    s["emb"], (packed, scale, zp) = _embeddings(g, H, VOCAB)
    s["unemb"] = ops.W4Linear(packed, scale, zp, VOCAB, H)
    s["token"] = int(torch.randint(0, VOCAB, (1,), device="cuda", generator=g))
    s["logits"] = torch.zeros(VOCAB, dtype=torch.float16, device="cuda")
    s["next"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    s["sample"] = ops.gemv_args(hidden, epilogue=cabi.EPI_ARGMAX, y=s["logits"], gamma=s["keep"][-1], d_token=s["next"])
    return s


def _linear_weights(case, g):
    out, inp = case["out"], case["in"]
    return [(_codes(g, out, inp), _scales(g, out // 128, 0.1), _zeros(g, out // 128, case["integral"])) for _ in range(case["count"])]


def prepare(case, seed):
    family = case["family"]
    g = _generator(seed)
    if family == "generate":
        vocab = MODELS[case["model"]]["vocab"]
        prompt = torch.randint(0, vocab, (case["prompt"],), device="cuda", generator=g).tolist()
        return {"family": family, "engine": _engine(case["model"], case["cluster"]), "prompt": prompt, "new": case["new"]}
    if family == "step":
        return dict(_prepare_step(case, g), family=family)
    ops = _ops()
    if family == "attention":
        heads, rows, pos0 = case["heads"], case["rows"], case["pos0"]
        max_pos = -(-(pos0 + rows) // 128) * 128
        return {"family": family, "ops": ops, "heads": heads, "rows": rows, "pos0": pos0, "max_pos": max_pos,
                "qkv": _normal(g, rows, 3 * heads * 128), "k": _normal(g, heads, max_pos, 128), "v": _normal(g, heads, max_pos, 128)}
    out, inp, count = case["out"], case["in"], case["count"]
    weights = [ops.W4Linear(*w, out, inp, zp_integral=case["integral"]) for w in _linear_weights(case, g)]
    s = {"family": family, "ops": ops, "ws": ops.Workspace(), "weights": weights}
    if family == "rows":
        s["x"] = _normal(g, case["rows"], inp)
        s["y"] = [torch.zeros(case["rows"], out, dtype=torch.float16, device="cuda") for _ in range(count)]
        return s
    cabi = ops.cabi
    epilogue = {"store": cabi.EPI_STORE, "gelu": cabi.EPI_GELU, "argmax": cabi.EPI_ARGMAX}[case["epilogue"]]
    s["x"] = _normal(g, inp)
    s["gamma"] = None if epilogue == cabi.EPI_STORE else _normal(g, inp, mean=1.0, std=0.02)
    s["y"] = [torch.zeros(out, dtype=torch.float16, device="cuda") for _ in range(count)]
    s["token"] = torch.zeros(count, dtype=torch.int32, device="cuda") if epilogue == cabi.EPI_ARGMAX else None
    s["args"] = [ops.gemv_args(s["x"], epilogue=epilogue, y=y, gamma=s["gamma"],
                               d_token=None if s["token"] is None else s["token"][i:i + 1]) for i, y in enumerate(s["y"])]
    s["noalloc"], s["integral"] = case["noalloc"], int(case["integral"])
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------------------

def _run_step(s):
    ops, ws, hidden, q = s["ops"], s["ws"], s["hidden"], s["q"]
    packed, scale, zp = s["emb"]
    hidden.copy_(ops.embed_gather_w4(packed, scale, zp, H, VOCAB, s["token"]))
    for w, kc, vc, qkv, up, down in s["layers"]:
        ops.gemv_w4a16(w["wqkv"], ws, qkv)
        ctx = ops.attn_decode(q, kc, vc, HEADS, s["max_pos"], s["pos"], ws)
        ops.gemv_w4a16(w["wo"], ws, ops.gemv_args(ctx, epilogue=ops.cabi.EPI_RESIDUAL, y=hidden))
        ops.gemv_w4a16(w["w1"], ws, up)
        ops.gemv_w4a16(w["w2"], ws, down)
    ops.gemv_w4a16(s["unemb"], ws, s["sample"])
    return {"token": s["next"], "logits": s["logits"], "hidden": hidden, "k": [x[1] for x in s["layers"]], "v": [x[2] for x in s["layers"]]}


def _run_noalloc(s):
    cabi = s["ops"].cabi
    stream = torch.cuda.current_stream().cuda_stream
    for w, y in zip(s["weights"], s["y"]):
        cabi.check(cabi.lib().qw3_gemv_w4a16_noalloc(w.packed.data_ptr(), w.scale.data_ptr(), w.zp.data_ptr(), w.scale.numel(), w.out_dim,
                                                     w.in_dim, s["integral"], s["x"].data_ptr(), y.data_ptr(), stream),
                   "qw3_gemv_w4a16_noalloc")


def run(s):
    family = s["family"]
    if family == "generate":
        ids = s["engine"].generateResponse(s["prompt"], s["new"])
        return {"ids": np.asarray(ids, dtype=np.int32), "logits": s["engine"].last_logits()}
    if family == "step":
        return _run_step(s)
    ops = s["ops"]
    if family == "attention":
        return ops.attn_prefill(s["qkv"], s["k"], s["v"], s["heads"], s["max_pos"], s["pos0"], s["rows"])
    if family == "rows":
        for w, y in zip(s["weights"], s["y"]):
            ops.gemm_w4a16(w, s["ws"], s["x"], y)
        return s["y"]
    if s["noalloc"]:
        _run_noalloc(s)
    else:
        for w, a in zip(s["weights"], s["args"]):
            ops.gemv_w4a16(w, s["ws"], a)
    # the winning index of a flat random logit vector can hang on its last bit: the logits themselves are what is compared
    return s["y"]


# ---- what a pass cannot do without, and how far two right answers lie apart -------------------------------------------------------

def _matrix_bytes(out, inp):
    return out * inp / 2 + 4 * (out // 128)


def work(case):
    family = case["family"]
    if family == "generate":
        c = MODELS[case["model"]]
        h, inter, layers, vocab, n, new = c["hidden"], c["inter"], c["layers"], c["vocab"], case["prompt"], case["new"]
        weights = layers * (_matrix_bytes(3 * h, h) + _matrix_bytes(h, h) + _matrix_bytes(inter, h) + _matrix_bytes(h, inter))
        params = layers * (4 * h * h + 2 * h * inter)
        contexts = sum(range(n + 1, n + new + 1))   # cache rows that the decode passes read
        return {"bytes": (1 + new) * weights + new * _matrix_bytes(vocab, h) + layers * 4 * h * (contexts + n + new) + 4 * vocab,
                "flops": 2 * params * (n + new) + 2 * vocab * h * new + layers * 4 * h * (n * (n + 1) / 2 + contexts)}
    if family == "step":
        per_layer = _matrix_bytes(3 * H, H) + _matrix_bytes(H, H) + _matrix_bytes(INTER, H) + _matrix_bytes(H, INTER) + 4 * H * (case["pos"] + 1)
        return {"bytes": case["layers"] * per_layer + _matrix_bytes(VOCAB, H) + 2 * VOCAB,
                "flops": 2 * (case["layers"] * (4 * H * H + 2 * H * INTER) + VOCAB * H) + case["layers"] * 4 * H * (case["pos"] + 1)}
    if family == "attention":
        width, rows, pos0 = 128 * case["heads"], case["rows"], case["pos0"]
        return {"bytes": 2 * width * (2 * rows + 2 * (pos0 + rows)), "flops": 4 * width * (rows * pos0 + rows * (rows + 1) / 2)}
    rows, out, inp = case.get("rows", 1), case["out"], case["in"]
    return {"bytes": case["count"] * (_matrix_bytes(out, inp) + 2 * rows * out) + 2 * rows * inp, "flops": 2.0 * case["count"] * rows * out * inp}


def tolerance(case):
    """fp16 results of fp32 sums: another order of the sums turns some results by one unit in the last place (2^-11 to
    2^-10 of the value).  Behind a chain of layers these add up; ids are whole numbers and stay the same."""
    if case["family"] in ("generate", "step"):
        return {"rel": 1e-2, "max": 0.1, "differ": 0.0}
    return {"rel": 1e-3, "max": 4e-3}


# ---- the same results in 64 bits, in plain torch ---------------------------------------------------------------------------------

def _exact_product(packed, scale, zp, out, inp, x):
    """x (rows of float64) times the dequantised matrix.  The weights themselves are fp16 by definition: fp16(fp16(q - zp) * scale)."""
    y = torch.empty(x.shape[0], out, dtype=torch.float64, device="cuda")
    j = torch.arange(inp, device="cuda")
    for b0 in range(0, out // 128, 32):   # 4096 outputs at a time
        b1 = min(b0 + 32, out // 128)
        block = packed.view(inp, out // 2)[:, 64 * b0:64 * b1]
        q = torch.stack((block & 15, block >> 4), 2).view(inp, -1, 128).half()
        group = ((torch.arange(b0, b1, device="cuda")[None, :] + j[:, None] * (out // 128)) % (inp // 128)) % scale.numel()
        w = (q - zp[group][:, :, None]) * scale[group][:, :, None]
        y[:, 128 * b0:128 * b1] = x @ w.view(inp, -1).double()
    return y


def exact(case, seed):
    """Linears, row blocks and attention.  A token pass rounds to fp16 between its operators by definition, and which logit
    wins decides what comes next: it has no 64-bit result that an implementation could come nearer to."""
    family = case["family"]
    if family in ("generate", "step"):
        return None
    g = _generator(seed)
    if family == "attention":
        heads, rows, pos0 = case["heads"], case["rows"], case["pos0"]
        max_pos = -(-(pos0 + rows) // 128) * 128
        qkv, k, v = _normal(g, rows, 3 * heads * 128), _normal(g, heads, max_pos, 128), _normal(g, heads, max_pos, 128)
        hidden = torch.arange(pos0 + rows, device="cuda")[None, :] > pos0 + torch.arange(rows, device="cuda")[:, None]
        y = torch.empty(rows, heads * 128, dtype=torch.float64, device="cuda")
        for h in range(heads):
            s = qkv[:, 128 * h:128 * h + 128].double() @ k[h, :pos0 + rows].double().T / math.sqrt(128.0)
            y[:, 128 * h:128 * h + 128] = torch.softmax(s.masked_fill(hidden, -math.inf), 1) @ v[h, :pos0 + rows].double()
        return y
    out, inp = case["out"], case["in"]
    weights = _linear_weights(case, g)
    if family == "rows":
        x = _normal(g, case["rows"], inp).double()
        return [_exact_product(*w, out, inp, x) for w in weights]
    x = _normal(g, inp)
    if case["epilogue"] != "store":   # the normalised vector is fp16 by definition, as its factor is: fp16(fp16(x * r) * gamma)
        gamma = _normal(g, inp, mean=1.0, std=0.02)
        r = (1.0 / torch.sqrt(x.double().square().mean() + 1e-6)).half()
        x = x * r * gamma
    ys = [_exact_product(*w, out, inp, x.double()[None, :])[0] for w in weights]
    if case["epilogue"] == "gelu":   # of the product as fp16
        ys = [0.5 * y * (1.0 + torch.erf(y * math.sqrt(0.5))) for y in (y.half().double() for y in ys)]
    return ys
