"""The work a user of this package has it do, as cases with sizes, inputs and one pass each.

Kinds of case (the key "kind"):

  linear   one quantised linear called on `rows` activation rows: 1 row is token-by-token decoding, up to 16
           a speculative verify or a small decode batch, up to a few hundred a short prompt or a large
           decode batch, thousands a prompt.
  mlp      the gated MLP of a dense model (gate|up group, GLU, down) on `rows` rows.
  moe      the stacked-expert SwitchGLU on `tokens` tokens with their top-k routing.
  step     one decode step of a dense decoder over a long KV cache, replayed from a CUDA graph as a
           serving loop does.
  encode   the exact trellis search of a converter on one matrix.

Trellis words are uniform random bits (every bitstream is a valid tile), sign vectors are random +-1,
output scales keep activations near unit size, activations are N(0, 1), routing is the top-k of N(0, 1)
logits.  Weights, modules, routing and the captured graph are what a program has in hand before the call.
"""

import math

import torch

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def listed():
    return [
        # decoding: one 4096 x 4096 layer (latency and launches), and a gate/up projection
        dict(name="linear 1 row, square", kind="linear", rows=1, n_in=4096, n_out=4096, k=4, cb=0, dtype="f16", bias=False),
        dict(name="linear 1 row, gate", kind="linear", rows=1, n_in=5120, n_out=17408, k=4, cb=0, dtype="f16", bias=False),
        # a small decode batch on a small layer of odd width, fp32 activations, bias, third codebook
        dict(name="linear 5 rows, odd, bias", kind="linear", rows=5, n_in=2944, n_out=1408, k=3, cb=2, dtype="f32", bias=True),
        # speculative verify of 16 positions through a down projection
        dict(name="linear 16 rows, down", kind="linear", rows=16, n_in=17408, n_out=5120, k=5, cb=1, dtype="bf16", bias=False),
        # a short prompt, a prompt chunk at a higher bit width, and a whole 8192-token prompt
        dict(name="linear 77 rows", kind="linear", rows=77, n_in=5120, n_out=5120, k=4, cb=0, dtype="bf16", bias=False),
        dict(name="linear 1000 rows, K=6", kind="linear", rows=1000, n_in=5120, n_out=17408, k=6, cb=0, dtype="f16", bias=False),
        dict(name="linear 8192 rows", kind="linear", rows=8192, n_in=5120, n_out=5120, k=4, cb=0, dtype="bf16", bias=False),
        # a prompt of 300 tokens through a dense MLP
        dict(name="mlp 300 rows", kind="mlp", rows=300, n_in=5120, hidden=17408, k=4, cb=0, dtype="bf16", act="silu"),
        # mixture of experts: a decode batch and a prompt
        dict(name="moe 16 tokens", kind="moe", tokens=16, experts=256, top_k=8, n_in=2048, hidden=512, k=4, cb=0, act="silu"),
        dict(name="moe 4096 tokens", kind="moe", tokens=4096, experts=256, top_k=8, n_in=2048, hidden=512, k=4, cb=0, act="silu"),
        # a decode step, a quarter of the 64-layer depth (every layer costs the same) and the whole head
        dict(name="decode step", kind="step", rows=1, layers=16, context=8192),
        # converting: 592 tiles of 16 x 16
        dict(name="encode 592 tiles", kind="encode", n_in=256, n_out=592, k=4, cb=0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _width(rng, lo, hi):
    """A feature count: any multiple of 128."""
    return 128 * max(1, round(_log(rng, lo, hi) / 128))


def draw(rng):
    kind = rng.choices(["linear", "mlp", "moe", "step", "encode"], [6, 2, 2, 1, 1])[0]
    k = rng.choices([1, 2, 3, 4, 5, 6, 7, 8], [1, 2, 2, 5, 3, 2, 1, 1])[0]
    cb = rng.choices([0, 1, 2], [2, 1, 1])[0]
    dtype = rng.choices(["f16", "bf16", "f32"], [3, 3, 1])[0]
    if kind == "linear":
        n_in, n_out = _width(rng, 512, 17408), _width(rng, 512, 17408)
        rows = min(round(_log(rng, 1, 8192)), 8192 * 5120 * 5120 // (n_in * n_out))
        return dict(kind=kind, rows=rows, n_in=n_in, n_out=n_out, k=k, cb=cb, dtype=dtype, bias=rng.random() < 0.25)
    act = rng.choice(["silu", "gelu"])
    if kind == "mlp":
        n_in, hidden = _width(rng, 1024, 5120), _width(rng, 2048, 17408)
        rows = min(round(_log(rng, 1, 2048)), 8192 * 5120 * 5120 // (3 * n_in * hidden))
        return dict(kind=kind, rows=rows, n_in=n_in, hidden=hidden, k=k, cb=cb, dtype=dtype, act=act)
    if kind == "moe":
        return dict(kind=kind, tokens=round(_log(rng, 1, 4096)), experts=rng.choice([64, 128, 256]), top_k=rng.randint(2, 8),
                    n_in=_width(rng, 1024, 2048), hidden=_width(rng, 256, 512), k=min(k, 6), cb=cb, act=act)
    if kind == "step":
        return dict(kind=kind, rows=rng.randint(1, 16), layers=rng.randint(2, 8), context=round(_log(rng, 500, 8192)))
    return dict(kind=kind, n_in=16 * rng.randint(2, 16), n_out=16 * rng.randint(4, 37), k=min(k, 6), cb=cb)


# ---- what a program has before the call -------------------------------------------------------------

def _words(gen, *shape):
    return torch.randint(-32768, 32768, shape, dtype=torch.int16, device="cuda", generator=gen)


def _signs(gen, *shape, scale=1.0):
    return (torch.randint(0, 2, shape, device="cuda", generator=gen) * 2 - 1).to(torch.float16) * scale


def _unit(n_in):
    """Output scale that brings a product over n_in unit activations back to unit size."""
    return 1.0 / (1.25 * math.sqrt(n_in))


def _linear(gen, n_in, n_out, k, cb, bias=False):
    from ponyexl3_b200 import EXL3Linear
    b = (torch.randn(n_out, device="cuda", generator=gen) * 0.1).to(torch.float16) if bias else None
    return EXL3Linear.from_device_tensors(trellis=_words(gen, n_in // 16, n_out // 16, 16 * k), k=k, cb=cb,
                                          suh=_signs(gen, n_in), svh=_signs(gen, n_out, scale=_unit(n_in)), bias=b)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        m = _linear(gen, case["n_in"], case["n_out"], case["k"], case["cb"], case["bias"])
        x = torch.randn((case["rows"], case["n_in"]), device="cuda", generator=gen).to(DTYPES[case["dtype"]])
        return dict(kind=kind, module=m, x=x)
    if kind == "mlp":
        from ponyexl3_b200 import EXL3MLPMonolith, FusedEXL3Group
        d, h, k, cb = case["n_in"], case["hidden"], case["k"], case["cb"]
        gate_up = FusedEXL3Group.from_device_tensors(
            trellis=_words(gen, d // 16, 2 * h // 16, 16 * k), k=k, cb=cb, suh_stack=_signs(gen, 2, d),
            svh_cat=_signs(gen, 2 * h, scale=_unit(d)), out_features=[h, h])
        m = EXL3MLPMonolith.from_fused_gate_up(gate_up, _linear(gen, h, d, k, cb), activation=case["act"])
        x = torch.randn((case["rows"], d), device="cuda", generator=gen).to(DTYPES[case["dtype"]])
        return dict(kind=kind, module=m, x=x)
    if kind == "moe":
        from ponyexl3_b200 import EXL3SwitchGLU
        e, d, h, k, t = case["experts"], case["n_in"], case["hidden"], case["k"], case["tokens"]
        m = EXL3SwitchGLU(
            gu_trellis=_words(gen, d // 16, e * 2 * h // 16, 16 * k), gu_suh=_signs(gen, e, 2, d),
            gu_svh=_signs(gen, e, 2 * h, scale=_unit(d)), dn_trellis=_words(gen, h // 16, e * d // 16, 16 * k),
            dn_suh=_signs(gen, e, h), dn_svh=_signs(gen, e, d, scale=_unit(h)), k=k, cb=case["cb"], activation=case["act"])
        x = torch.randn((1, t, d), device="cuda", generator=gen).to(torch.float16)
        logits = torch.randn((1, t, e), device="cuda", generator=gen)
        return dict(kind=kind, module=m, x=x, indices=torch.topk(logits, case["top_k"], dim=-1).indices)
    if kind == "step":
        from ponyexl3_b200.dense_step import SyntheticDenseDecoder
        cfg = _config(case)
        model = SyntheticDenseDecoder(cfg, torch.device("cuda", torch.cuda.current_device()), seed=seed)
        tokens = torch.randint(0, cfg.vocab, (case["rows"],), device="cuda", generator=gen)
        slot = tokens.clone()
        model.forward_logits(slot)               # a serving loop warms up once, then captures its step
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = model.forward_logits(slot)
        span = slice(cfg.context, cfg.context + case["rows"])
        new = [c[:, span] for layer in model.layers for c in (layer.k_cache, layer.v_cache)]
        return dict(kind=kind, model=model, tokens=tokens, slot=slot, graph=graph, outputs=[logits] + new)
    inner = torch.randn((case["n_in"], case["n_out"]), device="cuda", generator=gen)
    return dict(kind=kind, inner=inner, k=case["k"], cb=case["cb"])


def _config(case):
    from ponyexl3_b200.dense_step import DenseConfig
    return DenseConfig(layers=case["layers"], context=case["context"])


def run(state):
    kind = state["kind"]
    if kind == "moe":
        return state["module"](state["x"], state["indices"])
    if kind == "step":
        state["slot"].copy_(state["tokens"])
        state["graph"].replay()
        return state["outputs"]                  # logits, and the K and V rows this step appended
    if kind == "encode":
        from ponyexl3_b200 import ops
        return ops.quantize_inner(state["inner"], state["k"], state["cb"])
    return state["module"](state["x"])


def work(case):
    kind = case["kind"]
    if kind == "encode":
        tiles = case["n_in"] * case["n_out"] // 256
        # per weight and state a difference, a product and a sum, in the free pass and one pinned pass
        return {"bytes": tiles * (256 * 4 + 32 * case["k"]), "flops": 2 * 3 * 65536 * 256 * tiles}
    if kind == "step":
        cfg = _config(case)
        # a step reads all weights at the mean bit width and the whole cache
        ks = [4 + cfg.k5_fraction] * (4 * cfg.layers + 1)
        weights = cfg.packed_bytes([8] * len(ks))
        cache = cfg.layers * 2 * cfg.kv_heads * (cfg.context + case["rows"]) * cfg.head_dim
        return {"bytes": weights * ks[0] / 8 + 2 * cache + 2 * case["rows"] * (cfg.vocab + cfg.hidden),
                "flops": 2 * case["rows"] * (weights + cfg.group * cache)}
    d = case["n_in"]
    if kind == "moe":
        pairs, e, h = case["tokens"] * case["top_k"], case["experts"], case["hidden"]
        hit = e * (1 - (1 - case["top_k"] / e) ** case["tokens"])      # experts that get a token
        vectors = 2 * (2 * d + 2 * h + h + d)
        return {"bytes": hit * (3 * d * h * case["k"] / 8 + vectors) + 2 * d * case["tokens"] + 8 * pairs + 2 * d * pairs,
                "flops": 6 * d * h * pairs}
    rows, size = case["rows"], {"f16": 2, "bf16": 2, "f32": 4}[case["dtype"]]
    if kind == "mlp":
        h = case["hidden"]
        return {"bytes": 3 * d * h * case["k"] / 8 + 2 * (2 * d + 2 * h + h + d) + rows * d * (size + 2),
                "flops": 6 * d * h * rows}
    n = case["n_out"]
    return {"bytes": d * n * case["k"] / 8 + 2 * (d + n * (2 if case["bias"] else 1)) + rows * (d * size + 2 * n),
            "flops": 2 * d * n * rows}


def tolerance(case):
    """fp16 weights, rotated activations and outputs with fp32 sums: a different order of the sums flips
    roundings to fp16, about 1e-4 per linear in the 2-norm.  The chained linears of an MLP add up, and a
    step chains all its layers through fp16 residuals and attention.  The trellis search is exact."""
    if case["kind"] == "encode":
        return "exact"
    return {"rel": {"linear": 1e-3, "mlp": 2e-3, "moe": 2e-3, "step": 1e-2}[case["kind"]]}
