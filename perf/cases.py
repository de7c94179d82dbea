"""The work this package is timed on, through its public entry points.

Five kinds of pass, each over the whole range a user meets:

  linear    `QuantizedLinear(x)`, with or without the preceding RMSNorm: one quantised linear of a decoder layer
            (rotation, quantisation of the activations, packed product), from one decode row to a prefill batch.
  quant     `rms_norm_quant(x)`: hidden states to the packed operand a quantised linear consumes.
  weight    `QuantizedLinear.from_weight(w)`: what loading a bf16 checkpoint does for every linear.
  prefill   `ResQForwardB200.forward(ids)`: a prompt through the decoder stack, logits of the last position and the
            key / value cache it leaves.
  decode    `forward(ids)` and then `forward(token, pos0=...)` per token, as a server with its own sampler (or a
            scorer of given continuations) calls it: logits of every step and the cache.

Layer shapes are the package's two configurations (hidden 4096 / FFN 14336 and hidden 8192 / FFN 28672, head_dim 128)
with a bounded number of layers; weights and prompts are drawn from the seed, activations are N(0, 1) with 1 % of the
channels scaled by 20, as in bench.py.  The decoder's weights are scaled like a trained model's: the residual stream
starts at unit size and every projection adds a fraction of it.  (With the package's own random initialisation every
layer replaces the stream, and 4-bit rounding turns one flipped last bit into unrelated logits a few layers later.)
"""
import math

import torch

from plaquant_b200.quantize import QuantizedLinear
from plaquant_b200.forward_pass import LlamaConfig, ResQForwardB200, rms_norm_quant
from plaquant_b200.tp import outlier_count

EPS = 1e-6
# K -> N of the fused qkv, o, gate_up and down projections of the two configurations, and of the row-parallel
# linears of the larger one on one of eight ranks
SHAPES = [(4096, 6144), (4096, 4096), (4096, 28672), (14336, 4096),
          (8192, 10240), (8192, 8192), (8192, 57344), (28672, 8192), (1024, 8192), (3584, 8192)]


def listed():
    return [
        # one token of one sequence: launches and host work are what counts
        {"name": "linear_1_4096_4096", "kind": "linear", "m": 1, "k": 4096, "n": 4096, "norm": False},
        # a small decode batch on the widest projection, norm fused: streaming the weights
        {"name": "linear_8_4096_28672_norm", "kind": "linear", "m": 8, "k": 4096, "n": 28672, "norm": True},
        # the largest decode batch of the streaming kernel, the longest K
        {"name": "linear_16_14336_4096", "kind": "linear", "m": 16, "k": 14336, "n": 4096, "norm": False},
        # a few sequences' draft tokens or one short prompt: too many rows for decode, ragged against every tile
        {"name": "linear_77_4096_6144_norm", "kind": "linear", "m": 77, "k": 4096, "n": 6144, "norm": True},
        # one prompt of ordinary length
        {"name": "linear_512_4096_4096", "kind": "linear", "m": 512, "k": 4096, "n": 4096, "norm": False},
        # a prefill batch
        {"name": "linear_8192_14336_4096", "kind": "linear", "m": 8192, "k": 14336, "n": 4096, "norm": False},
        # the norm + rotation + quantiser in front of a prefill batch's projections
        {"name": "quant_4096_4096", "kind": "quant", "rows": 4096, "k": 4096, "layout": "tiled"},
        # loading: the widest weight of a layer
        {"name": "weight_28672_4096", "kind": "weight", "n": 28672, "k": 4096},
        # one user's prompt, ragged length
        {"name": "prefill_1x333", "kind": "prefill", "hidden": 4096, "layers": 16, "batch": 1, "tokens": 333, "kv_quant": False},
        # a full prefill batch of the larger configuration
        {"name": "prefill_16x2048_wide", "kind": "prefill", "hidden": 8192, "layers": 2, "batch": 16, "tokens": 2048, "kv_quant": False},
        # serving: a batch of prompts and the first tokens of their answers
        {"name": "decode_16x512_32", "kind": "decode", "hidden": 4096, "layers": 16, "batch": 16, "tokens": 512, "steps": 32, "kv_quant": False},
        # a long prompt with the NVFP4 key / value cache
        {"name": "decode_2x1500_16_kv4", "kind": "decode", "hidden": 4096, "layers": 16, "batch": 2, "tokens": 1500, "steps": 16, "kv_quant": True},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "quant", "weight", "prefill", "decode", "decode"])
    if kind == "linear":
        k, n = rng.choice(SHAPES)
        m = _log_int(rng, 1, 16) if rng.random() < 0.5 else _log_int(rng, 17, 8192)
        return {"kind": kind, "m": m, "k": k, "n": n, "norm": rng.random() < 0.5}
    if kind == "quant":
        rows, k = _log_int(rng, 1, 16384), 128 * _log_int(rng, 8, 112)
        # scale bytes of padding rows are unspecified in the tiled layout: whole 128-row groups there
        layout = rng.choice(["tiled", "rowmajor"])
        if layout == "tiled":
            rows = -(-rows // 128) * 128
            k = -(-k // 4096) * 4096
        return {"kind": kind, "rows": rows, "k": k, "layout": layout}
    if kind == "weight":
        return {"kind": kind, "n": 8 * _log_int(rng, 128, 4096), "k": 128 * _log_int(rng, 8, 112)}
    batch = _log_int(rng, 1, 16)
    case = {"kind": kind, "hidden": 4096, "layers": rng.randint(4, 16), "batch": batch}
    if kind == "prefill":
        case.update(tokens=_log_int(rng, 17, 8192 // batch), kv_quant=rng.random() < 0.25)
    else:
        case.update(tokens=_log_int(rng, 17, 2048 if batch < 5 else 640), steps=rng.randint(4, 24), kv_quant=rng.random() < 0.33)
    return case


def _config(hidden):
    return LlamaConfig.llama3_8b() if hidden == 4096 else LlamaConfig.llama3_70b()


def _activations(rows, k, g):
    x = torch.randn(rows, k, generator=g, device="cuda")
    scale = torch.ones(k, device="cuda")
    scale[torch.randperm(k, generator=g, device="cuda")[: max(1, k // 100)]] = 20.0
    return (x * scale).to(torch.bfloat16)


def _gamma(k, g):
    return (torch.rand(k, generator=g, device="cuda") + 0.5).to(torch.bfloat16)


def _weight(n, k, g):
    return (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16)


def _decoder_weights(cfg, layers, g):
    """A dict under the names `ResQForwardB200(weights=...)` takes."""
    h, f = cfg.hidden_size, cfg.intermediate_size
    q, kv = cfg.num_heads * cfg.head_dim, cfg.num_kv_heads * cfg.head_dim

    def normal(n, k, std):
        return torch.randn(n, k, generator=g, device="cuda", dtype=torch.bfloat16).mul_(std)
    w = {"embed": normal(cfg.vocab_size, h, 1.0), "lm_head": normal(cfg.vocab_size, h, 0.02), "final_norm": _gamma(h, g)}
    for i in range(layers):
        w.update({f"l{i}.ln1": _gamma(h, g), f"l{i}.ln2": _gamma(h, g),
                  f"l{i}.q_proj.weight": normal(q, h, 0.02), f"l{i}.k_proj.weight": normal(kv, h, 0.02),
                  f"l{i}.v_proj.weight": normal(kv, h, 0.02), f"l{i}.o_proj.weight": normal(h, q, 0.002),
                  f"l{i}.mlp.gate_proj.weight": normal(f, h, 0.02), f"l{i}.mlp.up_proj.weight": normal(f, h, 0.02),
                  f"l{i}.mlp.down_proj.weight": normal(h, f, 0.0003)})
    return w


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        lin = QuantizedLinear.from_weight(_weight(case["n"], case["k"], g))
        return {"kind": kind, "lin": lin, "x": _activations(case["m"], case["k"], g),
                "gamma": _gamma(case["k"], g) if case["norm"] else None}
    if kind == "quant":
        return {"kind": kind, "x": _activations(case["rows"], case["k"], g), "gamma": _gamma(case["k"], g),
                "k_hi": outlier_count(case["k"]), "layout": case["layout"]}
    if kind == "weight":
        return {"kind": kind, "w": _weight(case["n"], case["k"], g)}
    cfg = _config(case["hidden"])
    model = ResQForwardB200(cfg, "cuda", num_layers=case["layers"], kv_quant=case["kv_quant"],
                            weights=_decoder_weights(cfg, case["layers"], g))
    b, t, steps = case["batch"], case["tokens"], case.get("steps", 0)
    ids = torch.randint(0, cfg.vocab_size, (b, t + steps), generator=g, device="cuda")
    return {"kind": kind, "model": model, "ids": ids[:, :t].contiguous(),
            "next": [ids[:, t + i:t + i + 1].contiguous() for i in range(steps)]}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"](state["x"], norm_weight=state["gamma"], eps=EPS)
    if kind == "quant":
        p = rms_norm_quant(state["x"], state["gamma"], EPS, state["k_hi"], sf_layout=state["layout"])
        return [p.lo_codes, p.lo_sf, p.hi_codes, p.hi_sf]
    if kind == "weight":
        q = QuantizedLinear.from_weight(state["w"])
        return [q.w_main_int, q.w_main_scale, q.w_high_int, q.w_high_scale]
    model, ids = state["model"], state["ids"]
    logits = [model.forward(ids)]
    t = ids.shape[1]
    for i, tok in enumerate(state["next"]):
        logits.append(model.forward(tok, pos0=t + i))
    return {"logits": torch.stack(logits), "kv": [x for layer in model.kv for x in layer]}


def _packed_bytes(rows, k):
    """Codes and scale bytes of a packed [rows, k] operand."""
    k_hi = outlier_count(k)
    k_lo = k - k_hi
    return rows * (k_lo // 2 + k_lo // 16 + k_hi + k_hi // 32)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 2 * m * k + 2 * m * n + _packed_bytes(n, k) + (2 * k if case["norm"] else 0), "flops": 2 * m * n * k}
    if kind == "quant":
        rows, k = case["rows"], case["k"]
        return {"bytes": 2 * rows * k + 2 * k + _packed_bytes(rows, k), "flops": 0}
    if kind == "weight":
        return {"bytes": 2 * case["n"] * case["k"] + _packed_bytes(case["n"], case["k"]), "flops": 0}
    c, b, t, layers, steps = _config(case["hidden"]), case["batch"], case["tokens"], case["layers"], case.get("steps", 0)
    h, f, hd = c.hidden_size, c.intermediate_size, c.head_dim
    qkv = (c.num_heads + 2 * c.num_kv_heads) * hd
    linears = [(h, qkv), (c.num_heads * hd, h), (h, 2 * f), (f, h)]
    weights = layers * sum(_packed_bytes(n, k) for k, n in linears)
    head = 2 * c.vocab_size * h
    row_bytes = layers * 2 * c.num_kv_heads * (72 if case["kv_quant"] else 2 * hd)     # cache, one position of one sequence
    per_row = layers * sum(2 * n * k for k, n in linears)
    attn = lambda q, ctx: layers * 4 * c.num_heads * hd * q * ctx                     # noqa: E731
    total_bytes = weights + head + b * t * (2 * h + row_bytes) + 4 * b * c.vocab_size
    flops = b * (t * per_row + attn(t, (t + 1) / 2) + 2 * h * c.vocab_size)
    for i in range(steps):
        total_bytes += weights + head + b * (2 * h + (t + i + 1) * row_bytes) + 4 * b * c.vocab_size
        flops += b * (per_row + attn(1, t + i + 1) + 2 * h * c.vocab_size)
    return {"bytes": total_bytes, "flops": flops}


def tolerance(case):
    if case["kind"] in ("quant", "weight"):
        return "exact"
    if case["kind"] == "linear":
        # bf16 results of one float32 sum: another split of K flips the last bit of a few of them (measured between
        # the two product kernels: 2.3e-5, the largest difference 5.8e-3 = one bf16 step)
        return {"rel": 1e-4, "max": 2e-2}
    # Every projection rounds its input to 4 bits, so two correct evaluations of the attention sums end with rounding
    # noise of their own in every later layer.  Measured with the attention in plain float32 and the other product
    # kernel for the decode rows: 0.05 of the logits, 0.12 of the keys and values of layer 16 (it saturates there),
    # and 0.61 of the bytes of a 4-bit cache.
    return {"rel": 0.25, "differ": 0.7} if case["kv_quant"] else {"rel": 0.25}
