"""The work whose speed counts: what a program that uses locomp_b200 has it do, over the range of sizes
it does it at.

Five kinds of case, each one pass through the public entry points:

  linear    y = QuantLinear(x): int4 or int8 weights resident on the GPU, M rows of activations.  M = 1 is
            a single sequence's decode step, M <= 16 a small decode batch, M up to a few hundred a
            serving batch or a short prompt, M in the thousands a long prompt (prefill).
  stack     one token through DecodeStack: every linear of a Llama-style model with the embedding, norms,
            activation, residual adds and argmax between them, replayed from its CUDA graph.
  mlp       the MLP block of a prompt: RMS norm, gate and up projections, SiLU * up, down projection,
            residual add.
  dequant   packed weights back to floats.
  quantize  float weights to packed weights and scales (loading a model).

Weights are uniform over the integer range with |N(0, 1)| * 0.02 scales (int8: * 0.01), activations
N(0, 1), float weights N(0, 1) * 0.1: the distributions of the benchmark configurations.
"""
import math

import torch

import locomp_b200 as L

KINDS = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}
LARGEST_FLOPS = 2.0 * 8192 * 14336 * 4096          # the longest prompt of the listed cases


def _linear(m, k, n, bits=4, group=32, x="f16", scales="f16", name=None):
    case = {"kind": "linear", "m": m, "k": k, "n": n, "bits": bits, "group": group, "x": x, "scales": scales}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest call: int8 weights with one float32 scale per output, the reference's own types
        # (SmolLM2-135M MLP up projection); launch and host path are all there is
        _linear(1, 576, 1536, bits=8, group=576, x="f32", scales="f32", name="int8_matvec_small"),
        # one sequence, an attention projection of SmolLM2-1.7B: the ordinary small decode call
        _linear(1, 2048, 2048, name="decode_projection"),
        # three sequences against the vocabulary of SmolLM2-135M: odd batch, K no multiple of the tile
        _linear(3, 576, 49152, name="decode_head_ragged"),
        # one sequence, MLP up projection of a 70B-class model: as many weights as a decode call streams
        _linear(1, 8192, 28672, name="decode_70b_up"),
        # a full decode batch against the vocabulary of SmolLM2-1.7B
        _linear(16, 2048, 49152, name="decode_head_batch16"),
        # a serving batch on the 70B-class shape: between decode and prefill
        _linear(64, 8192, 28672, name="serving_batch64"),
        # a short prompt through the MLP up projection of an 8B-class model
        _linear(512, 4096, 14336, x="bf16", name="prompt_512"),
        # the longest prompt: the largest case
        _linear(8192, 14336, 4096, x="bf16", name="prompt_8192"),
        # a prompt of no round length through a whole MLP block
        {"name": "mlp_block_prompt_1000", "kind": "mlp", "m": 1000, "hidden": 4096, "inter": 14336, "x": "bf16"},
        # one token of SmolLM2-135M: 30 layers of small dependent kernels
        {"name": "decode_step_30_layers", "kind": "stack", "layers": 30, "hidden": 576, "inter": 1536, "q_heads": 9,
         "kv_heads": 3, "vocab": 49152},
        # weights of the largest prefill layer back to float32
        {"name": "dequant_int4", "kind": "dequant", "bits": 4, "n": 4096, "k": 14336, "group": 32, "scales": "f16", "out": "f32"},
        # the same layer quantised when the model is loaded
        {"name": "quantize_int4", "kind": "quantize", "bits": 4, "n": 4096, "k": 14336, "group": 32, "x": "f32"},
    ]


def _log_int(rng, lo, hi, multiple=1):
    """An integer between lo and hi, uniform in its logarithm, rounded to a multiple (of 1: odd ones too)."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    what = rng.choices(("decode", "batch", "prompt", "float", "stack", "mlp", "dequant", "quantize"),
                       (6, 4, 3, 3, 2, 1, 2, 2))[0]
    if what == "decode":                           # M <= 16, any K that is whole groups of 64, any N
        k = _log_int(rng, 576, 28672, rng.choice((64, 256, 256)))
        return _linear(_log_int(rng, 1, 16), k, _log_int(rng, 192, min(128256, 8192 * 128256 // k)), x=rng.choice(("f16", "f16", "bf16")))
    if what == "batch":
        k = _log_int(rng, 576, 14336, rng.choice((64, 256, 256)))
        return _linear(_log_int(rng, 17, 512), k, _log_int(rng, 1024, 28672), x=rng.choice(("f16", "bf16")))
    if what == "prompt":
        m, k = _log_int(rng, 513, 8192), _log_int(rng, 2048, 14336, 256)
        n = _log_int(rng, 1024, 14336, 8)
        while 2.0 * m * k * n > LARGEST_FLOPS:
            m //= 2
        return _linear(m, k, n, x=rng.choice(("f16", "bf16", "bf16")))
    if what == "float":                            # the reference's types (float32), int8, other group sizes
        bits, group = rng.choice((4, 8)), rng.choice((32, 64, 128))
        kind = rng.choice(("f32", "f32", "f16"))
        return _linear(_log_int(rng, 1, 8), _log_int(rng, 512, 8192, 128), _log_int(rng, 192, 16384), bits=bits, group=group,
                       x=kind, scales=kind)
    if what == "stack":
        if rng.random() < 0.5:
            shape = {"hidden": 576, "inter": 1536, "q_heads": 9, "kv_heads": 3}
            layers = rng.randint(6, 30)
        else:
            shape = {"hidden": 2048, "inter": 8192, "q_heads": 32, "kv_heads": 32}
            layers = rng.randint(2, 8)
        return {"kind": "stack", "layers": layers, **shape, "vocab": 64 * rng.randint(256, 768)}
    if what == "mlp":
        step = rng.choice((64, 256, 256))
        hidden = _log_int(rng, 576, 4096, step)
        return {"kind": "mlp", "m": _log_int(rng, 100, 2048), "hidden": hidden, "inter": _log_int(rng, 2.5 * hidden, 3.5 * hidden, step),
                "x": rng.choice(("f16", "bf16"))}
    group = rng.choice((32, 32, 64, 128))
    k, n = _log_int(rng, 576, 14336, group), _log_int(rng, 192, 14336)
    if what == "dequant":
        return {"kind": "dequant", "bits": rng.choice((4, 4, 8)), "n": n, "k": k, "group": group, "scales": rng.choice(("f16", "f32")),
                "out": rng.choice(("f32", "f16", "bf16"))}
    return {"kind": "quantize", "bits": rng.choice((4, 4, 8)), "n": n, "k": k, "group": group, "x": rng.choice(("f32", "f16", "bf16"))}


# ------------------------------------------------------------------------------------------ inputs
def _packed(gen, n, k, bits, group, scales):
    if bits == 4:
        w = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
    else:
        w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device="cuda", generator=gen)
    s = torch.randn(n, k // group, device="cuda", generator=gen).abs_() * (0.02 if bits == 4 else 0.01)
    return w, s.to(KINDS[scales])


def _rows(gen, m, k, kind):
    return torch.randn(m, k, device="cuda", generator=gen).to(KINDS[kind])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    c = case
    if c["kind"] == "linear":
        w, s = _packed(gen, c["n"], c["k"], c["bits"], c["group"], c["scales"])
        return {"kind": "linear", "linear": L.QuantLinear(w, s, c["group"], c["bits"]), "x": _rows(gen, c["m"], c["k"], c["x"])}
    if c["kind"] == "stack":
        stack = L.DecodeStack(layers=c["layers"], hidden=c["hidden"], inter=c["inter"], q_heads=c["q_heads"], kv_heads=c["kv_heads"],
                              vocab=c["vocab"], fused=True, glue=True, seed=seed)
        stack.token.fill_(seed % c["vocab"])
        stack.capture()
        # what a token leaves behind: the logits, the hidden state, and each layer's q|k|v (which go to the KV cache).
        # The argmax runs in the step too; its one integer is not compared, since two logits may tie.
        return {"kind": "stack", "stack": stack, "outputs": [stack.logits, stack.hidden] + [call[2] for call in stack.calls[:-1:4]]}
    if c["kind"] == "mlp":
        h, i = c["hidden"], c["inter"]
        gate, up, down = (L.QuantLinear(*_packed(gen, n, k, 4, 32, "f16")) for n, k in ((i, h), (i, h), (h, i)))
        norm = (1 + 0.1 * torch.randn(h, device="cuda", generator=gen)).to(KINDS[c["x"]])
        return {"kind": "mlp", "gate": gate, "up": up, "down": down, "norm": norm, "x": _rows(gen, c["m"], h, c["x"])}
    if c["kind"] == "dequant":
        w, s = _packed(gen, c["n"], c["k"], c["bits"], c["group"], c["scales"])
        return {"kind": "dequant", "w": w, "scales": s, "n": c["n"], "k": c["k"], "group": c["group"], "bits": c["bits"], "out": c["out"]}
    w = (torch.randn(c["n"], c["k"], device="cuda", generator=gen) * 0.1).to(KINDS[c["x"]])
    return {"kind": "quantize", "w": w, "group": c["group"], "bits": c["bits"]}


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["linear"](state["x"])
    if kind == "stack":
        state["stack"].replay()
        return state["outputs"]
    if kind == "mlp":
        normed = L.rms_norm(state["x"], state["norm"])
        act = L.silu_mul(state["gate"](normed), state["up"](normed))
        return L.add_inplace(state["down"](act), state["x"])
    if kind == "dequant":
        return L.dequantize(state["w"], state["scales"], state["n"], state["k"], state["group"], bits=state["bits"], out_dtype=state["out"])
    q = L.quantize(state["w"], state["group"], bits=state["bits"])
    return q.w, q.scales


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _weight_bytes(n, k, bits, group, scales):
    return n * k * bits // 8 + n * (k // group) * BYTES[scales]


def work(case):
    c = case
    if c["kind"] == "linear":
        return {"bytes": _weight_bytes(c["n"], c["k"], c["bits"], c["group"], c["scales"]) + c["m"] * (c["k"] + c["n"]) * BYTES[c["x"]],
                "flops": 2.0 * c["m"] * c["n"] * c["k"]}
    if c["kind"] == "stack":
        h, i, qkv, o = c["hidden"], c["inter"], 64 * (c["q_heads"] + 2 * c["kv_heads"]), 64 * c["q_heads"]
        weights = c["layers"] * (h * qkv + o * h + 3 * h * i) + h * c["vocab"]
        norms = (2 * c["layers"] + 1) * h
        return {"bytes": weights // 2 + weights // 16 + 2 * (norms + h + c["vocab"] + c["layers"] * qkv), "flops": 2.0 * weights}
    if c["kind"] == "mlp":
        weights = 3 * c["hidden"] * c["inter"]
        return {"bytes": weights // 2 + weights // 16 + (2 * c["m"] + 1) * c["hidden"] * BYTES[c["x"]], "flops": 2.0 * c["m"] * weights}
    if c["kind"] == "dequant":
        return {"bytes": _weight_bytes(c["n"], c["k"], c["bits"], c["group"], c["scales"]) + c["n"] * c["k"] * BYTES[c["out"]],
                "flops": 1.0 * c["n"] * c["k"]}
    return {"bytes": c["n"] * c["k"] * BYTES[c["x"]] + _weight_bytes(c["n"], c["k"], c["bits"], c["group"], "f32"),
            "flops": 2.0 * c["n"] * c["k"]}


def tolerance(case):
    c = case
    if c["kind"] in ("dequant", "quantize"):
        return "exact"
    if c["kind"] == "linear":
        return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 5e-3}[c["x"]]}
    return {"rel": 1e-2}                           # a chain of 16-bit results, each rounded where it is stored
