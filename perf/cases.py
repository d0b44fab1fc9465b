"""What the speed of this package is measured on: the calls a user of it makes, over their range.

A user loads weights once (`quantize_weight`), decodes one token per sequence for a batch of
sequences (captured once per batch size in a CUDA graph and replayed, or eagerly), and runs
prompts through the same layers (eagerly, hundreds to thousands of rows).  Widths are those of
`projection_set.StackShapes` (hidden 4096, intermediate 12288, vocabulary 248320); `draw` varies
them over generic widths.  Mixers (scan, attention) are not part of this package: their outputs are
stood in for by N(0, 1) tensors, as in `projection_set`.

Operations (`op`):
  weight  `quantize_weight` of one [out, in] weight: loading a checkpoint
  linear  `linear` of one [rows, in] activation with one FP8 weight: the smallest call
  mlp     `mlp_forward` with the residual added: the MLP of one layer, eager
  layer   every projection of one decoder layer, eager: pre-norm -> project -> mixer output ->
          output projection (+ residual) -> pre-norm -> MLP (+ residual); `kind` "gdn" or "attn"
  step    one decode step of a stack of `layers` layers, every fourth an attention layer, captured
          in a CUDA graph as the engine's decoder captures it; a pass is one replay
  head    final norm -> greedy pick over the vocabulary, logits kept
"""
from __future__ import annotations

import math

import torch

from braid_b200 import quant as Q

EPS = 1e-6
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed():
    return [
        # one weight of a loaded checkpoint (32 layers hold 200 of them)
        {"name": "weight_load", "op": "weight", "out": 12288, "in": 4096, "dtype": "bf16"},
        # a single projection for a handful of sequences: the smallest call there is
        {"name": "linear_8_rows", "op": "linear", "rows": 8, "out": 4096, "in": 4096, "dtype": "bf16"},
        # an fp32 engine's K projection over a short ragged prompt
        {"name": "linear_fp32_ragged", "op": "linear", "rows": 413, "out": 1024, "in": 4096, "dtype": "fp32"},
        # one sequence decoded without a graph: launches and host work count
        {"name": "mlp_1_row", "op": "mlp", "rows": 1, "hidden": 4096, "dtype": "bf16"},
        # an eager decode layer at a small batch (engines that do not capture)
        {"name": "layer_16_rows", "op": "layer", "kind": "gdn", "rows": 16, "hidden": 4096, "dtype": "bf16"},
        # graphed decode: one sequence, an odd fp16 batch, the batch the package is quoted at
        {"name": "step_1_row", "op": "step", "layers": 4, "rows": 1, "hidden": 4096, "dtype": "bf16"},
        {"name": "step_27_rows_fp16", "op": "step", "layers": 4, "rows": 27, "hidden": 4096, "dtype": "fp16"},
        {"name": "step_128_rows", "op": "step", "layers": 4, "rows": 128, "hidden": 4096, "dtype": "bf16"},
        # the vocabulary projection of a decode batch
        {"name": "head_64_rows", "op": "head", "rows": 64, "hidden": 4096, "vocab": 248320, "dtype": "bf16"},
        # one short ragged prompt, a longer one, and 16 packed sequences
        {"name": "prompt_333_rows", "op": "layer", "kind": "gdn", "rows": 333, "hidden": 4096, "dtype": "bf16"},
        {"name": "prompt_1500_rows_fp16", "op": "layer", "kind": "attn", "rows": 1500, "hidden": 4096,
         "dtype": "fp16"},
        {"name": "prompt_9658_rows", "op": "layer", "kind": "gdn", "rows": 9658, "hidden": 4096, "dtype": "bf16"},
    ]


def _between(rng, lo, hi):
    """A whole number, spread evenly over the logarithm of the range."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    op = rng.choice(["weight", "linear", "linear", "mlp", "mlp", "layer", "layer", "layer", "step", "step",
                     "step", "head"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "bf16", "fp16", "fp16", "fp32"])
    hidden = rng.choice([1024, 2048, 2560, 4096, 4096, 5120])
    # no drawn pass costs more than the 9658-row layer
    most = min(9658, int(9658 * 4096 * 4096 / (hidden * hidden)))
    if dtype == "fp32":
        most = min(most, 4096)       # twice the bytes of activations
    if op == "weight":
        return {"op": op, "out": 16 * _between(rng, 16, 960), "in": hidden, "dtype": dtype}
    if op == "linear":
        return {"op": op, "rows": _between(rng, 1, most), "out": 16 * _between(rng, 32, 768), "in": hidden,
                "dtype": dtype}
    if op == "mlp":
        return {"op": op, "rows": _between(rng, 1, most), "hidden": hidden, "dtype": dtype}
    if op == "layer":
        return {"op": op, "kind": rng.choice(["gdn", "attn"]), "rows": _between(rng, 1, most), "hidden": hidden,
                "dtype": dtype}
    if op == "step":
        return {"op": op, "layers": 4, "rows": _between(rng, 1, 256), "hidden": hidden,
                "dtype": "bf16" if dtype == "fp32" else dtype}
    return {"op": op, "rows": _between(rng, 1, 256), "hidden": min(hidden, 4096),
            "vocab": 16 * rng.randint(2000, 15520), "dtype": "bf16" if dtype == "fp32" else dtype}


# ---- inputs -----------------------------------------------------------------------------------
class _Maker:
    def __init__(self, seed, dtype):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype = dtype

    def randn(self, *shape, std=1.0, dtype=None):
        x = torch.randn(*shape, generator=self.g, device="cuda")
        return (x * std).to(dtype or self.dtype)

    def activation(self, rows, cols):
        """N(0, 1) with 0.1 % of the entries 50 times larger, as residual streams have outliers."""
        x = torch.randn(rows, cols, generator=self.g, device="cuda")
        out = torch.rand(rows, cols, generator=self.g, device="cuda") < 1e-3
        return torch.where(out, x * 50.0, x).to(self.dtype)

    def gamma(self, n):
        return 1.0 + 0.1 * torch.randn(n, generator=self.g, device="cuda")

    def weight(self, n, k):
        """N(0, 0.02), quantized as a loader does; in bands, so that a vocabulary fits."""
        w = torch.empty(n, k, device="cuda", dtype=torch.bfloat16)
        for i in range(0, n, 16384):
            w[i:i + 16384] = torch.randn(min(16384, n - i), k, generator=self.g, device="cuda") * 0.02
        return Q.quantize_weight(w)


def _mlp_weights(m, hidden):
    inter = 3 * hidden
    return {"gate": m.weight(inter, hidden), "up": m.weight(inter, hidden), "down": m.weight(hidden, inter)}


def _layer(m, kind, rows, hidden):
    s = {"kind": kind, "norm1": m.gamma(hidden), "norm2": m.gamma(hidden), **_mlp_weights(m, hidden)}
    if kind == "gdn":
        gates = hidden // 128
        s.update(qkv=m.weight(2 * hidden, hidden), z=m.weight(hidden, hidden),
                 a=m.randn(gates, hidden, std=0.02), b=m.randn(gates, hidden, std=0.02),
                 out=m.weight(hidden, hidden), norm_h=m.gamma(128),
                 scan=m.randn(rows, hidden, dtype=torch.float32))
    else:
        s.update(q=m.weight(2 * hidden, hidden), k=m.weight(hidden // 4, hidden), v=m.weight(hidden // 4, hidden),
                 o=m.weight(hidden, hidden), attn=m.randn(rows, hidden))
    return s


def _run_layer(s, x):
    """The layer's calls as a decoder layer makes them; returns the projections and the output."""
    if s["kind"] == "gdn":
        h = Q.rms_norm_quant(x, s["norm1"], EPS, keep_dense=True)
        qkv, z, a, b = Q.project(h, s["qkv"], s["z"], s["a"], s["b"])
        core = Q.gated_rms_norm_quant(s["scan"], z, s["norm_h"], EPS, 128)
        x = Q.linear(core, s["out"], residual=x)
        seen = (qkv, z, a, b)
    else:
        h = Q.rms_norm_quant(x, s["norm1"], EPS)
        qg, k, v = Q.project(h, s["q"], s["k"], s["v"])
        heads = qg.shape[-1] // 512
        gate = qg.view(qg.shape[0], heads, 512)[..., 256:]
        with Q.residual_into(s["o"], x) as slot:
            y = Q.gated_output_projection(s["attn"], gate, s["o"])
        x = y if slot.taken else x + y
        seen = (qg, k, v)
    h = Q.rms_norm_quant(x, s["norm2"], EPS)
    return seen, Q.mlp_forward(h, s["gate"], s["up"], s["down"], residual=x)


def _run_stack(layers, x):
    for s in layers:
        seen, x = _run_layer(s, x)
    return seen, x


def _capture(fn):
    """Warm up on a side stream, then capture, as an engine's graphed decoder does."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


def prepare(case, seed):
    Q.warm_fused(True)
    op = case["op"]
    m = _Maker(seed, DTYPES[case["dtype"]])
    if op == "weight":
        return {"op": op, "w": m.randn(case["out"], case["in"], std=0.02)}
    if op == "linear":
        return {"op": op, "x": m.activation(case["rows"], case["in"]), "w": m.weight(case["out"], case["in"])}
    hidden, rows = case["hidden"], case["rows"]
    x = m.activation(rows, hidden)
    if op == "mlp":
        return {"op": op, "x": x, "res": m.randn(rows, hidden), **_mlp_weights(m, hidden)}
    if op == "layer":
        return {"op": op, "x": x, "layer": _layer(m, case["kind"], rows, hidden)}
    if op == "step":
        layers = [_layer(m, "attn" if i % 4 == 3 else "gdn", rows, hidden) for i in range(case["layers"])]
        graph, out = _capture(lambda: _run_stack(layers, x))
        return {"op": op, "graph": graph, "out": out, "layers": layers, "x": x}
    return {"op": op, "x": x, "norm": m.gamma(hidden), "w": m.weight(case["vocab"], hidden)}


def run(state):
    op = state["op"]
    if op == "weight":
        w = Q.quantize_weight(state["w"])
        return w.data.view(torch.uint8), w.scale
    if op == "linear":
        return Q.linear(state["x"], state["w"])
    if op == "mlp":
        return Q.mlp_forward(state["x"], state["gate"], state["up"], state["down"], residual=state["res"])
    if op == "layer":
        return _run_layer(state["layer"], state["x"])
    if op == "step":
        state["graph"].replay()
        return state["out"]
    h = Q.rms_norm_quant(state["x"], state["norm"], EPS)
    return Q.lm_head_argmax(h, state["w"], return_logits=True)


# ---- what a pass cannot do without ------------------------------------------------------------
def _layer_work(kind, rows, hidden, es):
    """Every weight once, the layer's inputs once, its outputs once."""
    gates = hidden // 128
    mlp = 9 * hidden * hidden
    if kind == "gdn":
        fp8 = 4 * hidden * hidden + mlp
        dense = 2 * gates * hidden
        outs = 3 * hidden + 2 * gates + hidden
        ins = es * hidden + 4 * hidden
    else:
        fp8 = 3 * hidden * hidden + hidden * hidden // 2 + mlp
        dense = 0
        outs = 2 * hidden + hidden // 2 + hidden
        ins = 2 * es * hidden
    return fp8 + es * dense + rows * (ins + es * outs), 2 * rows * (fp8 + dense)


def work(case):
    op = case["op"]
    es = 4 if case["dtype"] == "fp32" else 2
    if op == "weight":
        n = case["out"] * case["in"]
        return {"bytes": n * (es + 1), "flops": 3 * n}
    if op == "linear":
        m, n, k = case["rows"], case["out"], case["in"]
        return {"bytes": n * k + es * m * (k + n), "flops": 2 * m * n * k}
    m, h = case["rows"], case["hidden"]
    if op == "mlp":
        return {"bytes": 9 * h * h + 3 * es * m * h, "flops": 18 * m * h * h}
    if op == "layer":
        b, f = _layer_work(case["kind"], m, h, es)
        return {"bytes": b, "flops": f}
    if op == "step":
        got = [_layer_work("attn" if i % 4 == 3 else "gdn", m, h, es) for i in range(case["layers"])]
        return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}
    n = case["vocab"]
    return {"bytes": n * h + es * m * (h + n) + 8 * m, "flops": 2 * m * n * h}


def tolerance(case):
    if case["op"] == "weight":
        return "exact"
    if case["op"] == "head":
        # the codes are whole numbers and K is summed inside one accumulator; a logit on a rounding
        # boundary may move by one step of the output type, and a pick between equal logits with it
        return {"rel": 4e-3, "differ": 0.01}
    if case["op"] == "linear":
        return {"rel": 4e-3 if case["dtype"] != "fp32" else 1e-5}
    # a chain: one rounding of a 16-bit intermediate that falls the other way may move the scale of
    # a whole quantized activation by one step of that type, and some of its 3-bit codes with it
    return {"rel": 2e-2}
