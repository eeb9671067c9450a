"""Performance cases of the split W4A4 + tail linear.

What a program does with this package, by kind:

  linear   one `SplitLinear` forward: rotation + INT4 + tail split of the activations, then the fused linear.  Decode
           (1..64 rows), chunked prefill and speculative batches (65..1000 rows), prefill (up to 4096 rows); with and
           without a tail, with RMSNorm / SwiGLU fused, with a bias.
  layer    the four linears of a decoder layer in their order (qkv with the input norm; o; gate_up with the norm and
           SwiGLU; down on its result), called one by one or replayed as a CUDA graph, as serving loops do.
  adapter  `split_linear_forward` on q / k / v of one input: what a model patched module by module calls.
  prepare  `prepare_weight`: rotating and packing a weight matrix when a model is loaded.
  t4       the entry points named after the reference's extensions: select + pack of fp16 / bf16 activations, the INT4
           matmul, the epilogue that adds the INT4 tail; all buffers preallocated.
  gather   `SplitLinear(tail_engine="gather")`: the engine with the fixed summation order.

Widths are those the rotations are built for; layer shapes are the ones of bench.py (Qwen3-8B and Llama-3-8B
projections).  Activations are N(0, 1) with K/256 channels x50, weights N(0, 0.02), as in bench.py and the tests.
"""
import math

import torch

from tailquant_kernel_b200 import SplitLinear, interleave_gate_up, ops, split_linear_forward

WIDTHS = (512, 1024, 2048, 4096, 6144, 8192, 12288, 14336)
RATIOS = (0.0, 0.01, 0.05, 0.05, 0.05, 0.10)
QKV, HIDDEN = 6144, 4096                 # bench.py's layer: 32 query + 2 x 8 key / value heads of 128
LARGEST = 4096 * 28672 * 4096            # rows x channels x width of the largest listed case
MAX_ROWS = 4096


def listed():
    def linear(name, rows, n, k, ratio=0.05, norm=False, act=False, bias=False):
        return {"name": name, "kind": "linear", "rows": rows, "n": n, "k": k, "ratio": ratio, "norm": norm, "act": act,
                "bias": bias}
    return [
        # one token through one projection: the smallest call, launches and host work
        linear("decode_1_o", 1, 4096, 4096),
        # one token through a layer in a captured graph: what a serving loop replays
        {"name": "decode_1_layer_graph", "kind": "layer", "rows": 1, "inter": 12288, "ratio": 0.05, "graph": True},
        # a decode batch, the widest projection with its fused norm and activation
        linear("decode_24_gate_up", 24, 24576, 4096, norm=True, act=True),
        # verification of drafted tokens / a nearly full decode batch, odd count
        linear("decode_61_down", 61, 4096, 12288),
        # a short prompt or a prefill chunk, ragged; block-diagonal rotation
        linear("chunk_300_down", 300, 4096, 14336, bias=True),
        # the headline: a layer's linears at 2048 tokens
        {"name": "prefill_2048_layer", "kind": "layer", "rows": 2048, "inter": 12288, "ratio": 0.05, "graph": False},
        # the largest projection of the Llama sweep
        linear("prefill_4096_gate_up", 4096, 28672, 4096, ratio=0.01, norm=True, act=True),
        # pure W4A4 (a policy entry of ratio 0)
        linear("w4a4_1000_qkv", 1000, 6144, 4096, ratio=0.0),
        # a patched model's q / k / v
        {"name": "adapter_777_qkv", "kind": "adapter", "rows": 777, "nq": 4096, "nkv": 1024, "k": 4096, "ratio": 0.05},
        # loading a model: the fused gate_up matrix, with every layout that decode and prefill read
        {"name": "prepare_gate_up", "kind": "prepare", "n": 24576, "k": 4096, "t16": True, "t4": False},
        # the reference's own sequence of extension calls
        {"name": "t4_256_fp16", "kind": "t4", "rows": 256, "n": 4096, "k": 4096, "ratio": 0.01, "fp16": True},
        # exact-order engine
        linear("gather_200_o", 200, 4096, 4096) | {"kind": "gather"},
    ]


def _spread(rng, lo, hi, step=1):
    """A multiple of `step` from lo to hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choices(("linear", "layer", "adapter", "prepare", "t4", "gather"), (9, 4, 2, 2, 2, 1))[0]
    ratio = rng.choice(RATIOS)
    if kind == "layer":
        inter = rng.choice((12288, 14336))
        rows = _spread(rng, 1, 2048)
        return {"kind": kind, "rows": rows, "inter": inter, "ratio": ratio, "graph": rows <= 64 and rng.random() < 0.5}
    if kind == "adapter":
        nkv = _spread(rng, 256, 2048, 8)
        return {"kind": kind, "rows": _spread(rng, 1, MAX_ROWS), "nq": nkv * rng.choice((1, 2, 4)), "nkv": nkv,
                "k": rng.choice(WIDTHS), "ratio": ratio}
    if kind == "prepare":
        k = rng.choice(WIDTHS)
        t4 = rng.random() < 0.3
        return {"kind": kind, "n": _spread(rng, 256, 24576 * 4096 // max(k, 4096), 8), "k": k, "t16": not t4, "t4": t4}
    if kind == "t4":
        fp16 = rng.random() < 0.7
        return {"kind": kind, "rows": _spread(rng, 1, 2048), "n": _spread(rng, 512, 12288, 8),
                "k": rng.choice((4096, 12288)) if fp16 else rng.choice(WIDTHS), "ratio": rng.choice((0.005, 0.01, 0.02, 0.05)),
                "fp16": fp16}
    k = rng.choice(WIDTHS)
    if kind == "gather":
        return {"kind": kind, "rows": _spread(rng, 1, 512), "n": _spread(rng, 512, 8192, 8), "k": k,
                "ratio": max(ratio, 0.01), "norm": False, "act": False, "bias": rng.random() < 0.3}
    n = _spread(rng, 256, 28672, 16)
    rows = _spread(rng, 1, max(1, min(MAX_ROWS, LARGEST // (n * k))))
    act = rng.random() < 0.25
    return {"kind": kind, "rows": rows, "n": n, "k": k, "ratio": ratio, "norm": rng.random() < 0.4, "act": act,
            "bias": not act and rng.random() < 0.25}


# ------------------------------------------------------------------------------------------------ inputs
class _Maker:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def randn(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float32)

    def activations(self, rows, k):
        x = self.randn(rows, k)
        hot = torch.randperm(k, generator=self.g, device="cuda")[: max(1, k // 256)]
        x[:, hot] *= 50.0
        return x.to(torch.bfloat16)

    def weight(self, n, k):
        return torch.randn(n, k, generator=self.g, device="cuda", dtype=torch.bfloat16) * 0.02

    def gamma(self, k):
        return (1.0 + 0.1 * self.randn(k)).to(torch.bfloat16)


def _linear(m, c, engine="mma"):
    w = m.weight(c["n"], c["k"])
    if c["act"]:
        w = interleave_gate_up(w[: c["n"] // 2], w[c["n"] // 2:])
    lin = SplitLinear(w, bias=0.1 * m.randn(c["n"]) if c["bias"] else None, ratio=c["ratio"], tail_engine=engine,
                      epilogue="swiglu" if c["act"] else "none", rms_weight=m.gamma(c["k"]) if c["norm"] else None)
    if c["rows"] <= lin.small_m and engine == "mma":
        lin.prepare_decode()
    return lin


def prepare(case, seed):
    m, kind = _Maker(seed), case["kind"]
    if kind in ("linear", "gather"):
        return {"kind": "linear", "layer": _linear(m, case, "gather" if kind == "gather" else "mma"),
                "x": m.activations(case["rows"], case["k"])}
    if kind == "layer":
        mk = lambda n, k, norm, act: _linear(m, {"n": n, "k": k, "norm": norm, "act": act, "bias": False,  # noqa: E731
                                                 "ratio": case["ratio"], "rows": case["rows"]})
        s = {"kind": "layer", "qkv": mk(QKV, HIDDEN, True, False), "o": mk(HIDDEN, HIDDEN, False, False),
             "gate_up": mk(2 * case["inter"], HIDDEN, True, True), "down": mk(HIDDEN, case["inter"], False, False),
             "hidden": m.activations(case["rows"], HIDDEN), "attn": m.activations(case["rows"], HIDDEN),
             "post": m.activations(case["rows"], HIDDEN)}
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _layer(s)
            torch.cuda.current_stream().wait_stream(side)
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["out"] = _layer(s)
        return s
    if kind == "adapter":
        return {"kind": "adapter", "weights": [m.weight(n, case["k"]) for n in (case["nq"], case["nkv"], case["nkv"])],
                "x": m.activations(case["rows"], case["k"]), "ratio": case["ratio"]}
    if kind == "prepare":
        return {"kind": "prepare", "w": m.weight(case["n"], case["k"]), "t16": case["t16"], "t4": case["t4"]}
    rows, n, k = case["rows"], case["n"], case["k"]
    dt = torch.float16 if case["fp16"] else torch.bfloat16
    r, rank, _ = ops.split_select_params(k, ops.ceil_ratio_count(k, case["ratio"]))
    e = lambda *shape, dtype: torch.empty(shape, dtype=dtype, device="cuda")  # noqa: E731
    return {"kind": "t4", "a": m.randn(rows, k).to(dt), "r": r, "rank": rank, "k": k,
            "w": ops.prepare_weight(m.weight(n, k), t16=False, t4=True),
            "pack": e(rows, k // 2, dtype=torch.uint8), "body": e(rows, dtype=torch.float32),
            "top": e(rows, dtype=torch.float32), "top_q": e(rows, r, dtype=torch.int8),
            "idx": e(rows, r, dtype=torch.int32), "out": e(rows, n, dtype=dt)}


# ------------------------------------------------------------------------------------------------ one pass
def _layer(s):
    return [s["qkv"](s["hidden"]), s["o"](s["attn"]), s["down"](s["gate_up"](s["post"]))]


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "layer":
        if "graph" in state:
            state["graph"].replay()
            return state["out"]
        return _layer(state)
    if kind == "adapter":
        x = state["x"].detach()  # a tensor of its own on each pass, as a model's previous layer makes it
        return [split_linear_forward(x, w, ratio=state["ratio"]) for w in state["weights"]]
    if kind == "prepare":
        w = ops.prepare_weight(state["w"], t16=state["t16"], t4=state["t4"], keep_w_rot=state["t16"])
        return [t for t in (w.b_col, w.w_scale, w.w_rot, w.w_t, w.b_row) if t is not None]
    s = state
    ops.threshold_topr_pack(s["a"], s["r"], s["rank"], s["pack"], s["body"], s["top"], s["top_q"], s["idx"], ops.EPS)
    c = ops.matmul(s["pack"], s["w"].b_col)
    ops.scale_sparse_epilogue_oct(c, s["body"], s["top_q"], s["idx"], s["w"].b_row, s["top"], s["w"].w_scale, s["out"],
                                  s["k"])
    return [s["pack"], s["body"], s["top"], s["top_q"], s["idx"], c, s["out"]]


# ------------------------------------------------------------------------------------------------ what it takes
def _linear_work(rows, n, k, ratio, n_out=None):
    r = ops.ceil_ratio_count(k, ratio)
    used = k * (1.0 - (1.0 - r / k) ** rows)  # rows of the bf16 weights that some token's tail names
    return (2.0 * rows * k + n * k / 2 + 4 * n + 2.0 * used * n + 2.0 * rows * (n_out or n),
            2.0 * rows * n * (k + r))


def work(case):
    kind = case["kind"]
    if kind == "layer":
        rows, inter = case["rows"], case["inter"]
        parts = [_linear_work(rows, QKV, HIDDEN, case["ratio"]), _linear_work(rows, HIDDEN, HIDDEN, case["ratio"]),
                 _linear_work(rows, 2 * inter, HIDDEN, case["ratio"], inter),
                 _linear_work(rows, HIDDEN, inter, case["ratio"])]
    elif kind == "adapter":
        parts = [_linear_work(case["rows"], case["nq"] + 2 * case["nkv"], case["k"], case["ratio"])]
    elif kind == "prepare":
        nk = float(case["n"] * case["k"])
        parts = [(nk * (2 + 0.5 + (4.0 if case["t16"] else 0.0) + (0.5 if case["t4"] else 0.0)), 0.0)]
    elif kind == "t4":
        rows, n, k = case["rows"], case["n"], case["k"]
        r = ops.ceil_ratio_count(k, case["ratio"])
        used = k * (1.0 - (1.0 - r / k) ** rows)
        parts = [(2.5 * rows * k + 5.0 * rows * r + n * k / 2 + used * n / 2 + 6.0 * rows * n, 2.0 * rows * n * (k + r))]
    else:
        parts = [_linear_work(case["rows"], case["n"], case["k"], case["ratio"],
                              case["n"] // 2 if case["act"] else case["n"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """The codes, indices and scales are specified to the bit; sums of the tail may be taken in another order, which
    moves a bf16 result by a last place now and then.  In a layer the down projection quantises such a result again."""
    kind = case["kind"]
    if kind == "prepare":
        return "exact"
    if kind == "layer":
        return {"rel": 5e-3, "max": 5e-2}
    return {"rel": 2e-3, "max": 1.6e-2, "differ": 0.0}
