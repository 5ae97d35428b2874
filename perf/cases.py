"""The work that users of this package have it do, as cases that can be timed and compared.

Two kinds of case, both through the public entry points:

  step   one ``Muon(...).step()`` over a set of parameters that hold their gradients (with the
         ``FusedAdamW`` companion in the ``scalar_optimizer`` slot where the case has scalar rows);
         outputs: parameters, momentum buffers and the companion's parameters and moments
  ns     one batched Newton-Schulz call of ``CutlassNSInt8`` on a stack of matrices, by the entry
         point that its router names; output: the orthogonalised stack

Sizes are those of this repository's benchmark configurations, tests and examples, or generic ones.
Matrix sets are written as text: "768x3072*4 768x768*8" is four matrices of 768 x 3072 and eight of
768 x 768.  Momentum is the optimizer's default (0.95, 0.95) everywhere.
"""
import math

import torch

from i8muon_b200 import CutlassNSInt8, FusedAdamW, Muon, recommend_coefficients

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
SIZES = {"fp32": 4, "bf16": 2, "fp16": 2}


def _step(name, matrices, dtype, precision, graph=False, schedule="int8_safe", iters=5, decay=0.01, adjust="match_rms_adamw",
          scalar_rows=0, scalar_cols=0):
    case = dict(kind="step", matrices=matrices, dtype=dtype, precision=precision, graph=graph, schedule=schedule, iters=iters,
                decay=decay, adjust=adjust, scalar_rows=scalar_rows, scalar_cols=scalar_cols)
    return dict(case, name=name) if name else case


def _ns(name, batch, rows, cols, dtype, precision, gram=False, schedule="int8_safe", iters=5, std=0.02, outliers=False):
    case = dict(kind="ns", batch=batch, rows=rows, cols=cols, dtype=dtype, precision=precision, gram=gram, schedule=schedule,
                iters=iters, std=std, outliers=outliers)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the first contact: a small MLP in FP32 with the optimizer's defaults; launches and host time are all there is
        _step("step-mlp-fp32-auto", "128x128*3 32x128 512x128 128x512", "fp32", "auto", decay=0.0, adjust="spectral"),
        # a small language model (768 wide, five layers) with the default precision: FP16 for the attention
        # outputs, global INT8 for the larger matrices; eager, as the default is
        _step("step-768-bf16-auto", "768x2304*5 768x768*5 3072x768*5 768x3072*5", "bf16", "auto"),
        # matrices whose sizes fit no tile (pruned or factorised layers, odd head counts), in BF16
        _step("step-ragged-bf16", "1000x3001*2 517x300*3 1531x1531 77x2049*2 2050x1366", "bf16", "bfloat16"),
        # 1.3B-shaped transformer (2048 wide, four of its layers), FP16 with the eight Polar Express rows, captured
        # graphs, the 50257-row embedding on the AdamW companion
        _step("step-2048-fp16-polar", "2048x2048*16 8192x2048*4 2048x8192*4", "bf16", "float16", graph=True,
              schedule="polar_express", iters=8, scalar_rows=50257, scalar_cols=2048),
        # 8B-shaped parameter set (four of its layers), block-quantised INT8, captured graphs: the largest
        _step("step-4096-int8bq", "4096x4096*8 1024x4096*8 14336x4096*8 4096x14336*4", "bf16", "int8_bq", graph=True),
        # the same shapes in E4M3 FP8, one layer, eager
        _step("step-4096-fp8bq", "4096x4096*2 1024x4096*2 14336x4096*2 4096x14336", "bf16", "fp8"),
        # the smallest call on the engine itself: a few heads' worth of small matrices
        _ns("ns-fp16-small", 4, 256, 256, "fp16", "float16"),
        # one FP32 matrix at full precision
        _ns("ns-fp32-single", 1, 1024, 4096, "fp32", "float32", std=1.0),
        # a tall, ragged FP32 batch
        _ns("ns-fp32-ragged", 6, 1537, 700, "fp32", "float32"),
        # the MLP matrices of a small language model stacked into one BF16 call
        _ns("ns-bf16-stack", 48, 768, 3072, "bf16", "bfloat16"),
        # wide matrices through the Gram-space iteration
        _ns("ns-bf16-gram", 48, 1024, 8192, "bf16", "bfloat16", gram=True),
        # global-scale INT8 on heavy-tailed FP32 gradients: the largest single call
        _ns("ns-int8-outliers", 16, 4096, 4096, "fp32", "int8", iters=6, std=1e-3, outliers=True),
    ]


def _log_uniform(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _size(rng, low, high):
    """A size of the range: a multiple of 64 as models have them, or (one in three) whatever it is."""
    v = _log_uniform(rng, low, high)
    return max(low, int(v) if rng.random() < 1 / 3 else 64 * max(1, round(v / 64)))


def draw(rng):
    while True:
        case = _draw_step(rng) if rng.random() < 0.5 else _draw_ns(rng)
        # no dearer than the largest listed case; FP32 products cost about six times as much each
        heavy = 6.0 if case["precision"] == "float32" else 1.0
        if work(case)["flops"] * heavy < 2.5e13:
            return case


def _draw_step(rng):
    d = _size(rng, 64, 4096)
    layers = rng.randint(1, 4)
    form = rng.choice(("mlp", "fused", "split", "gated"))
    if form == "mlp":
        shapes = [(4 * d, d, layers), (d, 4 * d, layers)]
    elif form == "fused":
        shapes = [(d, 3 * d, layers), (d, d, layers), (4 * d, d, layers), (d, 4 * d, layers)]
    elif form == "split":
        shapes = [(d, d, 4 * layers), (4 * d, d, layers), (d, 4 * d, layers)]
    else:
        kv, mlp = max(16, d // rng.choice((2, 4))), int(d * rng.choice((8 / 3, 3.5)))
        shapes = [(d, d, 2 * layers), (kv, d, 2 * layers), (mlp, d, 2 * layers), (d, mlp, layers)]
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp32", "fp16"))
    precision = rng.choice(("auto", "auto", "int8_bq", "fp8", "bfloat16", "float16", "int8") + (("float32",) if dtype == "fp32" else ()))
    polar = precision in ("float16", "float32") and rng.random() < 0.4
    scalar = rng.random() < 0.3
    return _step("", " ".join("%dx%d*%d" % s for s in shapes), dtype, precision, graph=rng.random() < 0.4,
                 schedule="polar_express" if polar else "int8_safe", iters=8 if polar else rng.choice((5, 5, 5, 6)),
                 decay=rng.choice((0.0, 0.01)), adjust=rng.choice(("spectral", "match_rms_adamw", "original")),
                 scalar_rows=rng.randint(1000, 50257) if scalar else 0, scalar_cols=d if scalar else 0)


def _draw_ns(rng):
    low = _size(rng, 32, 4096)
    high = int(low * rng.choice((1.0, 1.0, 2.0, 4.0, rng.uniform(1.0, 4.5))))
    precision = rng.choice(("auto", "int8", "int8_bq", "fp8", "bfloat16", "float16", "float32"))
    gram = precision in ("bfloat16", "float16") and low <= 2048 and rng.random() < 0.3
    if gram:
        high = low * 8
    dtype = "fp32" if precision == "float32" else rng.choice(("bf16", "fp16", "fp32"))
    most = max(1, min(48, int(3e8 / (low * high))))
    batch = int(_log_uniform(rng, 1, most + 0.99))
    rows, cols = (low, high) if rng.random() < 0.6 else (high, low)
    return _ns("", batch, rows, cols, dtype, precision, gram=gram, iters=rng.choice((5, 5, 6)),
               outliers=precision == "int8" and rng.random() < 0.5)


def _matrices(text):
    shapes = []
    for word in text.split():
        size, _, count = word.partition("*")
        rows, cols = size.split("x")
        shapes += [(int(rows), int(cols))] * int(count or 1)
    return shapes


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]

    def normal(shape, std):
        return torch.randn(shape, device="cuda", generator=gen).mul_(std).to(dtype)

    rows = recommend_coefficients(case["iters"], method=case["schedule"])
    if case["kind"] == "ns":
        x = torch.randn((case["batch"], case["rows"], case["cols"]), device="cuda", generator=gen).mul_(case["std"])
        if case["outliers"]:   # one entry in a hundred fifty times larger: the heavy tail of gradients
            x.mul_(torch.rand(x.shape, device="cuda", generator=gen).lt_(0.01).mul_(49.0).add_(1.0))
        return dict(kind="ns", x=x.to(dtype), engine=CutlassNSInt8(), coeffs=rows,
                    route=(case["rows"], case["cols"], case["precision"], case["gram"], 5.0))
    params = []
    for shape in _matrices(case["matrices"]):
        p = torch.nn.Parameter(normal(shape, 0.02))
        p.grad = normal(shape, 1e-3)
        params.append(p)
    scalars, scalar_optimizer = [], None
    if case["scalar_rows"]:
        for shape in [(case["scalar_rows"], case["scalar_cols"]), (case["scalar_cols"],)]:
            p = torch.nn.Parameter(normal(shape, 0.02))
            p.grad = normal(shape, 1e-3)
            scalars.append(p)
        scalar_optimizer = FusedAdamW(scalars, lr=1e-3)
    optimizer = Muon(params, lr=0.02, weight_decay=case["decay"], ns_coefficients=rows, adjust_lr_fn=case["adjust"],
                     precision=case["precision"], use_cuda_graph=case["graph"], scalar_optimizer=scalar_optimizer)
    return dict(kind="step", optimizer=optimizer, params=params, scalars=scalars, scalar_optimizer=scalar_optimizer)


def run(state):
    if state["kind"] == "ns":
        function, compute = state["engine"].router(*state["route"])
        return function(state["x"], coeffs=state["coeffs"], precision=compute)
    optimizer = state["optimizer"]
    optimizer.step()
    out = dict(params=[p.data for p in state["params"]],
               momentum=[optimizer.state[p]["momentum_buffer"] for p in state["params"]])
    if state["scalars"]:
        held = state["scalar_optimizer"].state
        out["scalars"] = [p.data for p in state["scalars"]]
        out["moments"] = [held[p][key] for p in state["scalars"] for key in ("exp_avg", "exp_avg_sq")]
    return out


def work(case):
    """Flops: per iteration a symmetric l x h x l product and a symmetric l x l x l product (one triangle of
    each) and the l x l x h update; in the Gram space only the first product and two restarts touch h.
    Bytes: a step reads gradients and reads and writes momentum and parameters; a call reads and writes its stack."""
    size = SIZES[case["dtype"]]
    if case["kind"] == "ns":
        shapes = [(case["rows"], case["cols"])] * case["batch"]
        total = 2.0 * size * sum(r * c for r, c in shapes)
    else:
        shapes = _matrices(case["matrices"])
        scalars = case["scalar_rows"] * case["scalar_cols"] + case["scalar_cols"]
        total = 5.0 * size * sum(r * c for r, c in shapes) + (3.0 * size + 16.0) * scalars
    flops = 0.0
    for r, c in shapes:
        low, high = float(min(r, c)), float(max(r, c))
        if case.get("gram", True) and high >= 5.0 * low:
            flops += 2 * low * low * high + case["iters"] * 2 * low ** 3 + 4 * low * low * high
        else:
            flops += case["iters"] * (3 * low * low * high + low ** 3)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Relative distance between two correct evaluations at the same precision, as this repository's tests state it."""
    shapes = [(case["rows"], case["cols"])] if case["kind"] == "ns" else _matrices(case["matrices"])
    gram = case.get("gram", True) and any(max(s) >= 5 * min(s) for s in shapes)
    if case["precision"] == "float32":
        return {"rel": 2e-5}   # each within 1e-5 of the exact iteration
    if gram and case["precision"] == "bfloat16":
        return {"rel": 3e-2}   # the Gram-space iteration amplifies BF16 rounding
    # five or more iterations of FP16 / BF16 products; eight-bit operands are coarser
    return {"rel": 1e-2 if case["precision"] in ("float16", "bfloat16") else 2e-2}
