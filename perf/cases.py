"""The work that users of this library have it do, as a list of timed cases: single forward calls, training
steps (forward and backward), a whole attention layer, and steps whose tensors live in host memory.

`listed()` names twelve of them; `draw()` gives more of the same ranges.  Sizes are those of the
benchmark, its sweeps and the tests; inputs are seeded N(0,1) tensors as there.
"""
from __future__ import annotations

import math

import torch

from simplical_attn_b200 import TwoSimplicialAttention, TwoSimplicialSelfAttention, two_simplicial_attention
from simplical_attn_b200.host_pipeline import HostPipeline

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}

# What a case may say; what it leaves out has these values.
DEFAULTS = dict(
    kind="step",        # forward: inference call; step: forward + backward; layer: projections around it, forward + backward; host: host tensors
    dtype="bf16",
    B=1, N=512, H=4,
    Hkv=0,              # K/V heads; 0: as many as query heads
    D=64, w1=64, w2=64,
    layout="bnhd",      # storage order of the tensors: [B, N, H, D], or [B, H, N, D] passed as a transposed view
    k2_bias=0.0, v2_bias=0.0,
    halo1=0, halo2=0,   # K1/V1 (K2/V2) rows in front of the first query: a shard of a longer sequence
)


def listed():
    return [
        # One short sequence through the module for inference: a call that is all latency.
        dict(name="forward_tiny", kind="forward", B=1, N=256, H=2, D=64, w1=64, w2=16),
        # A training step of a toy model, the base shape of the benchmark's shape sweeps.
        dict(name="step_tiny", B=2, N=512, H=4, D=64, w1=32, w2=32),
        # fp32: the numerically careful small run (gradient checks, debugging against a reference).
        dict(name="step_fp32", dtype="fp32", B=1, N=256, H=2, D=64, w1=64, w2=16),
        # The narrow heads of the head-dimension sweep.
        dict(name="step_narrow_heads", B=2, N=512, H=4, D=32, w1=32, w2=32),
        # Prefill / evaluation of 8 K tokens, head-major storage.
        dict(name="forward_8k", kind="forward", B=2, N=8192, H=8, D=128, w1=512, w2=32, layout="bhnd"),
        # fp16, an odd length, grouped heads, w2 that is no power of two, both biases.
        dict(name="step_ragged_fp16", dtype="fp16", B=3, N=1999, H=6, Hkv=3, D=64, w1=200, w2=24, k2_bias=0.1, v2_bias=0.05),
        # An attention layer with its projections in a model of hidden size 1024, default windows.
        dict(name="layer_train", kind="layer", B=4, N=2048, H=16, D=64, w1=64, w2=64),
        # Short windows: the cheap corner of the window sweep.
        dict(name="step_short_window", B=4, N=8192, H=16, D=128, w1=128, w2=16),
        # Grouped heads at length: 16 query heads to a KV head.
        dict(name="step_gqa_16k", B=1, N=16384, H=32, Hkv=2, D=128, w1=512, w2=32),
        # One rank's share of a 64 K sequence cut along its length eight ways: halo rows in front of the K/V tensors.
        dict(name="step_shard", B=1, N=8192, H=16, D=128, w1=1024, w2=64, halo1=1023, halo2=63),
        # Host tensors in, host tensors out.
        dict(name="host_8k", kind="host", B=2, N=8192, H=16, D=128, w1=512, w2=32),
        # The benchmark's workload: a full training batch.
        dict(name="step_8k", B=16, N=8192, H=16, D=128, w1=512, w2=32),
    ]


def _full(case):
    c = dict(DEFAULTS, **{k: v for k, v in case.items() if k != "name"})
    c["Hkv"] = c["Hkv"] or c["H"]
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "forward", "layer", "host"], [55, 25, 10, 10])[0]
    dtype = rng.choices(["bf16", "fp16", "fp32"], [75, 15, 10])[0] if kind in ("step", "forward") else "bf16"
    D = rng.choices([64, 128, 32, 256], [35, 50, 10, 5])[0] if dtype != "fp32" and kind != "host" else rng.choice([64, 128])
    small = dtype == "fp32" or D not in (64, 128)       # what users run at toy sizes
    Hkv = rng.choice([1, 2, 3, 4, 8, 16])
    group = rng.choice([1, 1, 1, 2, 4, 8] if kind != "layer" else [1, 1, 2])
    N = _log_int(rng, 64, 1024 if small else 16384)
    B = _log_int(rng, 1, 8 if small else 16)
    w1 = rng.choice([_log_int(rng, 16, 1024), rng.choice([32, 64, 128, 256, 512, 1024])])
    w2 = rng.choice([_log_int(rng, 4, 128), rng.choice([16, 32, 64])])
    c = dict(kind=kind, dtype=dtype, B=B, N=N, H=Hkv * group, Hkv=Hkv, D=D, w1=w1, w2=w2)
    if kind in ("step", "forward"):
        if rng.random() < 0.25:
            c["layout"] = "bhnd"
        if rng.random() < 0.2:
            c["k2_bias"], c["v2_bias"] = 0.1, 0.05
        if rng.random() < 0.15:
            c["halo1"], c["halo2"] = w1 - 1, w2 - 1
    # No case beyond a share of the benchmark's workload (of a toy run's, for the types used at toy sizes).
    most_flops, most_rows = (4e10, 1 << 15) if small else (2e13, 1 << 20)
    while work(c)["flops"] > most_flops or c["B"] * c["N"] * c["H"] > most_rows:
        if c["B"] > 1:
            c["B"] = max(1, int(c["B"] * 0.7))
        elif c["N"] > 256:
            c["N"] = int(c["N"] * 0.8)
        elif c["H"] > c["Hkv"]:
            c["H"] = c["Hkv"]
        elif c["Hkv"] > 1:
            c["H"] = c["Hkv"] = c["Hkv"] // 2
        else:
            c["w1"] = int(c["w1"] * 0.8)
            c["halo1"] = min(c.get("halo1", 0), c["w1"] - 1)
    return c


def _randn(g, c, rows, heads, dtype):
    if c["layout"] == "bhnd":
        return torch.randn(c["B"], heads, rows, c["D"], generator=g, device="cuda", dtype=dtype).transpose(1, 2)
    return torch.randn(c["B"], rows, heads, c["D"], generator=g, device="cuda", dtype=dtype)


def prepare(case, seed):
    c = _full(case)
    dtype = DTYPES[c["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(c=c)
    if c["kind"] == "layer":
        hidden = c["H"] * c["D"]
        with torch.device("cuda"):
            layer = TwoSimplicialSelfAttention(hidden, c["H"], c["D"], c["w1"], c["w2"], kv_heads=c["Hkv"], dtype=dtype)
        with torch.no_grad():
            for p in layer.parameters():
                p.copy_(torch.randn(p.shape, generator=g, device="cuda", dtype=dtype) / math.sqrt(p.shape[1]))
        s["layer"] = layer
        s["x"] = torch.randn(c["B"], c["N"], hidden, generator=g, device="cuda", dtype=dtype).requires_grad_(True)
        s["dy"] = torch.randn(c["B"], c["N"], hidden, generator=g, device="cuda", dtype=dtype)
        s["wrt"] = [s["x"]] + list(layer.parameters())
        return s
    rows = (c["N"], c["N"] + c["halo1"], c["N"] + c["halo2"], c["N"] + c["halo1"], c["N"] + c["halo2"])
    heads = (c["H"],) + (c["Hkv"],) * 4
    inputs = [_randn(g, c, r, h, dtype) for r, h in zip(rows, heads)]
    if c["kind"] == "host":
        def pinned(t):
            return torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
        device_side = inputs + [_randn(g, c, c["N"], c["H"], dtype)]
        s["inputs"] = [pinned(t).copy_(t) for t in device_side]
        s["out"] = [pinned(device_side[i]) for i in (0, 0, 1, 2, 3, 4)]
        s["pipeline"] = HostPipeline("cuda")
        return s
    s["module"] = TwoSimplicialAttention(c["D"], c["w1"], c["w2"], k2_bias=c["k2_bias"], v2_bias=c["v2_bias"])
    s["inputs"] = inputs
    if c["kind"] == "step":
        s["inputs"] = [t.requires_grad_(True) for t in inputs]
        s["d_o"] = _randn(g, c, c["N"], c["H"], dtype)
    return s


def _attend(s):
    c = s["c"]
    if c["halo1"] or c["halo2"]:
        return two_simplicial_attention(*s["inputs"], c["w1"], c["w2"], None, c["k2_bias"], c["v2_bias"], c["halo1"], c["halo2"])
    return s["module"](*s["inputs"])


def run(state):
    s = state
    kind = s["c"]["kind"]
    if kind == "forward":
        with torch.no_grad():
            return _attend(s)
    if kind == "step":
        o = _attend(s)
        return (o,) + torch.autograd.grad(o, s["inputs"], s["d_o"])
    if kind == "layer":
        y = s["layer"](s["x"])
        return (y,) + torch.autograd.grad(y, s["wrt"], s["dy"])
    return s["pipeline"].forward_backward(*s["inputs"], s["c"]["w1"], s["c"]["w2"], out=s["out"])


def _pairs(c):
    """(j, k) pairs over all queries of one head: windows are cut at the first row that exists."""
    total = 0
    ramp = min(c["N"], max(c["w1"], c["w2"]))
    for i in range(ramp):
        total += min(i + 1 + c["halo1"], c["w1"]) * min(i + 1 + c["halo2"], c["w2"])
    return total + (c["N"] - ramp) * c["w1"] * c["w2"]


def work(case):
    c = _full(case)
    size = 4 if c["dtype"] == "fp32" else 2
    # one contraction: 2 D flops per pair; forward has two of them, backward six
    unit = 2.0 * c["B"] * c["H"] * c["D"] * _pairs(c)
    q = c["B"] * c["N"] * c["H"] * c["D"] * size
    kv = 2 * c["B"] * (2 * c["N"] + c["halo1"] + c["halo2"]) * c["Hkv"] * c["D"] * size // 2
    if c["kind"] == "forward":
        return {"bytes": 2 * q + kv, "flops": 2 * unit}
    if c["kind"] == "layer":
        hidden = c["H"] * c["D"]
        widths = (2 * c["H"] + 4 * c["Hkv"]) * c["D"]             # in_proj and out_proj
        x = c["B"] * c["N"] * hidden * size
        return {"bytes": 4 * x + 2 * hidden * widths * size,
                "flops": 8 * unit + 6.0 * c["B"] * c["N"] * hidden * widths}
    return {"bytes": 4 * q + 2 * kv, "flops": 8 * unit}           # inputs and dO read, O and the gradients written


def tolerance(case):
    # P, dS and the operand products are rounded to the tensors' type before the contractions
    return {"rel": {"bf16": 1e-2, "fp16": 3e-3, "fp32": 2e-5}[_full(case)["dtype"]]}
