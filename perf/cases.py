"""Performance cases of the attention library: the calls a user makes, over the sizes they are made at.

Every case is one forward pass (or one batch of them) through the package's public calls on tensors that stay in
device memory, enqueued on the current stream without waiting for it.  `listed()` has the cases, `draw()` picks more
from the ranges they stand for.  A case is
    family   which row of FAMILIES it belongs to
    dtype    "f32", "bf16" or "f16" (inputs and output; products accumulate in fp32)
    pe       positional encoding applied to Q and K: none, rope (interleaved pairs), rope_half, rope_half_q (K comes
             rotated), sinusoidal
    B H Lq Lk D   Q is [B, H, Lq, D], K and V are [B, H, Lk, D]
    n        independent problems per pass (1: one `forward`; more: one `forward_many`)
"""
import importlib
import math

import torch

b200attn = importlib.import_module("accelerated-final-project_b200")

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
PE = {"none": b200attn.PE_NONE, "rope": b200attn.PE_ROPE_INTERLEAVED, "rope_half": b200attn.PE_ROPE_HALF,
      "rope_half_q": b200attn.PE_ROPE_HALF_Q_ONLY, "sinusoidal": b200attn.PE_SINUSOIDAL}

# The ranges: (dtypes, encodings, batch * heads, query length, key length or None for "as the queries", head widths, n).
FAMILIES = {
    # fp32, sequences of 16 to 64, head_d 512 to 8192: what the library's fp32 entry points are called for; one call
    # at a time, so that the latency of a launch counts
    "f32_short": (("f32",), ("none",), (1, 32), (16, 64), (16, 64), (512, 1000, 1024, 2048, 4096, 8192), 1),
    # the same problems handed over as one batch of independent ones
    "f32_batch": (("f32",), ("none",), (1, 32), (16, 64), (16, 64), (512, 1024, 2048, 4096), 16),
    # the same regime with the positional encoding fused into the load
    "f32_short_pe": (("f32",), ("rope", "sinusoidal"), (1, 32), (16, 64), (16, 64), (512, 1000, 1024, 2048, 4096, 8192), 1),
    # fp32 at ordinary model sizes, where a caller wants no 16-bit rounding
    "f32_long": (("f32",), ("none", "rope"), (1, 32), (80, 2048), (80, 2048), (64, 128, 512), 1),
    # 16-bit tensors at the short, wide sizes of the fp32 path
    "b16_short": (("bf16", "f16"), ("none", "rope", "sinusoidal"), (1, 32), (16, 64), (16, 64), (512, 1024, 2048, 4096, 8192), 1),
    # decoding: one to a few queries against a long key cache whose keys are stored rotated
    "decode": (("bf16",), ("none", "rope_half_q"), (8, 128), (1, 16), (2000, 40000), (128,), 1),
    # self-attention of transformer models: the usual head widths, prefill lengths, ragged and whole
    "narrow": (("bf16", "f16"), ("none", "rope"), (8, 128), (100, 8192), None, (64, 128, 256), 1),
    # head widths that are not a multiple of 64, and keys of another length than the queries
    "narrow_odd": (("bf16",), ("none",), (8, 64), (100, 2048), (100, 2048), (80, 96, 160), 1),
    # wide heads on the tensor cores, with and without an encoding
    "wide": (("bf16",), ("none", "rope_half", "sinusoidal"), (8, 512), (300, 4096), None, (512, 1024), 1),
}


def _case(family, dtype, pe, B, H, Lq, Lk, D, n=1):
    return {"family": family, "dtype": dtype, "pe": pe, "B": B, "H": H, "Lq": Lq, "Lk": Lk, "D": D, "n": n}


def listed():
    cases = {
        # the smallest call of the fp32 regime: all latency
        "f32_small": _case("f32_short", "f32", "none", 1, 4, 64, 64, 512),
        # its widest head: 25 MB of inputs, one call on its own
        "f32_wide": _case("f32_short", "f32", "none", 1, 4, 64, 64, 8192),
        # sixteen independent problems of the middle size in one call
        "f32_batch": _case("f32_batch", "f32", "none", 1, 4, 64, 64, 2048, n=16),
        # the rotary encoding fused into the fp32 path
        "f32_rope": _case("f32_short_pe", "f32", "rope", 1, 4, 64, 64, 2048),
        # fp32 attention of a small model over a ragged thousand tokens
        "f32_long": _case("f32_long", "f32", "none", 1, 8, 1000, 1000, 64),
        # the bf16 drop-in with the sinusoidal encoding at the short, wide size
        "bf16_short": _case("b16_short", "bf16", "sinusoidal", 1, 4, 64, 64, 2048),
        # four new tokens against a cache of 32768 keys
        "decode": _case("decode", "bf16", "rope_half_q", 1, 32, 4, 32768, 128),
        # prefill at the most common head width
        "narrow128": _case("narrow", "bf16", "none", 4, 16, 4096, 4096, 128),
        # fp16, narrow heads, ragged length, rotary encoding
        "narrow64_f16": _case("narrow", "f16", "rope", 8, 12, 1000, 1000, 64),
        # cross-attention at a head width between the tile sizes
        "narrow96": _case("narrow_odd", "bf16", "none", 2, 16, 777, 1000, 96),
        # head_d 1024 with the rotate-half encoding
        "wide1024": _case("wide", "bf16", "rope_half", 4, 32, 2048, 2048, 1024),
        # head_d 512 with the sinusoidal encoding: the benchmark's default workload, the largest
        "wide512": _case("wide", "bf16", "sinusoidal", 16, 32, 4096, 4096, 512),
    }
    return [dict(c, name=name) for name, c in cases.items()]


MAX_FLOPS = 4.0 * 16 * 32 * 4096 * 4096 * 512          # of the largest listed case
MAX_BYTES = 2.0 * 16 * 32 * 512 * 4 * 4096
F32_MAX_FLOPS = 4.0 * 32 * 2048 * 2048 * 64             # fp32 at model sizes, and the odd head widths


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], uniform in its logarithm where the range spans more than a factor of ten."""
    if hi > 10 * lo:
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    return rng.randint(lo, hi)


def draw(rng):
    while True:
        family = rng.choice(sorted(FAMILIES))
        dtypes, pes, bh, lq, lk, widths, n = FAMILIES[family]
        BH = _spread(rng, *bh)
        B = rng.choice([b for b in (1, 2, 4, 8, 16) if BH % b == 0])
        Lq = _spread(rng, *lq)
        c = _case(family, rng.choice(dtypes), rng.choice(pes), B, BH // B, Lq, Lq if lk is None else _spread(rng, *lk), rng.choice(widths), n)
        w = work(c)
        limit = F32_MAX_FLOPS if family in ("f32_long", "narrow_odd") else MAX_FLOPS
        if w["flops"] <= limit and w["bytes"] <= MAX_BYTES:
            return c


def _tensors(case, gen):
    td = DTYPES[case["dtype"]]
    out = []
    for L in (case["Lq"], case["Lk"], case["Lk"]):
        t = torch.empty((case["B"], case["H"], L, case["D"]), dtype=td, device="cuda")
        # the fp32 entry points' own test inputs are uniform in [-1, 1); activations are nearer to normal
        t.uniform_(-1.0, 1.0, generator=gen) if case["dtype"] == "f32" else t.normal_(generator=gen)
        out.append(t)
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    problems = []
    for _ in range(case["n"]):
        Q, K, V = _tensors(case, gen)
        problems.append((Q, K, V, torch.empty_like(Q)))
    state = {"pe": PE[case["pe"]], "problems": problems, "args": None}
    if case["n"] > 1:
        # the descriptors of a batch are filled once and handed over on every pass
        state["args"] = [b200attn.args_for(Q, K, V, out, pe=state["pe"], flags=b200attn.FLAG_ASYNC) for Q, K, V, out in problems]
    return state


def run(state):
    if state["args"] is not None:
        b200attn.forward_many(state["args"])
        return [out for _, _, _, out in state["problems"]]
    Q, K, V, out = state["problems"][0]
    return b200attn.forward(Q, K, V, out=out, pe=state["pe"], flags=b200attn.FLAG_ASYNC)


def work(case):
    esz = 4 if case["dtype"] == "f32" else 2
    heads = case["n"] * case["B"] * case["H"]
    return {"bytes": float(esz * heads * case["D"] * (2 * case["Lq"] + 2 * case["Lk"])),
            "flops": 4.0 * heads * case["Lq"] * case["Lk"] * case["D"]}


def tolerance(case):
    # Against the same pass in 64 bits: fp32 2e-7 to 3e-6 (the angles of a fp32 rotation at the far positions), bf16
    # 1.7e-3 to 4.7e-3 (operands and probabilities rounded to bf16), fp16 2e-4 to 4e-4.  Two implementations at the
    # same precision may err in different directions.
    return {"rel": {"f32": 1e-5, "bf16": 1e-2, "f16": 2e-3}[case["dtype"]]}
