"""Performance cases of the EXL3 projection engine: what a program that serves an EXL3-quantised model has the engine do.

A case is a dict of plain values; `prepare` makes what the program has in hand (weights, routing, activations, all from the
seed), `run` is one pass through the package's public entry points. The kinds:

  trunk   dense projections, one `linear` call each: a decode step's or a prompt's rows through attention, shared-expert
          or output projections. `shapes` x `bits` calls a pass.
  table   `matmul` of the quant-plugin table on HOST arrays: what a host application that binds the table calls.
  moe     a routed layer: `moe` / `moe_swiglu`, or with `shared` the layer's shared expert (a one-expert bank behind a
          sigmoid gate) and `moe_with_shared`.
  mixed   a routed layer whose experts were quantised at different rates (`mixed.mixed_rate_moe`).

Codes are uniform random halfwords (every pattern is a valid codeword), signs are random +-1, scaled by a power of two near
1/sqrt(in) for routed banks so that the SwiGLU product stays inside f16; activations are N(0, 1), router logits N(0, 1).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import turboexl3_b200 as t3
from turboexl3_b200 import mixed as mixed_rates
from turboexl3_b200 import synth
from turboexl3_b200 import table as quant_table

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
CODEBOOKS = {"mul1": t3.MUL1, "mcg": t3.MCG}
RATES = (1, 2, 3, 4, 5, 6, 8)


def trunk(name, shapes, bits, rows, dtype="f16", codebook="mul1"):
    return {"name": name, "kind": "trunk", "shapes": shapes, "bits": bits, "rows": rows, "dtype": dtype, "codebook": codebook}


def moe(name, hidden, inter, experts, topk, bits, rows, dtype="f16", codebook="mul1", router="softmax", shared=False, limit=0):
    return {"name": name, "kind": "moe", "hidden": hidden, "inter": inter, "experts": experts, "topk": topk, "bits": bits,
            "rows": rows, "dtype": dtype, "codebook": codebook, "router": router, "shared": shared, "limit": limit}


def listed():
    return [
        # one attention projection of a 2048-wide model for one token: the smallest call, all launch and latency
        trunk("linear_2048_1row", "2048x2048", "4", 1),
        # a 2048-wide trunk at one token, every bit width a pack may use: 21 calls
        trunk("trunk_sweep_1row", "2048x2048,2048x6144,6144x2048", "1,2,3,4,5,6,8", 1),
        # the largest attention projection of a 7168-wide model for one token, bf16 activations
        trunk("attn_o_1row", "16384x7168", "4", 1, "bf16"),
        # a decode batch of ragged size through an up projection
        trunk("linear_17rows", "2048x6144", "3", 17),
        # a host application's decode step through the plugin table: host arrays in and out
        {"name": "table_matmul_1row", "kind": "table", "in": 6144, "out": 2048, "bits": 4, "rows": 1, "dtype": "f16",
         "codebook": "mul1"},
        # a hybrid-MoE layer (512 experts, top-10, shared expert) for one token, and for a decode batch
        moe("moe_layer_1row", 2048, 512, 512, 10, 3, 1, shared=True),
        moe("moe_layer_29rows", 2048, 512, 512, 10, 3, 29, "bf16", shared=True),
        # a short prompt through a down projection
        trunk("linear_200rows", "6144x2048", "4", 200),
        # a long prompt through an up projection
        trunk("linear_4096rows", "2048x6144", "4", 4096),
        # the hybrid-MoE layer on a long prompt, experts at one rate
        moe("moe_layer_4096rows", 2048, 512, 512, 10, 3, 4096, shared=True),
        # the same layer with its experts at 2, 3 and 4 bits
        {"name": "mixed_rates_4096rows", "kind": "mixed", "hidden": 2048, "inter": 512, "experts": 512, "topk": 10,
         "bits": "2,3,4", "rows": 4096, "dtype": "f16", "codebook": "mul1", "router": "softmax"},
        # a large-MoE layer (256 experts of 7168 x 2048, top-8 sigmoid routing) on a long prompt
        moe("moe_large_8192rows", 7168, 2048, 256, 8, 4, 8192, "bf16", router="sigmoid"),
    ]


LARGEST_FLOPS = 2.0 * 8192 * 8 * 3 * 7168 * 2048
LARGEST_CODES = 256 * 3 * 7168 * 2048 * 4 // 8


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    return max(lo, min(hi, 128 * round(_log_int(rng, lo, hi) / 128)))


def _rows(rng, prompt):
    return _log_int(rng, 33, 8192) if prompt else _log_int(rng, 1, 32)


def draw(rng):
    """One more case: widths in steps of 128 (what the format takes), rows log-uniform over decode batches (1..32) or prompts
    (33 up), any bit width, dtype and codebook."""
    dtype = rng.choice(("f16", "bf16", "bf16", "f32"))
    codebook = rng.choice(("mul1", "mul1", "mcg"))
    router = rng.choice(("softmax", "sigmoid"))
    prompt = rng.random() < 0.5
    kind = rng.choice(("trunk", "trunk", "trunk", "table", "moe", "moe", "moe", "mixed"))
    if kind in ("trunk", "table"):
        in_dim, out_dim = _width(rng, 512, 16384), _width(rng, 512, 24576)
        while in_dim * out_dim > 16384 * 7168:
            in_dim, out_dim = _width(rng, 512, 16384), _width(rng, 512, 24576)
        if kind == "table":
            return {"kind": "table", "in": in_dim, "out": out_dim, "bits": rng.choice(RATES), "rows": _log_int(rng, 1, 32),
                    "dtype": "f16", "codebook": codebook}
        bits = sorted(rng.sample(RATES, rng.choice((1, 1, 3))))
        return {"kind": "trunk", "shapes": "%dx%d" % (in_dim, out_dim), "bits": ",".join(map(str, bits)),
                "rows": _rows(rng, prompt), "dtype": dtype, "codebook": codebook}
    while True:
        hidden, inter = _width(rng, 1024, 7168), _width(rng, 256, 2048)
        experts, topk = _log_int(rng, 32, 512), rng.randint(2, 10)
        rows = _rows(rng, prompt or kind == "mixed")
        bits = rng.choice(RATES)
        if (3 * experts * hidden * inter * 8 // 8 <= LARGEST_CODES and 6.0 * rows * topk * hidden * inter <= LARGEST_FLOPS / 2):
            break
    case = {"kind": kind, "hidden": hidden, "inter": inter, "experts": experts, "topk": topk, "rows": rows, "dtype": dtype,
            "codebook": codebook, "router": router}
    if kind == "mixed":
        case["bits"] = "2,3,4"
        return case
    shared = rng.random() < 0.5
    case.update(bits=bits, shared=shared, limit=0 if shared else rng.choice((0, 0, 10)))
    return case


# ---- inputs ----------------------------------------------------------------------------------------------------------


class _Source:
    """Seeded operands on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def codes(self, *shape):
        return torch.randint(-32768, 32768, shape, dtype=torch.int16, device="cuda", generator=self.gen)

    def signs(self, shape, magnitude=1.0):
        return torch.randint(0, 2, shape, device="cuda", generator=self.gen).mul_(2).sub_(1).mul(magnitude).to(torch.float16)

    def normal(self, shape, dtype):
        return torch.randn(shape, device="cuda", generator=self.gen).to(dtype)

    def linear(self, in_dim, out_dim, bits):
        return (self.codes(in_dim // 16, out_dim // 16, 16 * bits), self.signs((in_dim,)), self.signs((out_dim,)))

    def bank(self, experts, hidden, inter, bits):
        return t3.Bank(*(t3.Proj(self.codes(experts, i // 16, o // 16, 16 * bits), self.signs((experts, i)),
                                 self.signs((experts, o), synth.pow2_inv_sqrt(i)))
                         for i, o in ((hidden, inter), (hidden, inter), (inter, hidden))))

    def routing(self, rows, experts, topk, router):
        logits = torch.randn((rows, experts), device="cuda", generator=self.gen)
        probs = torch.softmax(logits, 1) if router == "softmax" else torch.sigmoid(logits)
        scores, inds = probs.topk(topk, 1)
        return inds.to(torch.int32), scores / scores.sum(1, keepdim=True)


def _linears(case):
    shapes = [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")]
    return [(i, o, int(b)) for i, o in shapes for b in case["bits"].split(",")]


class _TableWeight:
    """A linear held by the plugin table (released with its last user) and one step's host activations."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        trellis, suh, svh = synth.linear(seed, case["in"], case["out"], 16 * case["bits"])
        self.block = quant_table.Block('{"format":"exl3","codebook":"%s"}' % case["codebook"])
        verdict, self.weight = self.block.load_tensor(trellis, suh, svh, case["in"])
        if not (self.block.verdict.ok and verdict.ok):
            raise RuntimeError(self.block.verdict.why or verdict.why)
        self.x = rng.standard_normal((case["rows"], case["in"])).astype(np.float16)

    def __del__(self):
        quant_table.table().release(ctypes.byref(self.weight))
        self.block.close()


def prepare(case, seed):
    if case["kind"] == "table":
        return "table", _TableWeight(case, seed)
    src, dtype, dec = _Source(seed), DTYPES[case["dtype"]], t3.Decode(CODEBOOKS[case["codebook"]])
    rows = case["rows"]
    if case["kind"] == "trunk":
        calls = _linears(case)
        xs = {i: src.normal((rows, i), dtype) for i, _, _ in calls}
        return "trunk", [(xs[i], *src.linear(i, o, b), dec) for i, o, b in calls]
    hidden, inter, experts, topk = case["hidden"], case["inter"], case["experts"], case["topk"]
    inds, scores = src.routing(rows, experts, topk, case["router"])
    if case["kind"] == "mixed":
        # the rate of each expert, as the pack's producer chose it
        rates = np.random.default_rng(seed).choice([16 * int(b) for b in case["bits"].split(",")], experts)
        buckets = mixed_rates.bucket_by_rate(rates)
        buckets.bank_of, buckets.local_of = buckets.bank_of.cuda(), buckets.local_of.cuda()
        banks = [src.bank(len(m), hidden, inter, n // 16) for n, m in zip(buckets.rates, buckets.members)]
        return "mixed", (src.normal((rows, hidden), dtype), banks, buckets, inds, scores, dec)
    x = src.normal((1, rows, hidden), dtype)
    bank = src.bank(experts, hidden, inter, case["bits"])
    shared = None
    if case["shared"]:
        gate = torch.sigmoid(src.normal((1, rows, 1), torch.float32))
        shared = (src.bank(1, hidden, inter, case["bits"]), torch.zeros((1, rows, 1), dtype=torch.int32, device="cuda"), gate)
    return "moe", (x, bank, inds.view(1, rows, topk), scores.view(1, rows, topk), dec, shared, case["limit"])


# ---- one pass --------------------------------------------------------------------------------------------------------


def run(state):
    kind, s = state
    if kind == "trunk":
        return [t3.linear(*call) for call in s]
    if kind == "table":
        verdict, y = quant_table.matmul(s.weight, s.x)
        if not verdict.ok:
            raise RuntimeError(verdict.why)
        return y
    if kind == "mixed":
        return mixed_rates.mixed_rate_moe(*s)
    x, bank, inds, scores, dec, shared, limit = s
    if shared is not None:
        expert, first, gate = shared
        return t3.moe_with_shared(x, bank, inds, scores, dec, t3.moe(x, expert, first, gate, dec))
    return t3.moe_swiglu(x, bank, inds, scores, dec, limit) if limit else t3.moe(x, bank, inds, scores, dec)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------


def _linear_work(rows, in_dim, out_dim, bits, size):
    return in_dim * out_dim * bits / 8 + 2 * (in_dim + out_dim) + size * rows * (in_dim + out_dim), 2.0 * rows * in_dim * out_dim


def work(case):
    size = 4 if case["dtype"] == "f32" else 2
    rows = case["rows"]
    if case["kind"] == "table":
        parts = [_linear_work(rows, case["in"], case["out"], case["bits"], size)]
    elif case["kind"] == "trunk":
        calls = _linears(case)
        parts = [_linear_work(rows, i, o, b, size) for i, o, b in calls]
        # a call's x is another call's x where their widths agree
        parts.append((-size * rows * (sum(i for i, _, _ in calls) - sum({i for i, _, _ in calls})), 0.0))
    else:
        hidden, inter, experts, topk = case["hidden"], case["inter"], case["experts"], case["topk"]
        bits = [int(b) for b in str(case["bits"]).split(",")]
        # experts that this many rows reach under a uniform router
        reached = experts * (1.0 - (1.0 - topk / experts) ** rows)
        codes = 3 * hidden * inter * sum(bits) / len(bits) / 8 + 2 * (3 * hidden + 3 * inter)
        parts = [(reached * codes + 2 * size * rows * hidden + 8 * rows * topk, 6.0 * rows * topk * hidden * inter)]
        if case.get("shared"):
            parts.append((codes + 4 * rows, 6.0 * rows * hidden * inter))
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """The chain rounds to f16 after every rotation and every inner product, whatever the activations' type: a sum taken in
    another order flips a few of those roundings by one f16 step. bf16 results add one bf16 rounding."""
    return {"rel": 4e-3, "max": 2.5e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 1e-2}
