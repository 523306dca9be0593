"""The prefill GEMM's epilogue and the prepare where their variants meet: row tiles either side of the heights whose accumulators are
given back early (80 rows in pairs of output blocks, 128 one at a time), an odd last block, the prepare's walk over runs of positions
with sign and general scales mixed, and the one-expert chain that stores its rows without a final sum."""
import numpy as np
import pytest
import torch

import turboexl3_b200 as t3
from oracle import binding as ob
from turboexl3_b200 import synth

from gpu_util import TORCH_DT, bits16, check, dev, host_f32, x_as
from test_gpu_moe import check_moe, make_bank

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(640, 384, 48, t3.MUL1, "f16"), (384, 640, 64, t3.MCG, "f32"), (640, 384, 36, t3.MUL1, "bf16")])
def test_tile_heights_around_the_early_release(case):
    """A hundred experts, so that blocks go in pairs; neighbouring tiles alternate between early and late ones."""
    hidden, inter, n, cb, dt = case
    heights = [64, 79, 80, 81, 95, 96, 97, 112, 127, 128, 129, 16, 80, 144, 1, 80, 33, 256, 17, 48] * 5
    E = len(heights)
    bank, obank = make_bank(3100 + n, E, hidden, inter, n)
    inds = np.repeat(np.arange(E), heights).astype(np.int32)
    np.random.default_rng(3).shuffle(inds)
    rows = inds.size
    x = x_as(synth.activations(3101, rows, hidden), dt)
    y = t3.moe(x.view(1, rows, hidden), bank, dev(inds).view(1, rows, 1), torch.ones((1, rows, 1), device="cuda"), t3.Decode(cb, 16))
    sample = sorted({int(r) for e in range(0, E, 3) for r in np.flatnonzero(inds == e)[[0, -1]]})
    ref = ob.moe_rows(obank, host_f32(x)[sample], inds[sample].reshape(-1, 1), np.ones((len(sample), 1), np.float32), cb, 16, 0.0, 0)
    check_moe(host_f32(y).reshape(rows, hidden)[sample], ref, dt, ("early release", case))
    # a row's bytes do not depend on the tile it is in: the same rows of three experts in a call of their own
    few = np.flatnonzero(np.isin(inds, (3, 10, 17)))[:400]
    part = t3.moe(x[few].contiguous().view(1, few.size, hidden), bank, dev(inds[few]).view(1, few.size, 1),
                  torch.ones((1, few.size, 1), device="cuda"), t3.Decode(cb, 16))
    assert torch.equal(y.view(rows, hidden)[few], part.view(few.size, hidden))
    assert t3.device_error() == 0


@pytest.mark.parametrize("in_dim,out_dim,n,dt", [(256, 2560, 64, "f16"), (384, 128, 48, "bf16"), (256, 2560, 64, "f32")])
def test_dense_tiles_of_up_to_128_rows(in_dim, out_dim, n, dt):
    """One block at a time, tiles of 128 rows and fewer: several to a CTA, each freed before its rotation."""
    trellis, suh, svh = synth.linear(3110 + n, in_dim, out_dim, n, scaled=True)
    what = ob.reconstruct_inner(trellis, in_dim, out_dim, n, t3.MUL1, 16)
    t, a, b = dev(trellis), dev(suh), dev(svh)
    for rows in (120, 128, 1000, 2500):
        x = x_as(synth.activations(3111 + rows, rows, in_dim), dt)
        y = t3.linear(x, t, a, b)
        sample = sorted({0, 15, 16, 95, 96, 111, rows // 2, rows - 17, rows - 1})
        check(host_f32(y)[sample], ob.linear_rows_what(host_f32(x)[sample], what, suh, svh, in_dim, out_dim), dt, ("tiles to 128", in_dim, rows))
    assert t3.device_error() == 0


def test_the_prepare_walks_runs_of_positions():
    """Calls large enough that a quad of the prepare walks several positions (a ragged last run, nine blocks a row): the bytes of
    the same rows in a small call, where each position is prepared on its own. Every third expert's scales are not signs."""
    H, I, E, topk, n, rows = 1152, 128, 24, 7, 32, 4603
    rng = np.random.default_rng(3120)
    arrs = synth.bank(3121, E, H, I, n)
    for k in ("gate_suh", "up_suh"):
        arrs[k][::3] = (arrs[k][::3].astype(np.float32) * rng.uniform(0.5, 1.5, arrs[k][::3].shape)).astype(np.float16)
    d = {k: dev(v) for k, v in arrs.items()}
    bank = t3.Bank(*(t3.Proj(d[p + "_t"], d[p + "_suh"], d[p + "_svh"]) for p in ("gate", "up", "down")))
    inds, scores = synth.routing(3122, rows, E, topk)
    x = dev(synth.activations(3123, rows, H))
    call = lambda r: t3.moe(x[r].contiguous().view(1, -1, H), bank, dev(inds[r]).view(1, -1, topk), dev(scores[r]).view(1, -1, topk)).view(-1, H)
    whole = call(np.arange(rows))
    for r in (np.arange(40), np.arange(rows - 33, rows), np.arange(0, rows, 97)):
        assert torch.equal(whole[r], call(r))
    assert t3.device_error() == 0


@pytest.mark.parametrize("dt,score_dt", [("f16", torch.float32), ("bf16", torch.bfloat16), ("f32", torch.float16)])
def test_one_expert_prompts_are_weighted_in_the_epilogue(dt, score_dt):
    """A one-expert bank at one slot a row: the bytes of the same expert in a bank of two, which takes the final sum's launch."""
    H, I, n = 384, 256, 48
    arrs = synth.bank(3130, 2, H, I, n)
    bank = lambda e: t3.Bank(*(t3.Proj(*(dev(arrs[p + f][e]) for f in ("_t", "_suh", "_svh"))) for p in ("gate", "up", "down")))
    one, two = bank(slice(0, 1)), bank(slice(0, 2))
    obank = ob.Bank(2, H, I, n, *[arrs[p + f] for p in ("gate", "up", "down") for f in ("_t", "_suh", "_svh")])
    for rows in (33, 127, 129, 300, 2100):
        x = x_as(synth.activations(3131 + rows, rows, H), dt)
        scores = torch.from_numpy(np.random.default_rng(rows).standard_normal((rows, 1)).astype(np.float32)).cuda().to(score_dt)
        zeros = torch.zeros((1, rows, 1), dtype=torch.int32, device="cuda")
        y = t3.moe(x.view(1, rows, H), one, zeros, scores.view(1, rows, 1))
        assert y.dtype == TORCH_DT[dt]
        assert np.array_equal(bits16(y), bits16(t3.moe(x.view(1, rows, H), two, zeros, scores.view(1, rows, 1)))), rows
        sample = sorted({0, 31, 32, rows // 2, rows - 1})
        ref = ob.moe_rows(obank, host_f32(x)[sample], np.zeros((len(sample), 1), np.int32), scores.float().cpu().numpy()[sample])
        check_moe(host_f32(y).reshape(rows, H)[sample], ref, dt, ("one expert", dt, rows))
    assert t3.device_error() == 0
