"""The decode GEMM of the prefill rows at the sizes where its tiles can go wrong: tiles of every loaded height (32, 64, 96, 128,
192, 256 rows) with one row more and one less, both stage shapes (two blocks up to 128 rows, one block past that), an odd number
of 128-output blocks, the smallest K, and the two operand rings at the extreme rates."""
import numpy as np
import pytest
import torch

import turboexl3_b200 as t3
from oracle import binding as ob
from turboexl3_b200 import mixed, synth

from gpu_util import TORCH_DT, check, dev, host_f32, x_as
from test_gpu_moe import check_moe, make_bank

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(128, 128, 16, t3.MUL1, "f16"), (256, 384, 128, t3.MCG, "f32"), (384, 256, 36, t3.MUL1, "bf16"),
                                  (256, 128, 32, t3.MCG, "f16"), (128, 256, 64, t3.MUL1, "f32")])
def test_dense_tile_edges(case):
    in_dim, out_dim, n, cb, dt = case
    trellis, suh, svh = synth.linear(2100 + n, in_dim, out_dim, n, scaled=True)
    what = ob.reconstruct_inner(trellis, in_dim, out_dim, n, cb, 16)
    t, a, b = dev(trellis), dev(suh), dev(svh)
    for rows in (33, 48, 63, 65, 97, 127, 129, 191, 193, 255, 256, 513, 1100):
        x = x_as(synth.activations(2101 + rows, rows, in_dim), dt)
        y = t3.linear(x, t, a, b, t3.Decode(cb, 16))
        sample = sorted({0, 1, 15, 16, 31, 32, rows // 2, rows - 17, rows - 1})
        ref = ob.linear_rows_what(host_f32(x)[sample], what, suh, svh, in_dim, out_dim)
        check(host_f32(y)[sample], ref, dt, ("tile edges", case, rows))
    assert t3.device_error() == 0


@pytest.mark.parametrize("in_dim,out_dim,n,dt", [(4096, 1024, 32, "f16"), (4096, 512, 48, "f32"), (2048, 2048, 64, "bf16")])
def test_sliced_tile_heights(in_dim, out_dim, n, dt):
    """Calls in K slices whose row tiles follow the clusters that are resident at once: one tile, several, ragged last ones; a row's
    bytes do not depend on the height of its tile."""
    trellis, suh, svh = synth.linear(2120 + n, in_dim, out_dim, n, scaled=True)
    what = ob.reconstruct_inner(trellis, in_dim, out_dim, n, t3.MUL1, 16)
    t, a, b = dev(trellis), dev(suh), dev(svh)
    for rows, few in ((33, 33), (100, 33), (200, 100), (256, 200), (300, 257), (512, 300)):
        x = x_as(synth.activations(2121, rows, in_dim), dt)
        y = t3.linear(x, t, a, b)
        sample = sorted({0, 15, 16, few - 1, rows // 2, rows - 1})
        check(host_f32(y)[sample], ob.linear_rows_what(host_f32(x)[sample], what, suh, svh, in_dim, out_dim), dt, ("sliced tiles", in_dim, rows))
        assert torch.equal(y[:few], t3.linear(x[:few].contiguous(), t, a, b))
    assert t3.device_error() == 0


@pytest.mark.parametrize("case", [(384, 128, 48, t3.MUL1, "f16"), (256, 384, 128, t3.MCG, "f32"), (128, 256, 20, t3.MUL1, "bf16")])
def test_routed_tile_edges(case):
    """One expert for each height around the edges; every row goes to one expert at weight 1."""
    hidden, inter, n, cb, dt = case
    heights = [1, 15, 16, 17, 32, 33, 64, 65, 96, 97, 128, 129, 192, 193, 256, 257, 513]
    bank, obank = make_bank(2200 + n, len(heights) + 1, hidden, inter, n)  # the last expert gets no row
    inds = np.repeat(np.arange(len(heights)), heights).astype(np.int32)
    np.random.default_rng(7).shuffle(inds)
    rows = inds.size
    x = x_as(synth.activations(2201 + n, rows, hidden), dt)
    y = t3.moe(x.view(1, rows, hidden), bank, dev(inds).view(1, rows, 1), torch.ones((1, rows, 1), device="cuda"), t3.Decode(cb, 16))
    assert y.dtype == TORCH_DT[dt]
    sample = sorted(int(r) for e in range(len(heights)) for r in np.flatnonzero(inds == e)[[0, -1]])
    ref = ob.moe_rows(obank, host_f32(x)[sample], inds[sample].reshape(-1, 1), np.ones((len(sample), 1), np.float32), cb, 16, 0.0, 0)
    check_moe(host_f32(y).reshape(rows, hidden)[sample], ref, dt, ("routed tile edges", case))
    assert t3.device_error() == 0


def split_bank(seed, E, H, I, n):
    """A bank of 11 experts whole, and dealt over three banks (one of them with a single expert): bank, banks, bank_of, local_of."""
    bank, _ = make_bank(seed, E, H, I, n)
    bank_of = torch.tensor([0, 2, 0, 2, 2, 0, 1, 0, 2, 0, 2])
    local_of = torch.zeros_like(bank_of)
    for b in range(3):
        local_of[bank_of == b] = torch.arange(int((bank_of == b).sum()))
    pick = lambda p, b: t3.Proj(*(v[(bank_of == b).to(v.device)].contiguous() for v in (p.trellis.view(torch.int16), p.suh, p.svh)))
    return bank, [t3.Bank(pick(bank.gate, b), pick(bank.up, b), pick(bank.down, b)) for b in range(3)], bank_of, local_of


@pytest.mark.parametrize("rows,dt", [(33, "f16"), (300, "bf16")])
def test_mixed_banks_give_the_one_bank_bytes(rows, dt):
    H, I, E, topk, n = 384, 256, 11, 4, 48
    bank, banks, bank_of, local_of = split_bank(2300, E, H, I, n)
    inds, scores = synth.routing(2301, rows, E, topk)
    x, di, ds = x_as(synth.activations(2302, rows, H), dt), dev(inds), dev(scores)
    whole = t3.moe(x.view(1, rows, H), bank, di.view(1, rows, topk), ds.view(1, rows, topk))
    mixed = t3.api.moe_mixed(x, banks, bank_of.cuda(), local_of.cuda(), di, ds)
    assert torch.equal(whole.view(rows, H), mixed)
    assert t3.device_error() == 0


@pytest.mark.parametrize("rows", [5, 33, 300])
def test_mixed_map_entries_out_of_range_are_clamped(rows):
    """Banks, numbers in a bank and router ids past either end: the layer of the clamped map."""
    H, I, E, topk, n = 256, 128, 11, 4, 48
    _, banks, bank_of, local_of = split_bank(2310, E, H, I, n)
    bad_bank, bad_local = bank_of.clone(), local_of.clone()
    bad_bank[[0, 3, 6]] = torch.tensor([3, -1, 1 << 40])
    bad_local[[0, 2, 9]] = torch.tensor([1 << 33, -7, 99])
    good_bank = bad_bank.clamp(0, 2)
    size = torch.tensor([b.gate.suh.shape[0] for b in banks])
    good_local = torch.minimum(bad_local.clamp(min=0), size[good_bank] - 1)
    inds, scores = synth.routing(2311, rows, E, topk)
    x, di, ds = x_as(synth.activations(2312, rows, H), "f16"), dev(inds), dev(scores)
    bad_inds = di.clone()
    bad_inds[di == E - 1] = E + 1000
    bad_inds[0, 0] = -1  # as u32: past every id
    di[0, 0] = E - 1
    layer = lambda bank, local, ids: mixed.mixed_rate_moe(x, banks, mixed.RateBuckets([n] * 3, bank, local, []), ids, ds, t3.Decode.mul1)
    assert torch.equal(layer(bad_bank, bad_local, bad_inds), layer(good_bank, good_local, di))
    assert t3.device_error() == 0
