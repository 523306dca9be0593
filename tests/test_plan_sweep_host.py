"""Launch arithmetic of the decode-row kernels over a grid of shapes, rates and row counts, on the host: what a launch
needs to be a valid one (cluster, shared memory, grid) checked from the plan alone. No GPU is touched.

The reference plans its launches from the shape as well (src/hip/plan.zig, src/core/partition.zig:1-80); the splits here
are this library's own, so the properties are the ones any split must have.
"""
import ctypes
import itertools
import os
import re
import subprocess

import pytest

import turboexl3_b200 as t3
from turboexl3_b200.api import lib

DIMS = [128, 256, 384, 512, 1536, 2048, 4096, 6144, 7168, 8192, 16384, 24576, 32768]
RATES = [16, 32, 48, 64, 80, 96, 112, 128, 20, 36, 100]   # halfwords a tile: the eight with kernels of their own, three without
ROWS = [1, 2, 7, 8, 9, 12, 16, 17, 31, 32]
SMEM_LIMIT = 200 * 1024   # what the library admits a CTA (the hardware's 227 KB less a reserve)
CLUSTER_MAX = 16          # the non-portable cluster size the kernels opt into


def _row_cap(rows):
    return 8 if rows <= 8 else (16 if rows <= 16 else 32)


@pytest.mark.parametrize("codebook", [t3.MUL1, t3.MCG])
def test_dense_plans_are_launchable(codebook):
    dec = t3.Decode(codebook)
    name = "mul1" if codebook == t3.MUL1 else "mcg"
    seen_global = seen_cluster = 0
    for (i, o), n, rows in itertools.product(itertools.product(DIMS, DIMS), RATES, ROWS):
        plan = t3.plan_linear(rows, i, o, n, dec)
        gemv = plan[-1]
        own = n if n % 16 == 0 else 0
        assert gemv["symbol"] == f"t3_dense_gemv_{name}_n{own}_r{_row_cap(rows)}", (i, o, n, rows)
        assert gemv["block"] == 544 and gemv["group"] == "dense"
        gx, gy, gz = gemv["grid"]
        assert gy == o // 128 and gz == 1 and 1 <= gx <= i // 128, (i, o, n, rows, gemv)  # a K slice holds a block at least
        assert 0 < gemv["shared"] <= SMEM_LIMIT, (i, o, n, rows, gemv)
        assert 1 <= gemv["cluster"] <= CLUSTER_MAX and gx % gemv["cluster"] == 0
        ws = lib().t3_linear_workspace_bytes(rows, i, o, n)
        if gemv["cluster"] == 1 and gx > 1:
            # slices that meet in global memory: the call asked for a workspace that holds every slice's partial sums
            assert ws >= gy * gx * rows * 128 * 4 + gy * 4, (i, o, n, rows, ws)
            seen_global += 1
        else:
            assert gx == gemv["cluster"]  # one cluster a 128-output block
            seen_cluster += 1
        if len(plan) == 2:
            prep = plan[0]
            assert prep["symbol"] == "t3_dense_prep" and prep["block"] == 128 and prep["cluster"] == 1
            assert prep["grid"] == ((rows * (i // 128) + 3) // 4, 1, 1)
            assert ws >= rows * i * 2  # the prepared rows (f16)
        else:
            assert len(plan) == 1
    assert seen_global > 0 and seen_cluster > 0
    for i, o in [(2048, 2048), (2048, 6144), (6144, 2048), (1536, 24576), (512, 32768)]:
        assert lib().t3_linear_workspace_bytes(1, i, o, 64) == 0  # one row of a trunk-sized linear runs without a workspace


def _large(i, o, n):
    return i * o * n >= 24 * 1024 * 1024 * 128  # linears of 24 MB of codes and up: a rule of their own


ONE_A_SM = [0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7]     # clusters of each size resident at once, a CTA a multiprocessor
TWO_A_SM = {1: 296, 2: 148, 3: 88, 4: 71, 5: 50, 6: 45, 7: 37, 8: 33, 16: 14}  # and two, with those of three and five taken shorter


def _slice_cost(i, o, n, s):
    """Three times the time of a row plus that of 32 rows (10 ns) of `s` K slices, by the times a 128-input block takes; None where a CTA
    cannot hold the prepared rows of 32 rows (200 KB, two CTAs a multiprocessor up to 113 KB; 128 bytes are kept for alignment)."""
    nb, blocks, up = i // 128, o // 128, lambda v: (v + 127) // 128 * 128
    longest = -(-nb // s)
    stages = (longest + 1) // 2
    rows, tile = up(32 * (longest * 128 + 16) * 2), 32 * 136 * 4
    size = lambda least: 640 + rows + (0 if longest >= 4 else tile) + up(s * -(-32 // s) * 136 * 4) + 256 * n * min(stages, least)
    if size(1) > SMEM_LIMIT - 128:
        return None
    single = blocks <= ONE_A_SM[s]

    def rounds(at_once, block, last, fixed):
        full, rest = divmod(blocks, at_once)
        return full * (longest * block + fixed) + (longest * (last if rest <= ONE_A_SM[s] else block) + fixed if rest else 0)

    row = rounds(ONE_A_SM[s], 58, 58, 300 + 10 * s) if single else rounds(TWO_A_SM[s], 116, 58, 300 + 10 * s)
    if single or size(3) > 113 * 1024 - 128:
        many = rounds(ONE_A_SM[s], 80, 80, 640 + 10 * s)
    else:
        many = rounds(TWO_A_SM[s], 260, 80, 640 + 10 * s)
    return 3 * row + (many * 7 // 5 if size(2) > SMEM_LIMIT - 128 else many)


def test_a_shape_has_one_slice_count_and_it_is_no_dearer_than_a_power_of_two():
    """A row's bytes follow from how K is cut, so a dense linear under 24 MB of codes is cut the same way at every row count; and the
    cut is never one that a power of two up to eight beats by the rule's own times (12288 -> 4608 once ran one row uncut: 64 us for 24)."""
    outs = list(range(512, 16385, 512)) + [640, 896, 1408, 9728, 19456, 24576]
    for i, o, n in itertools.product(list(range(512, 16385, 512)) + [640, 1920, 13952], outs, (16, 32, 48, 64, 80, 96, 128)):
        if _large(i, o, n):
            continue
        counts = {t3.plan_linear(rows, i, o, n)[-1]["grid"][0] for rows in (1, 4, 8, 9, 16, 17, 32)}
        assert len(counts) == 1, (i, o, n, counts)
        own = _slice_cost(i, o, n, counts.pop())
        for s in (1, 2, 4, 8):
            if s <= i // 128 and (other := _slice_cost(i, o, n, s)) is not None:
                assert own is not None and own <= other, (i, o, n, s)


def test_a_smaller_device_holds_its_share_of_the_clusters(tmp_path):
    """The clusters resident at once are written down for 148 multiprocessors: on a device (or a share of one) with fewer, a launch that
    counts on a multiprocessor a CTA has no more clusters than their share."""
    so = str(tmp_path / "split.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", os.path.join(os.path.dirname(__file__), "host_emul", "split_emul.cpp"), "-o", so],
                   check=True)
    split = ctypes.CDLL(so).split_emul
    for sms, nb, blocks in itertools.product((148, 132, 74, 18), (4, 16, 48, 128), range(1, 200)):
        s, alone = split(sms, nb, blocks) % 100, split(sms, nb, blocks) >= 100
        assert 1 <= s <= min(nb, 16)
        assert not alone or blocks <= ONE_A_SM[s] * sms // 148, (sms, nb, blocks, s)
    assert split(148, 16, 16) == 106 and split(74, 16, 16) != 106  # 2048 -> 2048: sixteen clusters of six take 96 multiprocessors


def test_launches_that_do_not_overlap_leave_room_for_another_streams():
    """A decode-row launch that starts beside its predecessor keeps its multiprocessors to itself (more than half their shared memory, by
    one CTA); with no_overlap two CTAs fit one again (228 KB, 1 KB a CTA reserved), in the same cut of K."""
    shapes = [(2048, 2048), (2048, 6144), (6144, 2048), (3072, 3072), (7168, 1536)]
    plans = lambda: [t3.plan_linear(1, i, o, n)[-1] for i, o in shapes for n in (16, 64, 128)] + [t3.plan_moe(1, 10, 512, 2048, 512, 48)[0]]
    half = 228 * 1024 // 2 - 1024
    apart = plans()
    try:
        t3.configure(no_overlap=True)
        beside = plans()
    finally:
        t3.configure()
    assert all(p["shared"] > half for p in apart) and all(p["shared"] <= half for p in beside)
    assert [p["grid"] for p in apart] == [p["grid"] for p in beside]


def test_a_large_linear_keeps_its_multiprocessors_where_all_its_clusters_fit_so():
    """Linears of 24 MB of codes and up: CTAs that all find a multiprocessor each are not placed two to one beside empty ones (5760 -> 17920 K4 at
    one row once took 45.7 us for 30.7, by a ring that let two of them fit)."""
    asked = 0
    for i, o, n in itertools.product(range(2048, 16385, 640), range(2048, 24577, 640), (32, 48, 64, 80, 96, 128)):
        if not _large(i, o, n) or i * o > 16384 * 7168:
            continue
        for rows in (1, 8, 16):
            p = t3.plan_linear(rows, i, o, n)[-1]
            fits = p["grid"][1] <= ONE_A_SM[p["cluster"]] if p["cluster"] > 1 else p["grid"][0] * p["grid"][1] <= 148
            if fits:
                asked += 1
                assert p["shared"] > 113 * 1024, (rows, i, o, n, p)
    assert asked > 1000


def test_a_gate_up_launch_keeps_its_multiprocessors_only_where_all_its_clusters_fit_so():
    """CTAs that ask for more than half a multiprocessor's shared memory are one to a multiprocessor: no launch asks for that whose clusters
    do not all fit the device so (the ones left over would wait for a whole second round)."""
    asked = 0
    for rows, inter in itertools.product(range(1, 33), (128, 256, 384, 512, 1024)):
        for topk in (1, 2, 6, 8, 10, 16):
            gu = t3.plan_moe(rows, topk, 64, 2048, inter, 16)[0]  # (a ring small enough to leave room for a second CTA)
            if gu["shared"] > 113 * 1024:
                asked += 1
                assert rows * topk * (inter // 128) <= ONE_A_SM[gu["cluster"]], (rows, inter, topk, gu)
    assert asked > 0


def test_routed_plans_are_launchable():
    geoms = [(8, 128, 128), (10, 512, 2048), (64, 2048, 512), (128, 2048, 768), (256, 7168, 2048), (32, 4096, 1536), (16, 1024, 4096)]
    for (experts, hidden, inter), n, rows, topk in itertools.product(geoms, [16, 48, 64, 128, 36], [1, 3, 8, 16, 32], [1, 2, 8, 10]):
        if topk > experts:
            continue
        chain = t3.plan_moe(rows, topk, experts, hidden, inter, n)
        slots = rows * topk
        assert len(chain) == (2 if topk == 1 else 3), (experts, hidden, inter, n, rows, topk)
        gu, down = chain[0], chain[1]
        assert re.fullmatch(r"t3_dec_gate_up_mul1_n\d+_r(8|16)", gu["symbol"]) and re.fullmatch(r"t3_dec_down_mul1_n\d+_r(8|16)", down["symbol"])
        for l, blocks, k_blocks in ((gu, inter // 128, hidden // 128), (down, hidden // 128, inter // 128)):
            gx, gy, gz = l["grid"]
            assert (gy, gz) == (blocks, slots) and l["group"] == "decode" and l["block"] == 544
            assert gx == l["cluster"] and 1 <= l["cluster"] <= CLUSTER_MAX
            assert 0 < l["shared"] <= SMEM_LIMIT, (experts, hidden, inter, n, rows, topk, l)
        assert gu["cluster"] % 2 == 0 and gu["cluster"] // 2 <= hidden // 128  # gate and up side by side, a slice a block at least
        assert down["cluster"] <= inter // 128
        if topk > 1:
            merge = chain[2]
            assert merge["symbol"] == "t3_dec_merge" and merge["cluster"] == 1 and merge["shared"] < 48 * 1024


def test_plan_refusals_are_the_calls():
    for rows, i, o, n in [(0, 2048, 2048, 64), (1, 2048, 2040, 64), (1, 100, 2048, 64), (1, 2048, 2048, 14), (1, 2048, 2048, 130)]:
        with pytest.raises(t3.Exl3Error):
            t3.plan_linear(rows, i, o, n)
    with pytest.raises(t3.Exl3Error, match="BadExl3Shape"):
        t3.plan_moe(4, 33, 64, 512, 2048, 48)  # more slots a row than the merge takes (32)
    with pytest.raises(t3.Exl3Error, match="BadExl3Shape"):
        t3.plan_moe(4, 2, 10, 500, 2048, 48)  # hidden is not whole 128-blocks
    with pytest.raises(t3.Exl3Error, match="Exl3EngineNotImplemented"):
        t3.plan_moe(33, 2, 10, 512, 2048, 48)  # prefill rows: the plan covers the decode-row kernels


def test_prefill_workspace_holds_the_prepared_rows_and_a_bounded_slab():
    """Past 32 rows the workspace is the prepared rows (f16) plus, for calls of up to 512 rows that are cut into K slices, a slab
    of partial sums: a whole number of 64 KB tiles (128 x 128 f32 a slice a row tile), never more than two CTAs a
    multiprocessor's worth; nothing past 512 rows; and the same answer for every rate (the slab follows in and out alone)."""
    L = lib()
    up256 = lambda v: (v + 255) & ~255
    for i, o in itertools.product(DIMS, DIMS):
        for rows in (33, 128, 129, 256, 257, 512, 513, 4096):
            ws = L.t3_linear_workspace_bytes(rows, i, o, 64)
            xp = up256(rows * i * 2)
            assert ws >= xp, (i, o, rows)
            assert ws == L.t3_linear_workspace_bytes(rows, i, o, 36)
            if rows > 512:
                assert ws == xp, (i, o, rows)
                continue
            extra = ws - xp
            if extra:
                mtiles, ncol = (rows + 127) // 128, o // 128
                counters = up256(mtiles * ncol * 4)
                slab = extra - counters
                assert slab > 0 and slab % (mtiles * ncol * 65536) == 0, (i, o, rows, extra)
                slices = slab // (mtiles * ncol * 65536)
                assert 2 <= slices <= 8 and slices * 4 <= i // 64, (i, o, rows, slices)
                assert mtiles * ncol * slices <= 2 * 148, (i, o, rows, slices)  # two CTAs a multiprocessor at most (148 of them)
        # within an arm the slice count does not depend on the rows
        for lo, hi in ((33, 256), (257, 512)):
            per_tile = set()
            for rows in (lo, (lo + hi) // 2, hi):
                extra = L.t3_linear_workspace_bytes(rows, i, o, 64) - up256(rows * i * 2)
                mtiles, ncol = (rows + 127) // 128, o // 128
                per_tile.add((extra - up256(mtiles * ncol * 4)) // (mtiles * ncol * 65536) if extra else 1)
            assert len(per_tile) == 1, (i, o, lo, hi, per_tile)
