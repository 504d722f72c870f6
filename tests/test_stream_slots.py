"""Slots of partial sums in chains of more than 8 rows: a linear's may be written before the step before it is complete, so no other
linear that can still be at work then may have the same ones. Host logic, no GPU."""
import ctypes
import random

import pytest

from quantforge_b200 import _lib
from test_batched_plan import Memory, blob_bytes, layers, linear, plan

LARGE, SMALL = 64 << 20, 65536 + 592 * 32 * 128 * 8  # room for more slots at 9 to 32 rows, and at 32 rows for the fewest


def _check(calls, got):
    """Returns how many pairs of linears of one launch share slots."""
    behind, first = {}, {}
    for p in sorted(got, key=lambda p: (p["launch"], p["phase"])):
        key = (p["launch"], p["phase"])
        if p["phase"] < 0 or key in behind:
            continue
        of = lambda waits: set().union(*[{w} | behind[(p["launch"], w)] for w in waits if w >= 0])  # noqa: E731
        behind[key] = of((p["wait0"], p["wait1"]))  # phases that are complete when this one is
        first[key] = of((p["place"], p["wait1"]))   # when it writes partial sums
        assert p["place"] < p["phase"] and first[key] <= behind[key]
    shared = 0
    for j, pj in enumerate(got):
        for pi in got[:j] + got[j + 1:]:
            if pi["launch"] != pj["launch"] or pi["phase"] < 0 or pi["phase"] > pj["phase"] or not (pi["slots"] and pj["slots"]):
                continue
            if pi["slot"] < pj["slot"] + pj["slots"] and pj["slot"] < pi["slot"] + pi["slots"]:
                assert pi["phase"] in first[(pj["launch"], pj["phase"])]
                shared += 1
    return shared


@pytest.mark.parametrize("room", [LARGE, SMALL])
@pytest.mark.parametrize("M", [9, 16, 24, 32])
def test_layers(M, room):
    shared = 0
    for hidden, ffn, n in ((4096, 14336, 8), (1024, 2816, 12), (2048, 5632, 6), (8192, 28672, 3), (4096, 2048, 5)):
        calls = layers(M, hidden, ffn, n)
        shared += _check(calls, plan(calls, room))
    assert shared > 0


@pytest.mark.parametrize("seed", range(30))
def test_random_batches(seed):
    rng = random.Random(seed)
    mem, M = Memory(), rng.choice([9, 16, 17, 32])
    sizes = [rng.choice([256, 512, 1024, 2048, 4096]) for _ in range(3)]
    bufs = {n: [mem.take(M * n * 2) for _ in range(2)] for n in sizes}
    calls = []
    for _ in range(rng.randint(4, 40)):
        K, N = rng.choice(sizes), rng.choice(sizes)
        x, y = rng.choice(bufs[K]), rng.choice(bufs[N])
        if x != y:
            calls.append(linear(M, N, K, x, mem.take(blob_bytes(N, K)), y))
    _check(calls, plan(calls, rng.choice([LARGE, SMALL])))


@pytest.mark.parametrize("M", [9, 16, 32])
def test_scratch_that_a_batch_asks_for(M):
    calls = layers(M, 4096, 14336, 2)
    descs = (_lib.LinearDesc * len(calls))()
    for d, c in zip(descs, calls):
        d.M, d.N, d.K, d.group_size = c["M"], c["N"], c["K"], 128
        d.act_dtype, d.out_dtype, d.zero_mode, d.zero_const = _lib.QF_BF16, _lib.QF_BF16, _lib.QF_ZERO_U4, 8
        d.weight_layout = _lib.QF_LAYOUT_GEMV_SLAB
    asked = _lib.load().qf_w4a16_batched_workspace_bytes(len(calls), descs)
    assert asked == 65536 + 888 * ((M + 1) // 2 * 2) * 128 * 8
    # with less, down to 592 slots, it still is one launch
    for room in (asked, asked - 1, 65536 + 592 * ((M + 1) // 2 * 2) * 128 * 8):
        got = plan(calls, room)
        assert {p["launch"] for p in got} == {0}
        assert max(p["slot"] + p["slots"] for p in got) <= (888 if room == asked else 592)
