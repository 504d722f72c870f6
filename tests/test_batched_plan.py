"""How a batched call divides its linears into launches and phases (qf_w4a16_batched_plan): host logic, no GPU. Addresses are made up;
nothing reads them."""
import ctypes
import random

import pytest

from chain_index import library
from quantforge_b200 import _lib
from quantforge_b200._lib import QF_EPI_NONE, QF_EPI_RESIDUAL_ADD, QF_EPI_SILU_MUL

UNIT = 4352
ROOM = 64 << 20  # a workspace that is large enough


class Memory:
    """Addresses of tensors that do not meet."""

    def __init__(self):
        self.at = 1 << 40

    def take(self, nbytes):
        at, self.at = self.at, self.at + (nbytes + 1023) // 1024 * 1024 + 1024
        return at


def blob_bytes(N, K):
    return N // 64 * (K // 128) * UNIT


def linear(M, N, K, x, w, y, residual=0, epilogue=QF_EPI_NONE):
    return {"M": M, "N": N, "K": K, "x": x, "w": w, "y": y, "residual": residual, "epilogue": epilogue}


def plan(calls, workspace_bytes=ROOM):
    """Per entry: launch, phase, the phases it waits for, slots as a range, first place, thread blocks."""
    n = len(calls)
    descs = (_lib.LinearDesc * n)()
    for d, c in zip(descs, calls):
        d.M, d.N, d.K, d.group_size = c["M"], c["N"], c["K"], 128
        d.act_dtype, d.out_dtype, d.zero_mode, d.zero_const = _lib.QF_BF16, _lib.QF_BF16, _lib.QF_ZERO_U4, 8
        d.weight_layout, d.epilogue = _lib.QF_LAYOUT_GEMV_SLAB, c["epilogue"]
    x, w, y, r = ((ctypes.c_void_p * n)(*[c[k] for c in calls]) for k in ("x", "w", "y", "residual"))
    out = (ctypes.c_int32 * (8 * n))()
    assert _lib.load().qf_w4a16_batched_plan(n, descs, x, w, y, r, 1 << 20, workspace_bytes, out) == 0
    keys = ("launch", "phase", "wait0", "wait1", "slot", "slots", "place", "blocks")
    return [dict(zip(keys, out[8 * i:8 * i + 8])) for i in range(n)]


def layers(M, hidden, ffn, n, mem=None):
    """q, k, v | o | gate, up | down, each reading what the one before wrote."""
    mem = mem or Memory()
    act = lambda width: mem.take(M * width * 2)  # noqa: E731
    kv = hidden // 4
    h, q, k, v, o, gate, up = act(hidden), act(hidden), act(kv), act(kv), act(hidden), act(ffn), act(ffn)
    w = lambda N, K: mem.take(blob_bytes(N, K))  # noqa: E731
    calls = []
    for _ in range(n):
        calls += [linear(M, hidden, hidden, h, w(hidden, hidden), q), linear(M, kv, hidden, h, w(kv, hidden), k),
                  linear(M, kv, hidden, h, w(kv, hidden), v), linear(M, hidden, hidden, q, w(hidden, hidden), o),
                  linear(M, ffn, hidden, o, w(ffn, hidden), gate), linear(M, ffn, hidden, o, w(ffn, hidden), up),
                  linear(M, hidden, ffn, gate, w(hidden, ffn), h)]
    return calls


@pytest.mark.parametrize("M", [1, 8, 9, 16, 32])
def test_one_launch(M):
    calls = layers(M, 2048, 5632, 16)
    got = plan(calls)
    assert {p["launch"] for p in got} == {0} and got[-1]["phase"] >= 4 * 16 - 1


@pytest.mark.parametrize("rows", [0, 1, 8, 9])
def test_linears_without_rows(rows):
    """They have no launch, whatever their pointers are, and do not join the others'."""
    for empty in (linear(0, 2048, 2048, 0, 0, 0), linear(0, 2048, 2048, 8, 4, 2), linear(0, 2048, 2048, 16, 32, 48, 64, QF_EPI_RESIDUAL_ADD),
                  linear(0, 4096, 2048, 16, 32, 48, 0, QF_EPI_SILU_MUL)):
        got = plan([empty] * 40)
        assert all(p == dict.fromkeys(p, -1) for p in got)
        if rows:
            calls = layers(rows, 2048, 5632, 4)
            mixed = plan(calls[:14] + [empty] * 3 + calls[14:])
            assert [p["launch"] for p in mixed] == [0] * 14 + [-1] * 3 + [1] * 14


def _meet(a, b):
    return a[0] < b[1] and b[0] < a[1]


def _ranges(c):
    """What a linear reads (activations, residual, weights) and what it writes."""
    cols = c["N"] // 2 if c["epilogue"] == QF_EPI_SILU_MUL else c["N"]
    reads = [(c["x"], c["x"] + c["M"] * c["K"] * 2)]
    if c["epilogue"] == QF_EPI_RESIDUAL_ADD:
        reads.append((c["residual"], c["residual"] + c["M"] * cols * 2))
    return reads, (c["w"], c["w"] + blob_bytes(c["N"], c["K"])), (c["y"], c["y"] + c["M"] * cols * 2)


def _check(calls, got):
    """Every pair of linears of a launch of which one touches what the other writes has an order, and so do those that share slots."""
    launches = {}
    for c, p in zip(calls, got):
        launches.setdefault(p["launch"], []).append((c, p))
    for linears in launches.values():
        if len(linears) == 1:
            continue
        behind = {}  # phase -> all phases that are complete before it begins
        for _, p in sorted(linears, key=lambda cp: cp[1]["phase"]):
            if p["phase"] not in behind:
                waits = [w for w in (p["wait0"], p["wait1"]) if w >= 0]
                assert all(w < p["phase"] for w in waits)
                behind[p["phase"]] = set(waits).union(*[behind[w] for w in waits])
        for j, (cj, pj) in enumerate(linears):
            rj, wj, yj = _ranges(cj)
            for ci, pi in linears[:j]:
                ri, wi, yi = _ranges(ci)
                assert not _meet(yi, wj)  # weights are fetched ahead of all waits
                if any(_meet(yi, r) for r in rj + [yj]) or any(_meet(yj, r) for r in ri + [wi]):
                    assert pi["phase"] in behind[pj["phase"]], (ci, cj)
                side_by_side = pi["phase"] not in behind[pj["phase"]] and pj["phase"] not in behind[pi["phase"]]
                if side_by_side and pi["slots"] and pj["slots"]:
                    assert pi["slot"] + pi["slots"] <= pj["slot"] or pj["slot"] + pj["slots"] <= pi["slot"]
    return launches


@pytest.mark.parametrize("M", [1, 8, 9, 20])
def test_a_result_over_weights_that_an_earlier_linear_reads(M):
    # the last linear of each layer writes over the weights of the layer's k projection, which nothing waits for
    calls = layers(M, 2048, 5632, 4)
    for i in range(6, len(calls), 7):
        calls[i]["y"] = calls[i - 5]["w"]
        if i + 1 < len(calls):
            for c in calls[i + 1:i + 4]:
                c["x"] = calls[i]["y"]
    _check(calls, plan(calls))
    # pairs side by side but for that
    mem, calls = Memory(), []
    x = mem.take(M * 4096)
    for _ in range(8):
        w = mem.take(blob_bytes(2048, 2048))
        calls += [linear(M, 2048, 2048, x, w, mem.take(M * 4096)), linear(M, 2048, 2048, x, mem.take(blob_bytes(2048, 2048)), w + 8192)]
    got = plan(calls)
    assert {p["launch"] for p in got} == {0}
    _check(calls, got)


@pytest.mark.parametrize("seed", range(60))
def test_whatever_touches_has_an_order(seed):
    rng = random.Random(seed)
    M = rng.choice([1, 2, 5, 8, 9, 16, 17, 32])
    span = rng.choice([1 << 18, 1 << 21, 1 << 24, 1 << 28])  # a small one makes nearly everything meet
    mem, calls = Memory(), []
    spot = lambda: (1 << 36) + rng.randrange(span) // 1024 * 1024  # noqa: E731
    spots = [spot() for _ in range(rng.choice([3, 6, 12]))]
    for _ in range(rng.choice([9, 20, 60, 130])):
        N, K = rng.choice([256, 512, 1024, 2048]), rng.choice([256, 512, 1024, 5632])
        w = mem.take(blob_bytes(N, K)) if rng.random() < 0.9 else rng.choice(spots)
        y = rng.choice(spots) if calls == [] or rng.random() < 0.95 else rng.choice(calls)["w"]
        calls.append(linear(M, N, K, rng.choice(spots), w, y, rng.choice(spots), rng.choice([QF_EPI_NONE, QF_EPI_SILU_MUL, QF_EPI_RESIDUAL_ADD])))
    _check(calls, plan(calls))


def test_random_batches_become_chains():
    """What the test above looks at is not all linears that go one by one."""
    chained = 0
    for seed in range(20):
        rng = random.Random(1000 + seed)
        M, calls, mem = rng.choice([1, 8, 9, 32]), [], Memory()
        spots = [mem.take(1 << 20) for _ in range(6)]
        for _ in range(60):
            N, K = rng.choice([256, 1024, 2048]), rng.choice([256, 1024, 2048])
            calls.append(linear(M, N, K, rng.choice(spots), mem.take(blob_bytes(N, K)), rng.choice(spots)))
        launches = _check(calls, plan(calls))
        chained += max(len(v) for v in launches.values()) > 20
    assert chained >= 15


@pytest.mark.parametrize("seed", range(20))
def test_places_of_a_step(seed):
    """Up to 8 rows: no thread block has work of two linears of a step (its four warps count their ends together)."""
    rng = random.Random(seed)
    mem = Memory()
    spots = [mem.take(1 << 20) for _ in range(4)]
    calls = []
    for _ in range(100):
        N, K = rng.choice([128, 256, 1024, 4096]), rng.choice([128, 256, 1024, 2048])
        calls.append(linear(4, N, K, rng.choice(spots), mem.take(blob_bytes(N, K)), rng.choice(spots)))
    got = plan(calls)
    steps = {}
    for p in got:
        steps.setdefault((p["launch"], p["wait0"], p["wait1"]), []).append(p)
    assert max(len(s) for s in steps.values()) > 1
    for s in steps.values():
        taken = set()
        for p in s:
            per_sm, first_sm, home = -(-p["blocks"] // 148), p["place"] // 4, p["place"] % 4
            mine = {at for at in range(4 * 148) if 0 <= library().number(148, home, per_sm, first_sm, at) < p["blocks"]}
            assert len(mine) == p["blocks"] and not taken & mine
            taken |= mine


def _row(M, H, F, n):
    """n linears H -> F -> H -> ..., each reading the one before."""
    mem = Memory()
    a, b = mem.take(M * H * 2), mem.take(M * F * 2)
    return [linear(M, *((F, H) if i % 2 == 0 else (H, F)), (a, b)[i % 2], mem.take(blob_bytes(H, F)), (b, a)[i % 2]) for i in range(n)]


def _beside(M, H, F, n):
    mem = Memory()
    x = mem.take(M * H * 2)
    return [linear(M, F, H, x, mem.take(blob_bytes(F, H)), mem.take(M * F * 2)) for _ in range(n)]


@pytest.mark.parametrize("M", [9, 16])
def test_small_linears_that_wait_for_one_another_are_no_chain(M):
    for calls in (_row(M, 512, 512, 2), _row(M, 512, 512, 8), _row(M, 1024, 2816, 2), _row(M, 1024, 2816, 4), _row(M, 2048, 2048, 3),
                  _row(M, 768, 768, 6), _beside(M, 256, 256, 2), _beside(M, 1024, 14336, 2)):
        assert [p["launch"] for p in plan(calls)] == list(range(len(calls)))


@pytest.mark.parametrize("M", [9, 16, 17, 32])
def test_what_gains_is_a_chain(M):
    for calls in (_row(M, 4096, 14336, 2), _row(M, 2048, 5632, 4), _row(M, 256, 18944, 2), _beside(M, 512, 512, 4), _beside(M, 4096, 4096, 2),
                  layers(M, 512, 1024, 1), layers(M, 2048, 5632, 1), layers(M, 8192, 28672, 1)):
        assert {p["launch"] for p in plan(calls)} == {0}
    for calls in (_row(M, 512, 512, 2), _row(M, 512, 512, 8), _beside(M, 256, 256, 2)):
        assert {p["launch"] for p in plan(calls)} == set(range(len(calls)))
    assert {p["launch"] for p in plan(_row(M, 1024, 2816, 8))} == (set(range(8)) if M <= 16 else {0})


@pytest.mark.parametrize("fuse", [True, False])
def test_stacks_that_lay_out_for_chains_get_them(fuse):
    """A stack of 9 to 32 rows chooses its layout by the size of its linears, before there is a batch."""
    from quantforge_b200.stack import runs_as_chain
    rng = random.Random(fuse)
    seen = 0
    while seen < 150:
        H, KV, F = 128 * rng.randint(2, 80), rng.choice([128, 512, 1024]), 128 * rng.randint(2, 224)
        M, n = rng.randint(9, 32), rng.choice([1, 2, 6])
        if not runs_as_chain({"hidden": H, "kv": KV, "ffn": F}, M, fuse):
            continue
        seen += 1
        mem, calls = Memory(), []
        act = {k: mem.take(M * w * 2) for k, w in dict(h=H, attn=H, q=H, k=KV, v=KV, qkv=H + 2 * KV, o=H, gate=F, up=2 * F, act=F, d=H).items()}
        h = act["h"]
        for _ in range(n):
            if fuse:
                names = [(h, "qkv", H + 2 * KV, H, 0), (act["attn"], "o", H, H, h), (act["o"], "act", 2 * F, H, 0), (act["act"], "d", H, F, act["o"])]
            else:
                names = [(h, "q", H, H, 0), (h, "k", KV, H, 0), (h, "v", KV, H, 0), (act["q"], "o", H, H, 0), (act["o"], "gate", F, H, 0),
                         (act["o"], "up", F, H, 0), (act["gate"], "d", H, F, 0)]
            for x, y, N, K, r in names:
                epi = QF_EPI_RESIDUAL_ADD if r else QF_EPI_SILU_MUL if y == "act" else QF_EPI_NONE
                calls.append(linear(M, N, K, x, mem.take(blob_bytes(N, K)), act[y], r, epi))
            h = act["d"]
        assert {p["launch"] for p in plan(calls)} == {0}, (M, H, KV, F, n)


@pytest.mark.parametrize("M", [1, 8, 9, 32])
def test_scratch_for_single_linears_only(M):
    """With what the largest linear alone needs, and anything up to what a chain needs, linears go one by one."""
    lib = _lib.load()
    calls = layers(M, 512, 1024, 2)
    descs = (_lib.LinearDesc * len(calls))()
    for d, c in zip(descs, calls):
        d.M, d.N, d.K, d.group_size, d.act_dtype, d.out_dtype = M, c["N"], c["K"], 128, _lib.QF_BF16, _lib.QF_BF16
        d.zero_mode, d.weight_layout = _lib.QF_ZERO_U4, _lib.QF_LAYOUT_GEMV_SLAB
    alone = max(lib.qf_w4a16_workspace_bytes(ctypes.byref(d)) for d in descs)
    chain = lib.qf_w4a16_batched_workspace_bytes(len(calls), descs)
    assert alone < chain
    for room in (alone, chain - 1):
        assert [p["launch"] for p in plan(calls, room)] == list(range(len(calls)))
    assert {p["launch"] for p in plan(calls, chain)} == {0}


@pytest.mark.parametrize("M", [1, 2, 4, 8])
def test_linears_of_which_each_waits_for_the_one_before(M):
    """Up to 8 rows a launch that begins beside its predecessor is shorter than a step of a chain, however many there are."""
    for H, F, n in ((512, 1408, 16), (1024, 2816, 16), (2048, 5632, 16), (4096, 14336, 32), (1024, 1024, 100)):
        assert [p["launch"] for p in plan(_row(M, H, F, n))] == list(range(n))
    calls = layers(M, 2048, 5632, 8)
    for c, before in zip(calls[1:], calls):
        c["K"], c["x"] = before["N"], before["y"]
    assert [p["launch"] for p in plan(calls)] == list(range(56))
    # what stands side by side shares a step
    assert {p["launch"] for p in plan(layers(M, 2048, 5632, 8))} == {0}


@pytest.mark.parametrize("hidden,ffn,batch,fuse,chain", [
    (2048, 5632, 9, True, True), (2048, 5632, 16, True, True), (1024, 2816, 9, True, False), (2048, 5632, 17, True, False),
    (1792, 18944, 20, True, False), (6912, 3584, 24, True, False), (4096, 14336, 24, True, True), (4096, 14336, 25, True, False),
    (5120, 13824, 32, True, False), (7680, 25856, 28, True, False), (1536, 4096, 32, False, False), (2048, 5632, 32, False, True),
    (8192, 28672, 32, False, True), (4096, 14336, 33, False, False), (1024, 2816, 8, True, True)])
def test_stacks_of_more_than_8_rows_that_run_as_chains(hidden, ffn, batch, fuse, chain):
    """Where it is the faster way by the times beside the rule; up to 8 rows the batched call decides."""
    from quantforge_b200.stack import runs_as_chain
    cfg = {"hidden": hidden, "kv": 1024 if hidden >= 4096 else 512, "ffn": ffn}
    assert runs_as_chain(cfg, batch, fuse) == chain
    assert not runs_as_chain(cfg, batch, fuse, world=2)
    assert not runs_as_chain(dict(cfg, kv=64), batch, fuse)
