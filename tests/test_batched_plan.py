"""How a batched call divides its linears into launches and phases (qf_w4a16_batched_plan): host logic, no GPU. Addresses are made up;
nothing reads them."""
import ctypes

import pytest

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
