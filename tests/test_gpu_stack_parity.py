"""DecodeLinearStack.check_parity looks at what a step runs: its chains as well as the linears by themselves."""
import pytest
import torch

from oracle import qf_oracle as O
from quantforge_b200.stack import DecodeLinearStack

pytestmark = pytest.mark.gpu


def _oracle(x, qweight_rows, scales, zeros, group):
    return O.w4a16_linear(x, qweight_rows, scales, zeros, group, "bf16", O.F32, accumulate="f64")


def _stack(M, fuse=True, cfg=None):
    cfg = cfg or {"hidden": 2048, "kv": 512, "ffn": 5632, "layers": 4}
    st = DecodeLinearStack(cfg, M, torch.bfloat16, torch.device("cuda", 0), seed=M, fuse=fuse, epilogues=fuse)
    for name in ("h_in", "attn"):
        st.buf[name].mul_(0.02)
    return st


@pytest.mark.parametrize("M,fuse", [(1, True), (8, False), (9, True), (16, False), (32, False)])
def test_a_step_is_checked(M, fuse):
    st = _stack(M, fuse)
    assert st.chain and st.launches_per_step() == 1
    got = st.check_parity(_oracle, O.silu_mul)
    assert got["max_rel_err"] < 1e-2 and got["ranks_bit_identical"] and got["step_bits_identical"] is True
    # a step that leaves something else behind is noticed
    batch, out = st._chained()

    class Wrong:
        @staticmethod
        def run():
            batch.run()
            out[-1, -1] += 1

    st._chained = lambda: (Wrong, out)
    assert st.check_parity(_oracle, O.silu_mul)["step_bits_identical"] is False


@pytest.mark.parametrize("M", [9, 16])
def test_linears_of_a_chain_are_compared_with_the_oracle(M):
    """Above 8 rows a chain has its own order of sums: the four linears of a layer are compared by themselves and in a batch."""
    assert _stack(M).check_parity(_oracle, O.silu_mul)["cases"] == 8


def test_stacks_that_call_their_linears():
    st = _stack(64)
    got = st.check_parity(_oracle, O.silu_mul)
    assert got["max_rel_err"] < 1e-2 and got["cases"] == 4 and got["step_bits_identical"] is None
