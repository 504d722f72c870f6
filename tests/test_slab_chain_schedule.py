"""How a chain of linears of up to 8 rows numbers its thread blocks: every block takes a place of its own whatever SMs the hardware
gives the blocks, and every share of a linear has one place, apart from those of the linears beside it. (The kernel's arithmetic,
compiled for the host.)"""
import ctypes
import random

import pytest

from chain_index import library

PER_SM = 4


def _claim(sm, sms, n_sm, started, given):
    return library().place(n_sm, sm, sms, started, given)


def _number(place, n_sm, home, per_sm, first_sm):
    v = library().number(n_sm, home, per_sm, first_sm, place)
    return v if v >= 0 else None


@pytest.mark.parametrize("n_sm,sms,uneven", [(148, 148, False), (148, 160, False), (148, 160, True), (20, 32, True)])
def test_places(n_sm, sms, uneven):
    rng = random.Random(n_sm + sms)
    for _ in range(5):
        ids = rng.sample(range(sms), n_sm)
        on = [rng.choice(ids) for _ in range(PER_SM * n_sm)] if uneven else ids * PER_SM
        rng.shuffle(on)
        started, given = (ctypes.c_uint * sms)(), (ctypes.c_uint * PER_SM)()
        assert sorted(_claim(s, sms, n_sm, started, given) for s in on) == list(range(PER_SM * n_sm))


@pytest.mark.parametrize("n_sm", [148, 132, 7])
def test_shares_of_a_step(n_sm):
    rng = random.Random(n_sm)
    home = first_sm = 0
    for _ in range(200):
        left, taken = PER_SM, set()
        while left:
            grid = rng.randint(1, left * n_sm)
            per_sm = -(-grid // n_sm)
            mine = {}
            for place in range(PER_SM * n_sm):
                v = _number(place, n_sm, home, per_sm, first_sm)
                if v is not None and v < grid:
                    assert v not in mine
                    mine[v] = place
            assert sorted(mine) == list(range(grid)) and not taken & set(mine.values())
            taken |= set(mine.values())
            home, first_sm = (home + per_sm) % PER_SM, (first_sm + -(-grid // per_sm)) % n_sm
            left -= per_sm
            if rng.random() < 0.3:
                break
