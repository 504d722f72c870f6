"""How a chain of linears of up to 8 rows numbers its thread blocks, restated: every block takes a place of its own whatever SMs the
hardware gives the blocks, and every share of a linear has one place, apart from those of the linears beside it."""
import random

import pytest

PER_SM = 4


def _claim(sm, sms, n_sm, seen, given):
    i = min(seen.get(sm, 0), PER_SM - 1)
    seen[sm] = seen.get(sm, 0) + 1
    if sms == n_sm:
        return sm * PER_SM + i
    for _ in range(PER_SM):
        n, given[i] = given[i], given[i] + 1
        if n < n_sm:
            return n * PER_SM + i
        i = (i + 1) % PER_SM
    raise AssertionError("no place left")


def _number(place, n_sm, home, per_sm, first_sm):
    i = (place - home) % PER_SM
    sm = (place // PER_SM - first_sm) % n_sm
    return sm * per_sm + i if i < per_sm else None


@pytest.mark.parametrize("n_sm,sms,uneven", [(148, 148, False), (148, 160, False), (148, 160, True), (20, 32, True)])
def test_places(n_sm, sms, uneven):
    rng = random.Random(n_sm + sms)
    for _ in range(5):
        ids = rng.sample(range(sms), n_sm)
        on = [rng.choice(ids) for _ in range(PER_SM * n_sm)] if uneven else ids * PER_SM
        rng.shuffle(on)
        seen, given = {}, [0] * PER_SM
        assert sorted(_claim(s, sms, n_sm, seen, given) for s in on) == list(range(PER_SM * n_sm))


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
