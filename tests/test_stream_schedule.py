"""How the streaming tcgen05 kernel divides work: every unit and every piece has one stream, and the members of a row block are the
streams that have chunks of it. (The kernel's arithmetic, compiled for the host.)"""
import random

import pytest

from chain_index import library


def _range(id_, q, r):
    return library().range_first(id_, q, r), library().range_units(id_, q, r)


def _stream_of(u, q, r):
    return library().of(u, q, r)


@pytest.mark.parametrize("blocks,chunks,streams", [(1, 1, 2), (1, 4, 4), (32, 32, 296), (448, 64, 296), (3, 224, 296), (5, 7, 34), (149, 3, 296)])
def test_ranges(blocks, chunks, streams):
    units = blocks * chunks
    q, r = units // streams, units % streams
    members, slots = {}, set()
    seen = 0
    for s in range(streams):
        u, n = _range(s, q, r)
        assert u == seen
        seen += n
        while n:
            b, c = u // chunks, u % chunks
            length = min(chunks - c, n)
            assert _stream_of(u, q, r) == s and _stream_of(u + length - 1, q, r) == s
            members.setdefault(b, []).append((s, c))
            u, n = u + length, n - length
    assert seen == units
    for b, who in members.items():
        first, last = _stream_of(b * chunks, q, r), _stream_of(b * chunks + chunks - 1, q, r)
        assert [s for s, _ in who] == list(range(first, last + 1))
        if len(who) > 1:
            for s, c in who:
                slot = streams + s if c == 0 else s  # the first member's slot, the others'
                assert slot not in slots and slot < 2 * streams
                slots.add(slot)


@pytest.mark.parametrize("flip", [0, 1])
@pytest.mark.parametrize("pieces,streams", [(1, 2), (5, 10), (296, 296), (297, 296), (496, 296), (1000, 148), (592, 296), (240, 72)])
def test_pieces_are_dealt_once(pieces, streams, flip):
    home = 296 - streams if streams < 296 else 0  # a late phase goes to the streams from `home` on
    for other in list(range(home)) + [home + streams]:
        assert library().piece(pieces, streams, home, flip, other, 0) >= pieces
    dealt, working = [], 0
    for s in range(streams):
        k = 0
        while True:
            j = library().piece(pieces, streams, home, flip, home + s, k)
            if j >= pieces:
                break
            dealt.append(j)
            k += 1
        working += k > 0
    assert sorted(dealt) == list(range(pieces)) and working == min(pieces, streams)


def test_a_walk_that_ends_early_misses_nothing():
    # a stream stops at its first round without a piece: no later round has one for it
    rng = random.Random(1)
    for _ in range(200):
        streams, pieces = rng.randint(1, 40), rng.randint(1, 200)
        for s in range(streams):
            rounds = [k for k in range(pieces // streams + 2) if library().piece(pieces, streams, 0, 0, s, k) < pieces]
            assert rounds == list(range(len(rounds)))
