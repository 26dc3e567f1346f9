"""The planner that cuts decode items into shares of about equal length (host side only)."""
import random

import numpy as np

from llm_steadyinfer_b200.csrc import ops
from llm_steadyinfer_b200.csrc.ops import split_work


def _shares(work):
    live = work[work[:, 0] >= 0]
    return {int(i): int(live[live[:, 0] == i][0, 2]) for i in set(live[:, 0].tolist())}, live


def test_every_share_is_listed_once_and_slots_do_not_overlap():
    rng = random.Random(3)
    for _ in range(300):
        n = rng.randint(1, 70)
        tiles = [rng.choice([0, 1, 2, 3, 5, 17, 64, 128, 500]) for _ in range(n)]
        budget = rng.choice([1, 5, 37, 148])
        entries = budget + n
        work = split_work(tiles, budget, entries, 32, rng.choice([1, 2, 4]), second_round=rng.random() < 0.5)
        assert work.shape == (entries, 4) and work.dtype == np.int32
        sp, live = _shares(work)
        assert set(sp) == {i for i, t in enumerate(tiles) if t > 0}
        taken = set()
        for i, k in sp.items():
            mine = live[live[:, 0] == i]
            assert sorted(mine[:, 1].tolist()) == list(range(k)) and (mine[:, 2] == k).all()
            first = int(mine[0, 3])
            assert (mine[:, 3] == first).all() and 1 <= k <= 32
            slots = set(range(first, first + k))
            assert not slots & taken and max(slots) < entries
            taken |= slots
        rest = work[len(live):]
        assert (rest[:, 0] == -1).all(), "live entries come first"


def test_equal_items_get_equal_shares_within_the_budget():
    sp, live = _shares(split_work([128] * 8, 37, 45, 32, 2))
    assert set(sp.values()) == {4} and len(live) == 32          # 5 each would need 40 > 37
    sp, _ = _shares(split_work([128] * 5, 37, 42, 32, 2))
    assert set(sp.values()) == {7}


def test_a_long_item_among_short_ones_is_cut_most():
    sp, live = _shares(split_work([128] + [8] * 7, 37, 45, 32, 2))
    assert sp[0] >= 20 and all(sp[i] <= 2 for i in range(1, 8)) and len(live) <= 37
    # more items than shares that run at once: the long one is still cut, to the mean load of a share
    sp, live = _shares(split_work([128] + [4] * 63, 37, 37 + 64, 32, 2))
    assert sp[0] >= 10 and all(sp[i] == 1 for i in range(1, 64))


def test_no_share_is_shorter_than_the_least_and_no_item_has_more_than_the_most():
    sp, _ = _shares(split_work([3, 1, 1000], 200, 203, 32, 2))
    assert sp[0] <= 2 and sp[1] == 1 and sp[2] == 32


def test_more_items_than_slots():
    # many equal sequences stay whole: HBM is busy either way, and every share has its cost
    sp, live = _shares(split_work([128] * 64, 37, 37 + 256, 32, 2))
    assert set(sp.values()) == {1}
    sp, _ = _shares(split_work([16] * 100, 37, 37 + 400, 32, 2))
    assert set(sp.values()) == {1}
    # a few more sequences than slots: whole, the last three blocks of each head would run alone for as long
    # as all the others took; cut, the chains on the slots are about equal
    sp, live = _shares(split_work([128] * 40, 37, 37 + 160, 32, 2))
    assert len(set(sp.values())) == 1 and 3 <= sp[0] <= 5 and len(live) <= 37 + 160
    # with no room for finer cuts the items stay whole
    sp, _ = _shares(split_work([128] * 40, 37, 37 + 40, 32, 2))
    assert set(sp.values()) == {1}


def test_shares_that_run_at_once_need_no_more_entries():
    """With no more items than the budget, as many entries as the budget hold every cut (a fixed shape's plan has no others)."""
    rng = random.Random(3)
    for _ in range(200):
        budget = rng.randint(1, 80)
        tiles = [rng.choice([0, 1, rng.randint(1, 40), rng.randint(1, 2000)]) for _ in range(rng.randint(1, budget))]
        sp, live = _shares(split_work(tiles, budget, budget, 32, 2))
        assert len(live) <= budget and all((sp.get(i, 0) >= 1) == (t > 0) for i, t in enumerate(tiles))


def test_a_second_round_is_cut_by_the_longest_share_it_leaves():
    """Finer cuts than one round holds: only where the longest share shrinks by a quarter at least, with no more shares than that share needs
    (an item at its most cuts stays as long however short the others' shares are), and within the entries."""
    rng = random.Random(5)
    taken = clamped = 0
    for _ in range(300):
        n = rng.randint(38, 74)
        tiles = [max(1, int(32 ** rng.random())) for _ in range(n)]
        if rng.random() < 0.5:
            tiles[rng.randrange(n)] = rng.randint(100, 2000)
        entries = rng.choice([80, 111, 148])
        one, _ = _shares(split_work(tiles, 74, entries, 32, 2))
        two, live = _shares(split_work(tiles, 74, entries, 32, 2, second_round=True))
        longest = lambda sp: max(-(-tiles[i] // k) for i, k in sp.items())                       # noqa: E731
        assert len(live) <= entries and max(two.values()) <= 32 and all(k <= max(1, -(-tiles[i] // 2)) for i, k in two.items())
        if two == one:
            continue
        taken += 1
        clamped += max(two.values()) == 32
        assert longest(two) + 0.5 < 0.75 * (longest(one) + 0.5)
        assert len(live) == min(sum(min(32, -(-t // L)) for t in tiles) for L in range(2, max(tiles) + 1)
                                if max(-(-t // min(32, -(-t // L))) for t in tiles) <= longest(two))
    assert taken > 45 and clamped > 8


def test_sequences_of_one_length_class_stay_in_one_round():
    """A cut whose shares are hardly shorter than those of one round is not taken, whatever length was asked for."""
    rng = random.Random(6)
    for _ in range(200):
        tiles = [rng.randint(16, 32) for _ in range(61)]
        assert (split_work(tiles, 74, 111, 32, 2) == split_work(tiles, 74, 111, 32, 2, second_round=True)).all()


def test_a_second_thread_never_gets_another_call_s_cut(monkeypatch):
    """The last cut is kept for the next step. Another engine's call that comes in while it is being stored gets its own cut."""
    seen = []

    class Store(dict):
        def __setitem__(self, key, value):
            super().__setitem__(key, value)
            if not seen:
                seen.append(None)
                seen.append(split_work([128, 4], 37, 40, 32, 2))

    monkeypatch.setattr(ops, "_split_memo", Store())
    seen.append(None)
    want = split_work([128, 4], 37, 40, 32, 2).copy()
    split_work([3, 3, 3], 37, 40, 32, 2)
    seen.clear()
    split_work([128, 4], 37, 40, 32, 2)
    assert len(seen) == 2 and (seen[1] == want).all()
