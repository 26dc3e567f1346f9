"""The short way of a decode step through its preparation, beside the general one (host bookkeeping only)."""
import copy
import random
from types import SimpleNamespace

import pytest

from llm_steadyinfer_b200.cache import CacheLayout, CacheManager, OutOfPages
from llm_steadyinfer_b200.engine.step import ModelRunner, StepEntry, StepError
from llm_steadyinfer_b200.parts.base import CacheNeed

FULL, WINDOW = CacheNeed(2, 16, None), CacheNeed(2, 16, 20)


def runner(needs, pages=24, page_size=4, max_requests=6, max_width=10, prefix=False):
    mgr = CacheManager(CacheLayout(needs, [None] * len(needs)), page_size, pages, max_requests, prefix)
    rn = SimpleNamespace(manager=mgr, page_size=page_size, max_requests=max_requests, max_step_tokens=16, max_width=max_width)
    rn._check_pages_written = lambda entries: ModelRunner._check_pages_written(rn, entries)
    return rn


def pages_of(mgr):
    return [(dict(g.tables), g.pool.num_free) for g in mgr.groups]


@pytest.mark.parametrize("needs", [[FULL], [FULL, WINDOW], [WINDOW]])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_the_short_way_says_what_the_general_way_does(needs, seed):
    """Random steps of prompts and decode rows, refused ones among them: where the short way answers, the general way accepts the step, takes
    no pages, and has the same positions, lengths and slots; where it does not, nothing has changed."""
    rng = random.Random(seed)
    rn = runner(needs)
    mgr, short = rn.manager, 0
    for step in range(400):
        live = list(mgr.requests)
        entries = []
        for r in rng.sample(live, rng.randint(0, len(live))):
            n = rng.choice([1, 1, 1, 1, 1, 1, 3])
            entries.append(StepEntry(r, [rng.randrange(100) for _ in range(n)], rng.choice([[0], [0], [0], [0], [n - 1], []])))
        if rng.random() < 0.15:
            entries.append(StepEntry(f"n{step}", [1] * rng.randint(1, 9), [0]))
        if entries and rng.random() < 0.03:
            entries.append(entries[0])                    # a request twice
        before = copy.deepcopy(pages_of(mgr))
        got = ModelRunner._decode_rows(rn, entries)
        assert pages_of(mgr) == before
        try:
            ModelRunner._admit(rn, entries)
        except (StepError, OutOfPages, RuntimeError):
            assert got is None, entries
            for r in [r for r in mgr.requests if r not in live]:
                mgr.release(r)
        else:
            if got is not None:
                short += 1
                toks, pos, slots = got
                assert pages_of(mgr) == before, "the step takes no pages"
                assert toks == [e.tokens[0] for e in entries] and pos == [mgr.length(e.req) for e in entries]
                assert [p + 1 for p in pos] == rn._new_lengths and slots == [mgr.slot(e.req) for e in entries]
            for e, n in zip(entries, rn._new_lengths):
                mgr.commit(e.req, n)
        for r in list(mgr.requests):
            if rng.random() < 0.02 or mgr.length(r) > 36:
                mgr.release(r)
        mgr.check_invariant()
    assert short >= 20, "the short way is taken often enough to say so"


def test_the_short_way_leaves_shared_pages_and_full_requests_to_the_general_one():
    rn = runner([FULL], prefix=True, max_width=3)
    mgr = rn.manager
    mgr.admit("a")
    mgr.grow("a", 6)
    mgr.commit("a", 6)
    one = [StepEntry("a", [5], [0])]
    assert ModelRunner._decode_rows(rn, one) == ([5], [6], [mgr.slot("a")])
    mgr.groups[0].pool.retain(mgr.table(0, "a")[1])       # the page of the next place has another holder
    assert ModelRunner._decode_rows(rn, one) is None
    with pytest.raises(StepError):
        ModelRunner._admit(rn, one)
    mgr.groups[0].pool.release(mgr.table(0, "a")[1])
    mgr.grow("a", 12)
    mgr.commit("a", 12)                                   # at its limit of three pages
    assert ModelRunner._decode_rows(rn, one) is None
    with pytest.raises(StepError):
        ModelRunner._admit(rn, one)
    for entries in ([], [StepEntry("new", [1], [0])], [StepEntry("a", [1, 2], [0])], [StepEntry("a", [1], [])]):
        assert ModelRunner._decode_rows(rn, entries) is None
