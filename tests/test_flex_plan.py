"""The work lists of the general tensor-core attention (host side only; the kernels' own answers are stood in for)."""
from types import SimpleNamespace

import numpy as np
import pytest

from llm_steadyinfer_b200.parts import flex_plan
from llm_steadyinfer_b200.parts.attention import Attention


class Upload:
    """An uploaded list: the buffer's contents are whatever was uploaded under its name last."""

    def __init__(self, store, key, n):
        self.store, self.key, self.n = store, key, n

    def view(self, *shape):
        return self

    def items(self):
        return [tuple(r) for r in self.store[self.key][:self.n].reshape(-1, 4).tolist()]


class Ctx:
    """What a plan asks of a step: its sequences (rows they bring, keys they end with) and places to keep things."""

    def __init__(self, seqs, seq_cap=None):
        self.num_seqs, self.seq_cap, self.plans, self.uploads = len(seqs), seq_cap, {}, {}
        self.h_q_start = np.cumsum([0] + [n for n, _ in seqs])
        self.h_ctx_len = np.array([end for _, end in seqs])

    def upload_ints(self, key, values, capacity=None):
        self.uploads[key] = np.ascontiguousarray(values).reshape(-1)
        return Upload(self.uploads, key, values.size)

    def buf(self, key, shape, dtype):
        return (key, tuple(shape))


@pytest.fixture(autouse=True)
def kernels(monkeypatch):
    """What the kernels say of their items: 64 rows in parts of a divisor of the heads, two tiles of 128 rows."""
    def flex_tokens(H, KV):
        return 64 // max(g for g in range(1, min(H // KV, 64) + 1) if (H // KV) % g == 0)
    monkeypatch.setattr(flex_plan.ops, "attn_flex_tokens", flex_tokens)
    monkeypatch.setattr(flex_plan.ops, "attn_portion_tc05_tokens", lambda H, KV: 2 * (128 // (H // KV)))
    monkeypatch.setattr(flex_plan.ops, "attn_flex_scratch_floats", lambda items, H, KV, dv, nsplit: items * H * dv * nsplit)
    monkeypatch.setattr(flex_plan.ops, "sm_count", lambda device=None: 148)


def plan(ctx, H, KV, gen=True, dk=128, dv=128):
    return flex_plan.plan(ctx, None, H, KV, dk, dv, True, None, gen=gen)


@pytest.mark.parametrize("G", [1, 16, 128])
def test_a_fixed_shape_has_the_same_lists_for_every_number_of_sequences(G):
    """A recorded step is replayed with more or fewer sequences than it was recorded with: its lists keep their lengths."""
    shapes = set()
    for live in (1, 3, 4):
        p = plan(Ctx([(1, 700 + s) for s in range(live)], seq_cap=4), G, 1)
        assert p["gen"] is None and p["por"] is None
        items = p["dec"].items()
        assert [it[0] for it in items if it[2]] == list(range(live)), "every sequence has its item"
        shapes.add((len(items), p["nsplit"], p["scratch"], p["dec_rows"]))
    assert len(shapes) == 1


def test_single_rows_keep_their_shares_of_keys():
    """A row of 128 query heads a key head fills the prompt kernel's tile, but it is a decode row: its keys are cut over blocks."""
    p = plan(Ctx([(1, 9000)]), 128, 1)
    assert p["gen"] is None and p["nsplit"] > 1 and p["dec"].items() == [(0, 0, 1, 8999)]
    p = plan(Ctx([(2, 9000)]), 128, 1)
    assert p["dec"] is None and p["gen"].items() == [(0, 0, 2, 8998)]


def test_layers_that_differ_in_the_prompt_kernel_keep_lists_of_their_own():
    """Two layers of one head layout, one whose form the prompt kernel takes and one whose it does not, in one step: both plans are made
    before either is used, so neither upload may take the other's place."""
    seqs = [(100, 100), (300, 300)]                   # one key head a query head: 100 rows stay with the general kernel, 300 do not
    ctx = Ctx(seqs)
    with_gen, without = plan(ctx, 4, 4, gen=True), plan(ctx, 4, 4, gen=False)
    for p, want in ((with_gen, {0: 100}), (without, {0: 100, 1: 300})):
        rows = {}
        for seq, _, n, _ in p["por"].items():
            rows[seq] = rows.get(seq, 0) + n
        assert rows == want
    assert sum(n for _, _, n, _ in with_gen["gen"].items()) == 300


@pytest.mark.parametrize("first", [True, False])
def test_a_layer_whose_scores_the_extended_form_does_not_know_gets_no_items_there(first):
    """Layers of one head layout in one step, one with a gate (the extended form takes it), one with a bias by distance (it does not)."""
    ctx = Ctx([(400, 400)])
    layers = {ok: SimpleNamespace(H=4, KV=4, hs=128, window=None, chunk=None, _tag=lambda: "4_4_128_None", general_tc05_ok=lambda page, ok=ok: ok)
              for ok in (True, False)}
    got = {ok: Attention._plan_general_tc05(layers[ok], ctx, 16) for ok in (first, not first)}
    assert got[False] == {"skip": frozenset(), "all": False, "items": None}
    assert got[True]["all"] and sum(n for _, _, n, _ in got[True]["items"].items()) == 400


@pytest.mark.parametrize("H,KV,dk,dv,own_v,rows", [(16, 1, 576, 512, False, 16), (64, 1, 576, 512, False, 8), (8, 2, 256, 256, True, 8), (16, 4, 192, 128, True, 8),
                                                   (16, 4, 128, 128, True, 8), (16, 2, 128, 128, False, 8), (32, 8, 64, 64, True, 4), (8, 2, 320, 128, True, 3)])
def test_long_rows_are_cut_for_the_blocks_that_run_at_once(H, KV, dk, dv, own_v, rows):
    """No more blocks than three a multiprocessor where its 228 KB hold three (two stages of keys and, where they are others, of values, the
    query rows, the exchanged scores, 1 KB of the system's), two elsewhere; and no fewer than half of them."""
    p = flex_plan.plan(Ctx([(1, 8000)] * rows), None, H, KV, dk, dv, own_v, None)
    pitch, few = -(-dk // 64) * 64, p["dec_rows"] <= 16
    tile, columns = 64 if pitch <= 256 else 32, 128 if dv > 64 else 64
    slices = not own_v and few and dv > columns
    q_rows = 16 if slices or (few and tile == 64) else 64
    block = (q_rows + 2 * tile) * pitch * 2 + (2 * tile * columns * 2 if own_v else 0) + (tile * 256 if slices else 0) + 1024
    most = (3 if 3 * block <= 228 * 1024 else 2) * 148
    blocks = rows * p["nsplit"] * KV * (-(-dv // (4 * columns)) if slices else -(-dv // columns))
    assert most // 2 < blocks <= most or p["nsplit"] == 31
