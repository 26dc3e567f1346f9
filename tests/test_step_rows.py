"""Which form of a recurrence a step takes, from the rows that its sequences bring (host side only)."""
from types import SimpleNamespace

import numpy as np
import pytest

from llm_steadyinfer_b200.parts import delta_rule, time_mix
from llm_steadyinfer_b200.parts.delta_rule import GatedDeltaRule
from llm_steadyinfer_b200.parts.time_mix import TimeMix


def step(rows, seq_cap=None):
    return SimpleNamespace(h_q_start=np.cumsum([0] + rows), num_seqs=len(rows), seq_cap=seq_cap, plans={})


@pytest.mark.parametrize("rows,delta,decay", [
    ([1] * 40, False, False), ([2], False, False), ([27], False, False), ([28], False, True), ([63], False, True), ([64], True, True),
    ([16] * 2, False, False), ([8] * 3, False, False), ([10] * 3, False, True), ([2] * 16, False, True), ([2] * 160, False, True),
    ([16] * 9 + [16], True, True), ([54] * 3, False, True), ([4] * 40, True, True), ([64] + [1] * 7, True, True), ([9] + [1] * 30, False, False),
])
def test_short_portions_go_token_by_token(monkeypatch, rows, delta, decay):
    """Groups of four tokens have a launch more; they are for steps whose portions pay for it, and never for a fixed shape."""
    monkeypatch.setattr(delta_rule.ops, "channel_delta_groups_ok", lambda dk, dv: True)
    monkeypatch.setattr(time_mix.ops, "decay_groups_ok", lambda n: True)
    monkeypatch.setattr(time_mix.ops, "sm_count", lambda device=None: 148)
    T = sum(rows)
    d, m = SimpleNamespace(dk=128, dv=128), SimpleNamespace(H=32, n=64, device=None)
    assert GatedDeltaRule.by_groups(d, step(rows), T) == delta
    assert TimeMix.by_groups(m, step(rows), T) == decay
    assert not GatedDeltaRule.by_groups(d, step(rows, seq_cap=len(rows)), T) and not TimeMix.by_groups(m, step(rows, seq_cap=len(rows)), T)
