"""The pinned staging buffers of a step and of the sampler (host side only, with stand-ins for the device's events and streams)."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from llm_steadyinfer_b200.engine import step
from llm_steadyinfer_b200.sampling import sampler
from llm_steadyinfer_b200.sampling.sampler import Sampler


class Event:
    """As torch.cuda.Event: it belongs to the device of its first recording, and another device's stream is an error."""

    def __init__(self):
        self.device = None

    def record(self, stream=None):
        device = (stream or torch.cuda.current_stream()).device
        if self.device is not None and self.device != device:
            raise RuntimeError("Event device does not match recording stream's device")
        self.device = device

    def synchronize(self):
        pass


@pytest.fixture
def here(monkeypatch):
    """The calling thread's current device, to be changed between calls."""
    now = SimpleNamespace(device=torch.device("cuda:1"))
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(device=torch.device(device) if device is not None else now.device))
    return now


def test_a_ring_is_fed_by_threads_at_other_devices(here):
    ring = object.__new__(step._PinnedRing)
    ring.cap, ring.turn, ring.events = 8, 0, [None] * 4
    ring.hosts = [torch.zeros(8, dtype=torch.int32) for _ in range(4)]
    ring.arrays = [h.numpy() for h in ring.hosts]
    ring.dev = torch.zeros(8, dtype=torch.int32)
    for i in range(12):
        here.device = torch.device(f"cuda:{i // 4}")
        ring.next_host()[:2] = i
        ring.send(2)
        assert ring.dev[:2].tolist() == [i, i]
    assert {e.device for e in ring.events} == {ring.dev.device}


def test_a_sampler_is_called_by_threads_at_other_devices(here, monkeypatch):
    s = object.__new__(Sampler)
    s.max_rows, s._host_turn, s._host_events, s._device_views = 2, 0, [None] * 4, {}
    s._hosts = [torch.zeros(16, dtype=torch.int32) for _ in range(4)]
    s._arrays = [h.numpy() for h in s._hosts]
    s._dev, s._out, s.device = torch.zeros(16, dtype=torch.int32), torch.zeros(2, dtype=torch.int32), torch.device("cpu")
    seen = []
    monkeypatch.setattr(sampler.ops, "sample", lambda logits, out, **kw: seen.append(float(kw["temperature"][0])))
    for i in range(12):
        here.device = torch.device(f"cuda:{i // 4}")
        p = SimpleNamespace(temperature=1.0 + i, top_p=1.0, top_k=0, greedy=False)
        s.sample(torch.zeros(1, 5), [(p, 1, 2)])
    assert np.allclose(seen, 1.0 + np.arange(12))
