"""Device tensors behind the cache manager: per group one key and one value tensor
``[layers_in_group, num_pages, kv_heads, page_size, head_dim]`` (values with their own last size and head count, or
none at all for a group whose keys serve as values) and, for mixers with fixed-size state, one tensor ``[slots, *shape]`` per
layer; a place of the layout without a mixer (the embedder's, last) has its state here as well. The reference keeps
``[L, num_blocks, block_size, kv_dim]`` in fp32 (src/source/scheduler/kv_manager.cpp:41-53);
here a page holds each head's rows contiguously and has the compute dtype.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import List, Optional

import numpy as np
import torch

from .manager import CacheLayout, CacheManager


@dataclass
class LayerCache:
    """What one layer's mixer sees of the cache during a step."""
    k: Optional[torch.Tensor]              # [num_pages, kv_heads, page_size, head_dim]
    v: Optional[torch.Tensor]
    block_table: Optional[torch.Tensor]    # int32 [num_seqs, table_width] of the layer's group, this step
    page_size: int
    writes: bool                           # False for a layer that reads another layer's cache
    state: Optional[torch.Tensor]          # [slots, *shape] or None
    group: Optional[int]


class CacheStorage:
    def __init__(self, layout: CacheLayout, manager: CacheManager, dtype: torch.dtype, device):
        self.layout = layout
        self.manager = manager
        self.dtype = dtype
        self.device = torch.device(device)
        self.keys: List[torch.Tensor] = []
        self.values: List[torch.Tensor] = []
        ps = manager.page_size
        for g, grp in enumerate(manager.groups):
            shape = (len(grp.layers), grp.pool.num_pages, grp.need.num_kv_heads, ps)
            self.keys.append(torch.zeros(shape + (grp.need.head_dim,), dtype=dtype, device=self.device))
            # a group without values of their own (value_dim 0) has no second tensor
            vshape = (len(grp.layers), grp.pool.num_pages, grp.need.v_heads, ps, grp.need.v_dim)
            self.values.append(torch.zeros(vshape, dtype=dtype, device=self.device) if grp.need.v_dim else None)
        # every place's view of its group's tensors, made once: a step asks for all of them
        self._pages = []
        for i in range(len(layout.needs)):
            g, j = layout.layer_group[i], layout.layer_index_in_group[i]
            self._pages.append(None if g is None else (g, self.keys[g][j], None if self.values[g] is None else self.values[g][j]))
        self.states: List[Optional[torch.Tensor]] = []
        for s in layout.states:
            self.states.append(None if s is None else torch.zeros(
                (manager.slots.num_slots, *s.shape), dtype=s.dtype, device=self.device))

    def bytes(self) -> int:
        n = sum(t.numel() * t.element_size() for t in self.keys + self.values if t is not None)
        return n + sum(t.numel() * t.element_size() for t in self.states if t is not None)

    def zero_new_slots(self, upload=None) -> None:
        """State of requests admitted (or reset) since the last call starts at zero. ``upload(key, values, capacity)``: a device copy of
        a small int32 array that the host does not wait for (None: a copy that it waits for)."""
        slots = self.manager.new_slots
        if slots and any(t is not None for t in self.states):
            fresh = sorted(set(slots))
            if upload is None:
                idx = torch.tensor(fresh, dtype=torch.long, device=self.device)
            else:
                idx = upload("new_slots", np.asarray(fresh, dtype=np.int32), self.manager.slots.num_slots).to(torch.long)
            for t in self.states:
                if t is not None:
                    t.index_fill_(0, idx, 0)
        slots.clear()

    def layer_views(self, tables: List[Optional[torch.Tensor]]) -> List[LayerCache]:
        """``tables[g]``: this step's device block table of group g."""
        views = []
        ps = self.manager.page_size
        for i, pages in enumerate(self._pages):
            if pages is None:
                views.append(LayerCache(None, None, None, ps, False, self.states[i], None))
            else:
                g, k, v = pages
                views.append(LayerCache(k, v, tables[g], ps, self.layout.cache_from[i] is None, self.states[i], g))
        return views
