"""Work lists of the general tensor-core attention (``attention_flex.cu``), made on the host before a step.

A sequence's rows of the step become work items of at most ``ops.attn_flex_tokens`` tokens. Sequences that bring
few rows (decode rows, short ends of prompts: one item) form one launch whose items have their keys cut into
shares, as many as fill the device; longer portions form another without shares, or, where the caller's form is one that
the tcgen05 prompt kernel takes (``gen_ok``) and they fill a tile of its rows, go there. A plan is kept under a key of
the step's context, so layers with the same head layout make it once.
"""
from __future__ import annotations

import numpy as np
import torch

from ..csrc import ops
from .base import first_visible_key

MAX_SPLITS = 32
MIN_KEYS_PER_SPLIT = 256
GEN_MIN_ROWS = 128        # rows (tokens x query heads of a key head) of a sequence from which on the tcgen05 prompt kernel serves it


def gen_ok(H: int, KV: int, dk: int, dv: int, page_size: int, v_share: int = 1, bias: bool = False, cap: bool = False) -> bool:
    """True when portions of this form (values of their own; no slopes, temperature or gate) go to the tcgen05 prompt kernel."""
    return ops.attn_portion_gen_ok(H, KV, dk, dv, v_share, page_size, bias, cap)


def plan(ctx, device, H: int, KV: int, dk: int, dv: int, own_v: bool, window, skip=frozenset(), chunk=None, gen: bool = False) -> dict:
    """``skip``: sequences of the step that get no items (another path serves them). ``window``, ``chunk``: what a row sees. ``gen``: what
    ``gen_ok`` says of the form."""
    key = ("flex", H, KV, dk, dv, own_v, window, chunk, gen, tuple(sorted(skip)))
    got = ctx.plans.get(key)
    if got is not None:
        return got
    per_item = ops.attn_flex_tokens(H, KV)
    gen_item = ops.attn_portion_tc05_tokens(H, KV) if gen else 0
    fixed = ctx.seq_cap is not None
    dec, por, big = [], [], []
    qs, cl = ctx.h_q_start, ctx.h_ctx_len
    for s in range(ctx.num_seqs):
        if s in skip:
            continue
        row0, n = int(qs[s]), int(qs[s + 1] - qs[s])
        pos0 = int(cl[s]) - n
        # (never in a fixed shape, whose lists must not depend on the number of sequences, nor for what is one item of the other
        # kernel, which cuts its keys)
        if gen and not fixed and n > per_item and n * (H // KV) >= GEN_MIN_ROWS:
            big += [(s, row0 + b, min(gen_item, n - b), pos0 + b) for b in range(0, n, gen_item)]
        elif n <= per_item:
            dec.append((s, row0, n, pos0))
        else:
            for b in range(0, n, per_item):
                por.append((s, row0 + b, min(per_item, n - b), pos0 + b))
    if fixed:                                         # fixed shapes: pad with empty items, shares by the shape alone
        dec += [(0, 0, 0, 0)] * (ctx.seq_cap - len(dec))
    out = {"dec": None, "por": None, "gen": None, "nsplit": 1, "scratch": None, "dec_rows": 0}
    tag = f"{H}_{KV}_{dk}_{dv}_{int(own_v)}_{window}" + (f"_c{chunk}" if chunk else "") + ("_rest" if skip else "") + ("_gen" if gen else "")
    if dec:
        # blocks one item gets without shares: kv heads x parts of the query heads x slices of the value columns
        gb = max(g for g in range(1, min(H // KV, 64) + 1) if (H // KV) % g == 0)
        slices = -(-dv // (128 if dv > 64 else 64))
        # the most rows of any item; in a fixed shape every item is one token
        out["dec_rows"] = gb * (1 if fixed else max(d[2] for d in dec))
        if not own_v and slices > 1 and out["dec_rows"] <= 16:
            slices = -(-slices // 4)                  # a block's four warps take a slice each
        per = KV * ((H // KV) // gb) * slices
        # keys that are their own values are wide (a latent): a tile is 32 of them, so a share may be half as many keys
        # As many shares as blocks run at once. Where a multiprocessor has no room for three blocks, a cut for three begins a second round. Rows
        # of 8,000 keys in us, the store of the newest keys before it, cut for two and for three: 16 rows of a latent of 576 with 16 heads 65.2,
        # 83.9, 8 rows of one with 64 heads 230.8, 243.3; 8 rows of 2 x 256 with 8 heads 62.2, 85.0, of 4 x 192 with 16 heads 53.9, 71.1. Where
        # three fit: 8 rows of 4 x 128 with 16 heads and biases 62.3, 50.1 (for four 64.1), of 2 x 128 that are their own values 25.8, 22.0 (28.8).
        nsplit = max(1, min(MAX_SPLITS if own_v else 2 * MAX_SPLITS,
                            ops.attn_flex_blocks(dk, dv, own_v, out["dec_rows"]) * ops.sm_count(device) // (len(dec) * per)))
        if not fixed:
            longest = max(d[3] + d[2] - first_visible_key(d[3], window, chunk) for d in dec)
            nsplit = min(nsplit, max(1, longest // MIN_KEYS_PER_SPLIT))
        elif chunk:
            nsplit = min(nsplit, max(1, chunk // MIN_KEYS_PER_SPLIT))
        out["nsplit"] = nsplit
        out["dec"] = ctx.upload_ints("flex_dec_" + tag, np.asarray(dec, dtype=np.int32)).view(-1, 4)
        if nsplit > 1:
            out["scratch"] = ctx.buf("flex_split", (ops.attn_flex_scratch_floats(len(dec), H, KV, dv, nsplit),), torch.float32)
    if por:
        por.sort(key=lambda it: -(it[3] + it[2]))     # the items with most keys first: the last blocks to start are short
        out["por"] = ctx.upload_ints("flex_por_" + tag, np.asarray(por, dtype=np.int32)).view(-1, 4)
    if big:
        big.sort(key=lambda it: it[3] + it[2])        # this kernel starts with the last ones
        out["gen"] = ctx.upload_ints("flex_gen_" + tag, np.asarray(big, dtype=np.int32)).view(-1, 4)
    ctx.plans[key] = out
    return out


def attend(pl: dict, q, k_cache, v_cache, block_table, out, page_size, seq_slots, H, KV, dk, dv, scale, window,
           dist_bias=None, sink=None, status=None, softcap: float = 0.0, v_share: int = 1, slopes=None, q_temp=None,
           gate=None, chunk=None) -> None:
    args = (page_size, seq_slots, H, KV, dk, dv, scale, window or 0)
    if pl["dec"] is not None:                         # one item a sequence: all its rows of the step
        ops.attn_flex(q, k_cache, v_cache, block_table, pl["dec"], out, *args, dist_bias=dist_bias, sink=sink,
                      nsplit=pl["nsplit"], scratch=pl["scratch"], status=status, max_rows=pl["dec_rows"], softcap=softcap,
                      v_share=v_share, slopes=slopes, q_temp=q_temp, gate=gate, chunk=chunk or 0, ahead=True)
    if pl["por"] is not None:
        ops.attn_flex(q, k_cache, v_cache, block_table, pl["por"], out, *args, dist_bias=dist_bias, sink=sink, status=status,
                      softcap=softcap, v_share=v_share, slopes=slopes, q_temp=q_temp, gate=gate, chunk=chunk or 0)
    if pl["gen"] is not None:
        ops.attn_portion_gen(q, k_cache, v_cache, block_table, pl["gen"], out, *args, dist_bias=dist_bias, sink=sink, status=status,
                             softcap=softcap, v_share=v_share, chunk=chunk or 0)
