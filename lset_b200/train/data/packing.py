"""Sequence packing: token lists -> one flat stream with ``cu_seqlens``
(output contract of lset/train/data/packing.py:6-21 and the fixed-budget variant of
lset/train/data/packed_collator.py:27-67)."""
from __future__ import annotations

import itertools
from typing import List, Sequence

import numpy as np
import torch


def pack_sequences(sequences: Sequence[Sequence[int]]) -> dict:
    """``{input_ids [T] int64, cu_seqlens [N+1] int32, max_seqlen int, position_ids [T] int64}``;
    positions restart at 0 for every sequence."""
    lens = np.fromiter(map(len, sequences), dtype=np.int64, count=len(sequences))
    total = int(lens.sum())
    ids = np.fromiter(itertools.chain.from_iterable(sequences), dtype=np.int64, count=total)
    cu = np.zeros(len(lens) + 1, dtype=np.int32)
    np.cumsum(lens, out=cu[1:])
    pos = np.arange(total, dtype=np.int64) - np.repeat(cu[:-1].astype(np.int64), lens)
    return {"input_ids": torch.from_numpy(ids), "cu_seqlens": torch.from_numpy(cu),
            "max_seqlen": int(lens.max()) if len(lens) else 0, "position_ids": torch.from_numpy(pos)}


def pack_fixed_budget(sequences: Sequence[Sequence[int]], token_budget: int, pad_token_id: int = 0) -> dict:
    """Pack greedily until ``token_budget``: empty sequences and sequences that do not fit are
    skipped, and the stream is padded at the end to exactly ``token_budget`` tokens (pad tokens
    belong to no sequence, position 0) — fixed shapes for CUDA-graph replay. ``num_sequences``
    counts the packed sequences."""
    kept: List[Sequence[int]] = []
    used = 0
    for s in sequences:
        if len(s) == 0 or used + len(s) > token_budget:
            continue
        kept.append(s)
        used += len(s)
    out = pack_sequences(kept)
    pad = token_budget - used
    if pad > 0:
        out["input_ids"] = torch.cat([out["input_ids"], torch.full((pad,), pad_token_id, dtype=torch.int64)])
        out["position_ids"] = torch.cat([out["position_ids"], torch.zeros(pad, dtype=torch.int64)])
    out["max_seqlen"] = max(out["max_seqlen"], 1)
    out["num_sequences"] = len(kept)
    return out


_pack_fixed_budget = pack_fixed_budget
