"""The description of one step's batch that every part sees."""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import Any

import torch


@dataclass
class GroupView:
    """Per cache group (layers with the same cache needs): where the step's new tokens go
    and where each sequence's pages are."""
    slots: torch.Tensor          # int32 [T]: page * page_size + offset
    block_table: torch.Tensor    # int32 [S, P]: page ids, -1 where given back / not yet held
    page_size: int


# Steps whose longest portion has this many rows run their recurrences in chunks of 64, portions of CHUNK_FROM rows and more,
# the shorter ones row by row beside them. Measured, row by row against chunks, us: 16 heads of 128 x 128, delta rule with
# decays per channel 64 rows 35 / 56, 128 rows 68 / 59, 256 rows 128 / 83, 512 rows 253 / 96, portions of 281, 199 and 117 rows
# 221 / 126 (199 with the last one row by row), 17 single tokens beside 256 rows 210 / 111; gated linear attention 57 / 50 at 128
# rows, 109 / 57 at 256; state space with 32 heads 49 / 37 and 95 / 44. Four portions of 128 rows with 32 heads are level. Below 256
# rows a step waits for its launches, of which chunks take three.
LONG_FROM, CHUNK_FROM = 256, 64
# A walk row by row takes as long as its longest portion while there is room beside it; once heads and portions fill the GPU, chunks
# take about as many FMAs and more traffic. `pairs` = heads x (rows of the portions in chunks / the longest), us row by row / in
# chunks, portions of 256: delta rule with a decay per head, 128 x 128: 64 pairs 193 / 117, 128 207 / 235, 256 375 / 430; decays per
# channel 64 244 / 135, 128 274 / 269, 256 487 / 488; state space, 128 x 64: 128 175 / 100, 256 189 / 200; heads of 64 x 64: 64 89 / 55,
# 128 111 / 105, 140 116 / 142, 256 159 / 197; gated linear attention of 128 64 153 / 92, 128 166 / 183. Its three passes over chunks,
# from 384 rows on, are the slower form at any number (128 x 128, 256 pairs of 512 rows 1,403 / 601; heads of 64 level at 64).
CHUNK_PAIRS, CHUNK_COLUMNS = 128, 96 * 128     # pairs, and value columns of all pairs, up to which a step's portions run in chunks


@dataclass
class StepContext:
    """One batch: T tokens of S sequences, rows of a sequence adjacent and in order.

    Device tensors (int32): `token_ids` [T], `positions` [T] (absolute position of each
    token in its sequence), `token_seq` [T] (which sequence), `cu_q` [S+1] (row range of
    each sequence), `kv_lens` [S] (keys visible to the sequence's last token, new ones
    included), `state_slots` [S]. Host mirrors (`q_lens`, `kv_lens_host`, ...) let a part
    choose a kernel without a device read."""
    backend: Any
    num_tokens: int
    num_seqs: int
    token_ids: torch.Tensor
    positions: torch.Tensor
    token_seq: torch.Tensor
    cu_q: torch.Tensor
    kv_lens: torch.Tensor
    state_slots: torch.Tensor | None
    q_lens_host: list[int]
    kv_lens_host: list[int]
    state_slots_host: list[int]
    groups: dict[int, GroupView] = field(default_factory=dict)
    max_q_len: int = 1
    max_kv_len: int = 1
    # decode-only steps captured in a CUDA graph read their sizes from device memory
    graph_safe: bool = False
    extras: dict[str, Any] = field(default_factory=dict)
    # what one forward pass shares between its layers (tables made at first use); the model
    # empties it when a pass begins, so nothing outlives the pass that made it
    per_forward: dict[str, Any] = field(default_factory=dict)

    @property
    def all_decode(self) -> bool:
        return self.max_q_len == 1

    def long_rows(self, heads: int, vdim: int, walked: bool = True) -> dict:
        """What a recurrence's scan is told about a step with a long portion: from how many rows on a sequence runs in
        chunks as products of matrices, whether there are shorter ones beside it, and how many such sequences and chunks of 64
        there are. Empty where chunks do not pay; `walked`: the other form goes row by row."""
        if self.graph_safe or self.max_q_len < LONG_FROM:
            return {}
        long = [n for n in self.q_lens_host if n >= CHUNK_FROM]
        pairs = heads * sum(long) / self.max_q_len
        if walked and (pairs > CHUNK_PAIRS or pairs * vdim > CHUNK_COLUMNS):
            return {}
        return {"long_from": CHUNK_FROM, "any_short": len(long) < self.num_seqs, "longs": len(long),
                "chunks": sum((n + 63) // 64 for n in long)}
