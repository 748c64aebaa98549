"""The tokens of one step and where they belong, as the kernels need it.

A step brings, for each of n sequences, its next tokens (all of a prompt, or one token); rows of all
sequences follow one another without padding.  Everything the device needs to place a row lies in
small int32 arrays: the row's position in its sequence, the sequence it belongs to, each sequence's
slot, first row and length after the step.  Causality is by position: the row at position p sees cached
positions up to p, so a continuation of several tokens onto a sequence that is already cached needs no
mask (the reference needs an explicit one there, fms/modules/attention.py:268-271).
"""
from __future__ import annotations

from typing import List, Optional, Sequence

import numpy as np
import torch


_copies = {}  # device -> the stream of its index arrays' copies


def int32_on(device, values) -> torch.Tensor:
    """Whole numbers on the device, there when this returns, for use on any stream.  The copy has a stream of its own: on the current one
    it would wait, and the host with it, for all that lies in front of it, and the GPU run dry behind it.  The memory is the copies'
    stream's and is not given out again before what the current stream had been given when the tensor is freed is done.  A capture refuses the
    copy."""
    device = torch.device(device)
    values = torch.from_numpy(np.array(values, dtype=np.int32))  # by way of numpy: 178 us for 6,000 numbers where torch.tensor took 314
    if device.type != "cuda" or torch.cuda.is_current_stream_capturing():
        return values.to(device)
    current = torch.cuda.current_stream(device)
    stream = _copies.get(current.device)
    if stream is None:
        stream = _copies.setdefault(current.device, torch.cuda.Stream(current.device))
    with torch.cuda.stream(stream):
        out = values.to(current.device)
    out.record_stream(current)
    return out


def row_sides(num_new: Sequence[int], least: int, device, in_runs: bool = False):
    """A step's rows by whether their sequence brings ``least`` tokens: (whether it does, first row, rows, None) for rows that lie one
    behind the other, (whether, 0, rows, their places: int32 on the device) for all of a side that does not; ``in_runs``: every run of
    neighbours for itself, which needs nothing on the device."""
    runs, at = {True: [], False: []}, 0
    for n in num_new:
        side = runs[n >= least]
        if side and side[-1][1] == at:
            side[-1][1] += n
        elif n:
            side.append([at, at + n])
        at += n
    out = []
    for many, side in runs.items():
        if len(side) > 1 and not in_runs:
            places = [r for a, b in side for r in range(a, b)]
            out.append((many, 0, len(places), int32_on(device, places)))
        else:
            out.extend((many, a, b - a, None) for a, b in side)
    return out


class Batch:
    """Device arrays of one step.  Built by ``Batch.from_lists`` for a general step, or filled in place
    by the decode loop (``engine.step.DecodeState``) when every sequence brings one token."""

    def __init__(self) -> None:
        self.n_seqs = 0
        self.n_tokens = 0
        self.decode = False  # every sequence brings exactly one token
        self.max_new = 0  # most tokens any sequence brings
        self.max_len_after = 0  # longest sequence after the step (host value; capacity when unknown)
        self.total_len = 0  # tokens of all sequences after the step, as far as the host knows (kernels are chosen by it)
        self.num_new: List[int] = []
        self.tokens: Optional[torch.Tensor] = None  # [n_tokens] int32
        self.positions: Optional[torch.Tensor] = None  # [n_tokens] int32: each token's place in its sequence's cache
        # [n_tokens] int32: the position each token's encoding sees, where that is not its place in the cache (a
        # sequence that started at another position than 0); None: the same
        self.position_ids: Optional[torch.Tensor] = None
        self.token_seq: Optional[torch.Tensor] = None  # [n_tokens] int32, index into the arrays below
        self.first_row: Optional[torch.Tensor] = None  # [n_seqs + 1] int32
        self.slots: Optional[torch.Tensor] = None  # [n_seqs] int32
        self.len_after: Optional[torch.Tensor] = None  # [n_seqs] int32
        self.want_rows: Optional[torch.Tensor] = None  # [n_wanted] int32 rows whose logits are returned
        self.n_wanted = 0
        self._tiles = {}
        self.len_before_host: Optional[List[int]] = None  # lengths before the step, where the host made the batch of lists
        self.scratch = {}  # what a step's layers share (a table of rotation angles, ...); emptied when a step starts

    @staticmethod
    def from_lists(slots: Sequence[int], len_before: Sequence[int], tokens: Sequence[Sequence[int]],
                   want: Sequence[Sequence[int]], device, offsets: Optional[Sequence[int]] = None) -> "Batch":
        """``offsets[i]``: the position at which sequence i started (its token at place p of the cache has the
        position p + offsets[i]); None: every sequence started at 0."""
        b = Batch()
        b.n_seqs = len(slots)
        b.num_new = [len(t) for t in tokens]
        b.n_tokens = sum(b.num_new)
        b.max_new = max(b.num_new)
        b.decode = b.max_new == 1
        b.max_len_after = max(lb + n for lb, n in zip(len_before, b.num_new))
        b.total_len = sum(len_before) + b.n_tokens
        flat, pos, seq, first, rows = [], [], [], [0], []
        for i, (lb, t, w) in enumerate(zip(len_before, tokens, want)):
            base = first[-1]
            flat.extend(int(x) for x in t)
            pos.extend(range(lb, lb + len(t)))
            seq.extend([i] * len(t))
            first.append(base + len(t))
            for j in w:
                if not (0 <= j < len(t)):
                    raise ValueError(f"wanted place {j} outside the {len(t)} tokens of this step")
                rows.append(base + j)
        len_after = [lb + n for lb, n in zip(len_before, b.num_new)]
        ids = [p + offsets[i] for p, i in zip(pos, seq)] if offsets is not None and any(offsets) else []
        packed = int32_on(device, flat + pos + seq + first + list(slots) + len_after + ids + rows)
        n, s = b.n_tokens, b.n_seqs
        o = 0
        b.tokens = packed[o:o + n]; o += n
        b.positions = packed[o:o + n]; o += n
        b.token_seq = packed[o:o + n]; o += n
        b.first_row = packed[o:o + s + 1]; o += s + 1
        b.slots = packed[o:o + s]; o += s
        b.len_after = packed[o:o + s]; o += s
        if ids:
            b.position_ids = packed[o:o + n]; o += n
        b.want_rows = packed[o:]
        b.n_wanted = len(rows)
        b.len_before_host = list(len_before)
        return b

    def row_chunks(self, chunk: int, chosen: Optional[Sequence[bool]] = None):
        """(chunk_rows [chunks, 2] int32: first row and end of every run of up to ``chunk`` rows of one sequence;
        first_chunk [n_seqs + 1] int32: where each sequence's runs start in that list), for kernels that walk a
        sequence's rows run by run.  ``chosen``: whether a sequence has runs at all (default: every one)."""
        key = self.row_chunks_key(chunk, chosen)
        if key not in self._tiles:
            rows, first, base = [], [0], 0
            for i, n in enumerate(self.num_new):
                if chosen is None or chosen[i]:
                    for r in range(0, n, chunk):
                        rows.append((base + r, base + min(n, r + chunk)))
                first.append(len(rows))
                base += n
            packed = int32_on(self.tokens.device, [v for p in rows for v in p] + first)
            self._tiles[key] = (packed[: 2 * len(rows)].view(-1, 2), packed[2 * len(rows):])
        return self._tiles[key]

    @staticmethod
    def row_chunks_key(chunk: int, chosen: Optional[Sequence[bool]] = None):
        """Where ``row_chunks`` keeps what it makes."""
        return ("chunks", chunk) if chosen is None or all(chosen) else ("chunks", chunk, tuple(chosen))

    def rows_seen(self, i: int, window: int) -> int:
        """How many rows ``key_rows`` lays out for sequence i."""
        before = self.len_before_host[i]
        return before + self.num_new[i] - (max(0, before - window + 1) // 64 * 64 if window > 0 else 0)

    def key_passes(self, window: int, most: int, members: Optional[Sequence[int]] = None) -> List[List[int]]:
        """The sequences (default: all) in runs that see at most ``most`` rows together; one that sees more is a run of its own."""
        passes, rows = [], 0
        for i in (range(self.n_seqs) if members is None else members):
            seen = self.rows_seen(i, window)
            if not passes or rows + seen > most:
                passes.append([])
                rows = 0
            passes[-1].append(i)
            rows += seen
        return passes

    def key_rows(self, window: int, members: Optional[Sequence[int]] = None):
        """(start, first, base: int32 [n_seqs + 1], [n_seqs], [n_seqs]; rows): the keys that a step of several tokens sees,
        laid one sequence behind the other.  Sequence i's are the rows start[i] .. start[i + 1] and begin at its position
        first[i] (0, or with a window the first of the cache block that holds the earliest key seen); its position p is row
        base[i] + p.  ``members``: the sequences that have rows (default: every one)."""
        key = ("keys", window, self._of(members))
        if key not in self._tiles:
            start, first = [0], []
            for i, (before, n) in enumerate(zip(self.len_before_host, self.num_new)):
                seen = self.rows_seen(i, window)
                first.append(before + n - seen)
                start.append(start[-1] + (seen if members is None or i in members else 0))
            base = [a - b for a, b in zip(start, first)]
            packed = int32_on(self.tokens.device, start + first + base)
            s = len(first)
            self._tiles[key] = (packed[: s + 1], packed[s + 1: 2 * s + 1], packed[2 * s + 1:], start[-1])
        return self._tiles[key]

    def row_sides(self, least: int, in_runs: bool = False):
        """``row_sides`` of the step's sequences; what the device needs for it is kept."""
        key = ("sides", least)
        if key in self._tiles:
            return self._tiles[key]
        out = row_sides(self.num_new, least, self.tokens.device, in_runs)
        if not in_runs:
            self._tiles[key] = out
        return out

    def query_tiles(self, tile_rows: int, members: Optional[Sequence[int]] = None) -> torch.Tensor:
        """[tiles, 2] int32: (sequence index, first row of the tile within the sequence's new tokens), for
        kernels that give each thread block ``tile_rows`` rows of one sequence.  ``members``: the sequences that have
        tiles (default: every one)."""
        key = (tile_rows, self._of(members))
        if key not in self._tiles:
            t = []
            for i, n in enumerate(self.num_new):
                if members is None or i in members:
                    t.extend((i, r) for r in range(0, n, tile_rows))
            self._tiles[key] = int32_on(self.tokens.device, t)
        return self._tiles[key]

    def _of(self, members: Optional[Sequence[int]]):
        """Part of a key: the sequences that something is made for, None for all of them."""
        return None if members is None or len(members) == self.n_seqs else tuple(members)
