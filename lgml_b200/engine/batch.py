"""The description of one step's batch, as the kernels read it.

A step holds, for each request in it, that request's next tokens: a prompt, a
portion of one, or a single decoded token.  All tokens of the step form one
ragged batch (mischief/lgml: ``M:batch_inputs``, ``lua/lgml/transformer.lua:2502-2551``):

* ``token_ids[N]``, ``positions[N]`` (= tokens already cached + index in the portion,
  ``:2441-2447``), ``seq_of_token[N]`` (the row of the request in this batch),
* ``seq_start[S+1]`` (first token of each request), ``seq_pos0[S]``, ``slots[S]``,
* one block table ``[S, width]`` per cache group, -1 where a request has no page,
* ``logit_rows[R]``: the token rows whose logits are wanted (``:2540-2545``).

Everything goes to the device in one copy from pinned memory; no dense mask is
built (the reference fills an (n, window) mask on the host each pass,
``src/lgml.c:2993-3010``; here the attention kernel walks the block table).
"""
from __future__ import annotations

from ctypes import byref, c_int64
from dataclasses import dataclass
from typing import Dict, List, Optional, Sequence

import numpy as np
import torch

from ..host import steps
from ..ops import sm_count


@dataclass
class CacheView:
    """What one layer call sees of the cache."""

    k: Optional[torch.Tensor] = None            # [pages, Hkv, page, D]
    v: Optional[torch.Tensor] = None
    block_table: Optional[torch.Tensor] = None  # int32 [S, width]
    writable: bool = True
    state: Optional[torch.Tensor] = None        # [max_slots, ...] for a fixed-state layer
    page_size: int = 0


def cache_view_of(cm, owner: int, block_tables, writable: bool = True) -> CacheView:
    """The cache of schedule entry ``owner`` as a step's requests see it: its pages with the step's block
    table, its state slots, or both when the layer keeps both."""
    view = CacheView(writable=False)
    g = cm.group_of_layer.get(owner)
    if g is not None:
        grp = cm.groups[g]
        view = CacheView(k=grp.k[owner], v=grp.v[owner], block_table=block_tables[g], writable=writable, page_size=cm.page_size)
    sg = cm.state_group_of_layer.get(owner)
    if sg is not None:
        view.state = cm.state_groups[sg].state[owner]
        view.writable = writable
    return view


@dataclass
class ScanChunks:
    """The tokens of a step's requests that bring more than ``longer_than`` of them, in chunks of consecutive tokens."""

    rows: torch.Tensor          # int32 [n_chunks, 2]: first token row, the row past the last; a request's chunks in a row
    first: torch.Tensor         # int32 [requests + 1]: the first chunk of every one of them
    requests: torch.Tensor      # int32 [requests]: which requests of the step they are
    longer_than: int
    short: bool                 # whether the step holds other requests too
    chunk_tokens: int = 0       # most tokens of a chunk (0: not said)


class StepBatch:
    """Host lists -> one int32 buffer -> one copy -> device views.

    ``table_widths`` forces the width of each group's block table and ``device_buffer``
    makes the views live in a buffer the caller keeps: both are what a captured CUDA graph
    needs, since its kernels were recorded with fixed addresses and strides.

    ``lists``: which tiles and pieces the layers of this model have asked for in steps so far; this step's then come
    with its one copy, and what a layer asks for that is not among them is added (a copy of its own this time)."""

    MAX_LISTS = 16

    def __init__(self, cache_manager, requests: Sequence, tokens: Sequence[Sequence[int]], want: Sequence[Sequence[int]],
                 device, pinned: Optional[torch.Tensor] = None, table_widths: Optional[Sequence[int]] = None,
                 device_buffer: Optional[torch.Tensor] = None, lists: Optional[Dict[tuple, None]] = None):
        cm = cache_manager
        self.cache_manager = cm
        self.requests = list(requests)
        S = len(self.requests)
        lens = [len(t) for t in tokens]
        N = sum(lens)
        self.n_tokens, self.n_seqs = N, S
        self.seq_lens = lens
        self.pos0 = [r.n_tokens for r in self.requests]
        self.kv_lens = [p + n for p, n in zip(self.pos0, lens)]
        self.max_q_len = max(lens) if lens else 0
        self.max_kv_len = max(self.kv_lens) if lens else 0
        self.min_kv_len = min(self.kv_lens) if lens else 0
        self.decode_splits = None       # a fixed split count (set by a captured graph)
        self.shared = {}                # what one layer of this step keeps for later layers (by name)
        self._tiles = {}
        self.replayed = False           # are its launches recorded, and run again for other contexts?
        self.replay_reach = 0           # ... of over half of so many tokens and up to all of them (0: any that are short)
        self.after_staged_copy = None   # called after a later copy out of the pinned buffer (its owner marks the buffer busy again)

        # Rows of tokens are written by C: a prompt portion brings thousands of them, and Python's way with them costs as much as
        # the step's first layers.
        self._lens, self._pos0 = (c_int64 * S)(*lens), (c_int64 * S)(*self.pos0)
        starts = [0]
        for n in lens:
            starts.append(starts[-1] + n)
        rows: List[int] = []
        self.rows_of_seq: List[List[int]] = []
        for s, w in enumerate(want):
            mine = []
            for i in w:
                if not 0 <= i < lens[s]:
                    raise IndexError(f"wanted place {i} is outside the {lens[s]} tokens request {self.requests[s].id!r} brings")
                mine.append(len(rows))
                rows.append(starts[s] + int(i))
            self.rows_of_seq.append(mine)
        self.n_rows = len(rows)

        tables = []
        for g in range(len(cm.groups)):
            tables.append(cm.block_table_rows(self.requests, g, table_widths[g] if table_widths else None))
        self.table_width = [len(t[0]) if t else 1 for t in tables]
        n_rows_field = max(len(rows), 1)
        described = total = 3 * N + (S + 1) + 3 * S + n_rows_field + S * sum(self.table_width)
        self._lists = lists
        ahead = [k for k in lists or () if self._wanted(k)]
        total += sum(self._room(k) + 3 for k in ahead)          # (each from a 16-byte boundary)
        if pinned is None or pinned.numel() < total or device_buffer is not None:
            ahead, total = [], described
        if pinned is not None and pinned.numel() >= total:
            host = pinned[:total]
            self._pinned, self._pinned_used = pinned, total
        else:
            host = torch.empty(total, dtype=torch.int32)
            self._pinned, self._pinned_used = None, 0
        h = host.numpy()
        off = 0
        for t, n in zip(tokens, lens):
            h[off:off + n] = t if isinstance(t, np.ndarray) else np.asarray(t, dtype=np.int64).reshape(-1)
            off += n
        steps().lgml_steps_rows(host.data_ptr() + 4 * N, S, self._lens, self._pos0)
        off = 3 * N
        off += S + 1
        h[off:off + S] = self.pos0
        off += S
        h[off:off + S] = [r.slot for r in self.requests]
        off += S
        h[off:off + S] = self.kv_lens
        off += S
        h[off:off + n_rows_field] = rows or [0]
        off += n_rows_field
        for t, w in zip(tables, self.table_width):
            if S:
                h[off:off + S * w] = np.asarray(t, dtype=np.int64).reshape(-1)
            off += S * w
        written = []
        for k in ahead:
            off = -(-off // 4) * 4
            n, shape = self._write(k, host.data_ptr() + 4 * off)
            written.append((k, off, n, shape))
            off += n
        if ahead:
            total = self._pinned_used = off
            host = pinned[:total]
        if device_buffer is not None:
            if device_buffer.numel() < total:
                raise ValueError("the step's description does not fit the buffer kept for it")
            dev = device_buffer[:total]
        else:
            dev = torch.empty(total, dtype=torch.int32, device=device)
        dev.copy_(host, non_blocking=True)
        self.h2d_bytes = total * 4
        self._dev = dev
        off = 0

        def take(n):
            nonlocal off
            v = dev[off:off + n]
            off += n
            return v

        self.token_ids = take(N)
        self.positions = take(N)
        self.seq_of_token = take(N)
        self.seq_start = take(S + 1)
        self.seq_pos0 = take(S)
        self.slots = take(S)
        self.seq_kv_len = take(S)
        r = take(max(len(rows), 1))
        self.logit_rows = r[: len(rows)]
        self.block_tables = [take(S * w).view(S, w) for w in self.table_width]
        for k, at, n, shape in written:
            self._tiles[k] = self._views(k, dev[at:at + n], shape)

    # ---- tiles and pieces: ("tiles", tokens, longer than), ("halves", tokens, CTAs a tile), ("pieces", tokens), ("chunks", tokens, longer than) ----
    def _wanted(self, key) -> bool:
        return key[0] != "chunks" or self.max_q_len > key[2]

    def _room(self, key) -> int:
        """Most 32-bit integers that the list takes."""
        n = sum(-(-x // (self._half(key) if key[0] == "halves" else key[1])) for x in self.seq_lens)
        return 4 * n if key[0] in ("tiles", "halves") else 2 * n + 2 * self.n_seqs + 1

    def _half(self, key) -> int:
        """Tokens of a tile of ("halves", tokens, CTAs a tile): half as many where a CTA for each of those has an SM to itself."""
        half = key[1] // 2
        return half if half and sum(-(-x // half) for x in self.seq_lens) * key[2] <= sm_count() else key[1]

    def _write(self, key, at: int):
        """The list at address ``at``: (integers, what ``_views`` has to know of it)."""
        if key[0] in ("tiles", "halves"):
            tokens, longer = (key[1], key[2]) if key[0] == "tiles" else (self._half(key), 0)
            n = steps().lgml_steps_tiles(at, self.n_seqs, self._lens, self._pos0, tokens, longer)
            return 4 * n, n
        reqs = c_int64()
        n = steps().lgml_steps_pieces(at, self.n_seqs, self._lens, key[1], key[2] if key[0] == "chunks" else -1, byref(reqs))
        return 2 * n + reqs.value + 1 + (reqs.value if key[0] == "chunks" else 0), (n, reqs.value)

    def _views(self, key, flat, shape):
        if key[0] in ("tiles", "halves"):
            return flat.view(-1, 4)
        n, reqs = shape
        rows, first = flat[:2 * n].view(-1, 2), flat[2 * n:2 * n + reqs + 1]
        return (rows, first) if key[0] == "pieces" else ScanChunks(rows, first, flat[2 * n + reqs + 1:], key[2], reqs < self.n_seqs, key[1])

    def _list(self, key, remember: bool = True):
        cached = self._tiles.get(key)
        if cached is None:
            if remember and self._lists is not None and len(self._lists) < self.MAX_LISTS:
                self._lists[key] = None
            arr = np.empty(self._room(key), dtype=np.int32)
            n, shape = self._write(key, arr.ctypes.data)
            cached = self._tiles[key] = self._views(key, self._to_device(arr[:n]), shape)
        return cached

    def attention_tiles(self, tile_tokens: int, longer_than: int = 0, remember: bool = True) -> torch.Tensor:
        """The new tokens cut into tiles of at most ``tile_tokens`` consecutive tokens of one
        request, for the prefill attention kernel: int32 [n_tiles, 4] on the device, rows
        (request row, first token row, tokens, 0), the tile with the most keys to visit first:
        the kernel starts its CTAs in this order, and a long tile that starts last would run on
        alone at the end.  Only of requests that bring more than ``longer_than`` tokens.  Made once per tile size (``remember``: for later
        steps of the model too).  (What comes fourth in a row has done its part when they are sorted.)"""
        return self._list(("tiles", tile_tokens, longer_than), remember)

    def twin_tiles(self, tile_tokens: int, ctas: int) -> torch.Tensor:
        """Tiles for the attention kernel that takes two tiles of rows a CTA, ``ctas`` CTAs each: of ``tile_tokens`` tokens, or of half as many, one
        tile of rows, where each such CTA has an SM to itself (the same bits; 16 heads on 4 of 128: 512 tokens behind 1,024 28.2 us in 32 CTAs
        and 23.6 in 64, 488 and 512 tokens 26.3 in 64 and 22.7 in 128, 252 CTAs of a quarter 35; 32 on 8: 512 tokens 17.3 and 14.5, 1,024
        tokens 26.7 in 128 CTAs and 28.0 in 256)."""
        return self._list(("halves", tile_tokens, ctas))

    def tiles_and_short(self, tile_tokens: int, limit, rule):
        """The step's requests in two: (tiles as ``attention_tiles`` of those that bring more than ``limit(seq_lens)`` tokens, the rows of the
        others' tokens, int32 on the device, the longest context among the others).  No tiles: None, and no rows either, they are all.  No
        others: None.  Made once per tile size and ``rule``, which stands for ``limit``."""
        key = ("short", tile_tokens, rule)
        cached = self._tiles.get(key)
        if cached is None:
            up_to = limit(self.seq_lens)
            lens = np.asarray(self.seq_lens, dtype=np.int64)
            rows = np.nonzero(np.repeat(lens <= up_to, lens))[0]
            longest = max((k for k, n in zip(self.kv_lens, self.seq_lens) if n <= up_to), default=0)
            if rows.size == self.n_tokens:
                cached = (None, None, longest)
            else:
                cached = (self.attention_tiles(tile_tokens, up_to if rows.size else 0, remember=False), self._to_device(rows.astype(np.int32)) if rows.size else None, longest)
            self._tiles[key] = cached
        return cached

    def _to_device(self, arr: np.ndarray) -> torch.Tensor:
        """A small int32 list of this step on the device, through the rest of the step's staging buffer when there
        is room (no copy then has to wait for pageable memory)."""
        n_ints = arr.size
        dev = self.token_ids.device
        if self._pinned is not None and self._pinned.numel() >= self._pinned_used + n_ints:
            stage = self._pinned[self._pinned_used:self._pinned_used + n_ints]
            self._pinned_used += n_ints
            stage.numpy()[:] = arr.reshape(-1)
            out = torch.empty(n_ints, dtype=torch.int32, device=dev)
            out.copy_(stage, non_blocking=True)
            if self.after_staged_copy is not None:
                self.after_staged_copy()
            return out
        return torch.from_numpy(np.ascontiguousarray(arr.reshape(-1), dtype=np.int32)).to(dev)

    def scan_pieces(self, piece_tokens: int):
        """Every request's tokens of this step cut into pieces of at most ``piece_tokens`` consecutive tokens, for a
        recurrence that runs the pieces side by side: (int32 [n_pieces, 2] rows [first token row, the row past the
        last), a request's pieces in a row; int32 [requests + 1], the first piece of every request).  Made once per
        piece size."""
        return self._list(("pieces", piece_tokens))

    def scan_chunks(self, chunk_tokens: int, longer_than: int) -> Optional[ScanChunks]:
        """The long requests of this step in chunks (None when no request brings more than ``longer_than`` tokens), for a
        recurrence that takes those as matrix products and the others token by token.  Made once per chunk size."""
        if self.max_q_len <= longer_than:
            return None
        return self._list(("chunks", chunk_tokens, longer_than))

    @staticmethod
    def buffer_ints(n_tokens: int, n_seqs: int, n_rows: int, table_widths: Sequence[int]) -> int:
        return 3 * n_tokens + (n_seqs + 1) + 3 * n_seqs + max(n_rows, 1) + n_seqs * sum(table_widths)

    def cache_view(self, owner: int, writable: bool = True) -> CacheView:
        """The cache of schedule entry ``owner`` as this batch's requests see it."""
        return cache_view_of(self.cache_manager, owner, self.block_tables, writable)
