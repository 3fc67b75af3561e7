"""The span tables of a ragged prefill pass: what the gated-delta-rule and attention kernels look their work up in."""

from __future__ import annotations

from dataclasses import dataclass

import numpy as np
import torch

from ..utils.upload import to_device

CHUNK = 64  # rows per chunk of the gated-delta-rule kernels
FEW = 6  # up to this many spans a loop over them takes less time than the same in whole arrays


def parts_of(starts, rows: int) -> int:
    """How many parts of ``rows`` rows the spans make."""
    return sum((b - a + rows - 1) // rows for a, b in zip(starts, starts[1:]))


def fill_tables(starts, chunks: np.ndarray, per_span: np.ndarray, tiles: np.ndarray, tile_rows: int | None) -> None:
    """``chunks [n, 4]``: (span, first row, rows, is the span's first chunk). ``per_span [spans, 2]``: (first chunk, chunks).
    ``tiles [n, 4]``: (span, first row in the span, the span's first row, the span's rows) per query tile of ``tile_rows``
    positions. All int32, of the sizes that ``parts_of`` gives."""
    if len(starts) <= FEW + 1:
        c = t = 0
        for i, (a, b) in enumerate(zip(starts, starts[1:])):
            k = (b - a + CHUNK - 1) // CHUNK
            part = chunks[c:c + k]
            part[:] = (i, 0, CHUNK, 0)
            part[:, 1] = np.arange(a, b, CHUNK)
            if k:
                part[0, 3], part[-1, 2] = 1, b - a - CHUNK * (k - 1)
            per_span[i] = (c, k)
            c += k
            if tile_rows:
                k = (b - a + tile_rows - 1) // tile_rows
                part = tiles[t:t + k]
                part[:] = (i, 0, a, b - a)
                part[:, 1] = np.arange(0, b - a, tile_rows)
                t += k
        return
    st = np.asarray(starts, dtype=np.int64)
    lens = st[1:] - st[:-1]
    for out, rows in ((chunks, CHUNK), (tiles, tile_rows)):
        if rows:
            per = (lens + (rows - 1)) // rows
            first = per.cumsum() - per
            span = np.repeat(np.arange(len(per)), per)
            at = rows * (np.arange(len(span)) - first[span])
            out[:, 0] = span
            if out is chunks:
                out[:, 1], out[:, 2], out[:, 3] = st[span] + at, np.minimum(rows, lens[span] - at), at == 0
                per_span[:, 0], per_span[:, 1] = first, per
            else:
                out[:, 1], out[:, 2], out[:, 3] = at, st[span], lens[span]


@dataclass
class SpanTables:
    """Tables on the device, with the host lists that they were built from. ``gdn`` and ``flash`` are what
    ``cuda_ops.gdn_prefill`` and ``cuda_ops.attention`` take as ``meta``."""

    starts: list[int]
    slots: list[int]
    pos0: list[int]
    gdn: tuple
    flash: tuple | None

    def of(self, starts, slots, pos0, tile_rows: int | None) -> bool:
        return (self.starts == starts and self.slots == slots and self.pos0 == pos0
                and (tile_rows is None or (self.flash is not None and self.flash[0] == tile_rows)))


def words(starts, tile_rows: int | None) -> list[int]:
    """The int32 words of the tables, in the order of ``write`` and ``tables``: chunks, tiles, per span, starts, slots, pos0.
    Kernels read the first two 16 bytes and the third 8 bytes at a time."""
    n = len(starts) - 1
    return [4 * parts_of(starts, CHUNK), 4 * parts_of(starts, tile_rows) if tile_rows else 0, 2 * n, n + 1, n, n]


def write(parts, starts, slots, pos0, tile_rows: int | None) -> None:
    chunks, tiles, per_span = parts[0].reshape(-1, 4), parts[1].reshape(-1, 4), parts[2].reshape(-1, 2)
    fill_tables(starts, chunks, per_span, tiles, tile_rows)
    parts[3][:], parts[4][:], parts[5][:] = starts, slots, pos0


def tables(parts, seq: torch.Tensor, starts, slots, pos0, tile_rows: int | None) -> SpanTables:
    """``parts``: the words on the device; ``seq``: the span of every row."""
    chunks, tiles, per_span, st, sl, p0 = parts
    return SpanTables(list(starts), list(slots), list(pos0), (len(slots), len(chunks) // 4, chunks, per_span, seq, st, sl),
                      (tile_rows, len(tiles) // 4, tiles, p0) if tile_rows else None)


def span_tables(starts, slots, pos0, tile_rows: int | None, device: torch.device) -> SpanTables:
    """The tables on ``device``, by one copy that is complete on return."""
    sizes = [*words(starts, tile_rows), starts[-1]]
    host = torch.empty(sum(sizes), dtype=torch.int32, pin_memory=device.type == "cuda")
    parts = np.split(host.numpy(), np.cumsum(sizes)[:-1])
    write(parts[:6], starts, slots, pos0, tile_rows)
    for i, (a, b) in enumerate(zip(starts, starts[1:])):
        parts[6][a:b] = i
    *parts, seq = to_device(host, device).split(sizes)
    return tables(parts, seq, starts, slots, pos0, tile_rows)
