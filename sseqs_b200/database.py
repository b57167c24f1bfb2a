"""HBM-resident sequence database.

The reference streams 1e9-byte .xbit chunks from pinned host RAM to the GPU
on every search and re-derives the segment structure of every batch
(sseqs/msa.py:13-64, :196-267).  Here a database is decoded once: for every
batch (``bs`` packed bytes of a chunk, decoded to ``bs*8/5`` symbols exactly as
sseqs/msa.py:217-220 slices it) the decoded bytes, the '@' positions and the
non-empty segment table stay resident in HBM, so a search touches no host
memory except its own results.

Trailing '@' padding of a batch (the zero fill of a chunk) is trimmed after
the first delimiter: padding only forms empty segments, which the reference
drops (sseqs/msa.py:253), after every real segment, so no index or result
changes.  A batch that is padding only is skipped (the reference fails on it
at sseqs/msa.py:261).
"""
from __future__ import annotations

import math
import os
from dataclasses import dataclass

import numpy as np
import torch

from . import select
from ._lib import check, lib, ptr, stream_ptr, workspace

CHUNK_BYTES = 1_000_000_000
DECODE_ON = "cuda"         # where chunks are decoded: the current CUDA device


@dataclass
class Batch:
    chunk: int
    index: int                 # batch number inside its chunk
    ascii: torch.Tensor        # decoded bytes, trimmed (device)
    n_symbols: int             # untrimmed batch size (bs*8/5)
    delim: torch.Tensor        # '@' positions, int32 (device)
    seg_index: torch.Tensor    # non-empty segment k of each filtered index
    lengths: torch.Tensor      # int32 lengths of the non-empty segments
    offsets: torch.Tensor      # int64 start of each (running sum of length+1)
    maxlen: int
    n_segments: int
    n_residues: int
    # segments 1 .. n_segments-2, the targets of a whole-batch scan, from the
    # longest to the shortest (select.length_order; target t is segment t + 1)
    order: torch.Tensor | None = None


class Database:
    """A list of packed chunks, decoded into resident batches."""

    def __init__(self, chunks, bs: int = CHUNK_BYTES, device="cuda", keep_packed: bool = False):
        self.device = torch.device(device)
        self.bs = int(bs)
        self.batches: list[Batch] = []
        self.packed = [] if keep_packed else None
        self.n_residues = 0
        self.index = None          # sidecar segment index (from_file), if any
        self.n_chunks = 0
        self.add_chunks(chunks)

    def add_chunks(self, chunks) -> None:
        """Decode more packed chunks into resident batches (after the ones
        already loaded), so a large database can be built a part at a time
        without holding all of it packed."""
        for ch in chunks:
            ci = self.n_chunks
            ch = ch if isinstance(ch, torch.Tensor) else torch.from_numpy(np.asarray(ch, np.uint8))
            ch = ch.to(self.device, torch.uint8)
            if ch.numel() % self.bs:
                raise ValueError("chunk size must be a multiple of bs (sseqs/msa.py:216)")
            if self.packed is not None:
                self.packed.append(ch)
            # the kernels take addresses: contiguous bytes on the device whose
            # stream they run on (a strided, expanded or host-held chunk is copied)
            src = ch.to(device=DECODE_ON).contiguous()
            for j in range(ch.numel() // self.bs):
                self._add_batch(ci, j, src)
            self.n_chunks += 1
            del ch, src

    def _add_batch(self, ci, j, ch):
        n_sym = int(self.bs * 8 / 5)
        lo = j * self.bs
        if lo + (5 * n_sym + 7) // 8 > ch.numel():
            raise ValueError("a batch reaches past its chunk")
        L, dev, st = lib(), ch.device, stream_ptr()
        # decode, and note the '@' on the way; one read of (last residue, '@' count)
        # by the host sizes everything else
        full = torch.empty(n_sym, dtype=torch.uint8, device=dev)
        info = torch.empty(5, dtype=torch.int64, device=dev)
        ws = workspace(L.sseqs_decode_scan_workspace_bytes(n_sym), dev)
        check(L.sseqs_decode_scan(ptr(ch), ptr(full), n_sym, lo, ptr(info), ptr(ws), ws.numel(),
                                  st), "decode_scan")
        last, total = info[:2].tolist()
        if last < 0:
            return
        # trimmed after the delimiter that closes the last residue; every
        # symbol past it is '@'
        eff = min(n_sym, last + 2)
        nd, trailing = total - (n_sym - eff), int(last + 1 == n_sym)
        delim = torch.empty(nd, dtype=torch.int32, device=dev)
        check(L.sseqs_decode_scan_delims(n_sym, nd, ptr(delim), ptr(ws), ws.numel(), st),
              "decode_scan_delims")
        seg_index, lengths = (torch.empty(nd + 1, dtype=torch.int32, device=dev)
                              for _ in range(2))
        offsets = torch.empty(nd + 1, dtype=torch.int64, device=dev)
        ws2 = workspace(L.sseqs_segments_workspace_bytes(nd + 1), dev)
        check(L.sseqs_segments(eff, ptr(delim), nd, trailing, ptr(seg_index), ptr(lengths),
                               ptr(offsets), ptr(info[2:]), ptr(ws2), ws2.numel(), st), "segments")
        # the scan order, for the usual batch without empty segments (queued before
        # the read below, after which everything is complete)
        nseg = nd + trailing
        order = select.length_order(delim, nseg - 2, g0=1) if nseg > 2 else None
        # a batch that is nearly full keeps its decoded buffer, a mostly empty
        # one a copy of the part that is used
        ascii = full[:eff] if 16 * (n_sym - eff) <= n_sym else full[:eff].clone()
        m, maxlen, res = info[2:].tolist()
        if m == 0:
            return
        self.n_residues += res
        if m != nseg:
            order = select.length_order(delim, m - 2, g0=1) if m > 2 else None
            torch.cuda.current_stream(dev).synchronize()
        self.batches.append(Batch(ci, j, ascii, n_sym, delim, seg_index[:m], lengths[:m],
                                  offsets[:m], maxlen, m, res, order))

    @classmethod
    def from_file(cls, path: str, chunks: int | None = None, bs: int = CHUNK_BYTES,
                  device="cuda", chunk_bytes: int = CHUNK_BYTES):
        """Read ``chunks`` chunks of ``chunk_bytes`` from an .xbit file
        (sseqs/msa.py:50-55); bytes past the end of the file read as 0.  A
        sidecar segment index next to the file (``dbtools.fasta_to_xbit``)
        is loaded as ``index`` when its chunk size matches."""
        from .dbtools import SeqIndex, index_path
        size = os.path.getsize(path)
        n = math.ceil(size / chunk_bytes) if chunks is None else int(chunks)
        out = []
        with open(path, "rb") as fh:
            for i in range(n):
                buf = np.zeros(chunk_bytes, np.uint8)
                fh.seek(i * chunk_bytes)
                fh.readinto(memoryview(buf))
                out.append(torch.from_numpy(buf))
        db = cls(out, bs=bs, device=device)
        if os.path.exists(index_path(path)):
            idx = SeqIndex.load(index_path(path))
            if idx.chunk_bytes == chunk_bytes:
                db.index = idx
        return db

    def hit_names(self, hits) -> list:
        """FASTA names of ranked hits ((…, batch, segment, …) rows as
        ``msa.search`` returns them): the sequence holding the first byte of
        the hit's window (``offsets[g]`` of its batch, the bytes the hit
        string shows), from the sidecar index; None where a position is not
        inside a sequence."""
        if self.index is None:
            raise ValueError("no sidecar segment index loaded for this database")
        if (self.bs * 8) % 5:
            raise ValueError("batch boundaries fall inside a 5-byte group (bs % 5 != 0)")
        by_batch: dict = {}
        for r, row in enumerate(hits):
            by_batch.setdefault(int(row[1]), []).append((r, int(row[2])))
        names = [None] * len(hits)
        for bi, items in by_batch.items():
            b = self.batches[bi]
            g = torch.tensor([x[1] for x in items], dtype=torch.int64, device=b.offsets.device)
            off = b.offsets.index_select(0, g).cpu().numpy()
            base = b.index * self.bs * 8 // 5
            for (r, _), o in zip(items, off.tolist()):
                k = self.index.locate(b.chunk, base + o)
                names[r] = self.index.names[k] if k >= 0 else None
        return names

    @property
    def n_segments(self) -> int:
        return sum(b.n_segments for b in self.batches)


_default: dict = {}


def default_database(bs: int | None = None) -> Database:
    """The database named by DBPATH / CHUNKS, decoded with batch size ``bs``
    and loaded on first use (sseqs/msa.py:13-25 loads it at import time and
    exits if it is missing)."""
    bs = 50_000_000 if bs is None else int(bs)
    if bs not in _default:
        path = os.environ.get("DBPATH", "uniref_bfd_mgy_cf.xbit")
        chunks = int(os.environ.get("CHUNKS", 4))
        if not os.path.exists(path):
            raise FileNotFoundError(f"Didn't find MSA database at `{path}` (set DBPATH)")
        _default.clear()
        _default[bs] = Database.from_file(path, chunks=chunks, bs=bs)
    return _default[bs]
