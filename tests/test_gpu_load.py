"""Loading a batch: decode with delimiters noted on the way, and the segment
table, against numpy restatements (exact)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _symbols(kind, n, rng):
    a = rng.integers(65, 96, n).astype(np.uint8)
    if kind == "ends":                 # '@' here and there, first and last symbol a residue
        a[rng.integers(0, n, max(1, n // 40))] = 64
        a[0] = a[-1] = 65
    elif kind == "padded":             # runs of '@', leading and trailing ones
        a[rng.integers(0, n, max(1, n // 5))] = 64
        a[:3] = 64
        a[-(n // 3):] = 64
    elif kind == "one":                # a single residue
        a[:] = 64
        a[n // 2] = 70
    elif kind == "none":
        pass
    elif kind == "blank":
        a[:] = 64
    return a


@pytest.mark.parametrize("kind", ["ends", "padded", "one", "none", "blank"])
@pytest.mark.parametrize("bs", [5, 20, 40, 5120, 5125, 10_240, 500_005])
def test_batches_match_restatement(kind, bs):
    from sseqs_b200.database import Database
    rng = np.random.default_rng(bs)
    n = bs * 8 // 5
    raw = [_symbols(kind, n, rng) for _ in range(2)]
    chunk = np.concatenate([O.xbit_compress(a) for a in raw])
    db = Database([torch.from_numpy(chunk)], bs=bs)
    want = []
    for j, a in enumerate(raw):
        live = np.flatnonzero(a != 64)
        if live.size:
            want.append((j, a[:min(n, live[-1] + 2)]))
    assert [b.index for b in db.batches] == [j for j, _ in want]
    for b, (j, a) in zip(db.batches, want):
        seg = O.segment(a)
        np.testing.assert_array_equal(b.ascii.cpu().numpy(), a)
        np.testing.assert_array_equal(b.delim.cpu().numpy(), np.flatnonzero(a == 64))
        np.testing.assert_array_equal(b.lengths.cpu().numpy(), seg["lengths"])
        np.testing.assert_array_equal(b.offsets.cpu().numpy(), seg["offsets"])
        d = np.flatnonzero(a == 64)
        allseg = np.diff(np.concatenate([[-1], d, [a.size] if a[-1] != 64 else []])) - 1
        np.testing.assert_array_equal(b.seg_index.cpu().numpy(), np.flatnonzero(allseg))
        assert (b.maxlen, b.n_segments, b.n_residues) == (
            seg["lengths"].max(), seg["lengths"].size, seg["lengths"].sum())
    assert db.n_residues == sum(int((a != 64).sum()) for _, a in want)


@pytest.mark.parametrize("form", ["strided", "column", "rows", "host"])
def test_views_of_a_chunk_load_as_its_contiguous_copy(form):
    from sseqs_b200.database import Database
    rng = np.random.default_rng(3)
    bs = 5120
    chunk = torch.from_numpy(np.concatenate(
        [O.xbit_compress(_symbols("ends", bs * 8 // 5, rng)) for _ in range(2)])).cuda()
    wide = torch.full((chunk.numel(), 3), 0xff, dtype=torch.uint8, device="cuda")
    wide[:, 1] = chunk
    view = {"strided": wide.reshape(-1)[1::3], "column": wide[:, 1], "rows": chunk.view(2, -1),
            "host": chunk}[form]
    want = Database([chunk], bs=bs).batches
    got = Database([view], bs=bs, device="cpu" if form == "host" else "cuda").batches
    assert len(got) == len(want) == 2
    for g, w in zip(got, want):
        assert (g.maxlen, g.n_segments, g.n_residues) == (w.maxlen, w.n_segments, w.n_residues)
        for f in ("ascii", "delim", "seg_index", "lengths", "offsets"):
            assert torch.equal(getattr(g, f), getattr(w, f)), f


def test_an_expanded_chunk_loads_as_its_contiguous_copy():
    from sseqs_b200.database import Database
    one = torch.full((1,), 0b00100001, dtype=torch.uint8, device="cuda")
    bs = 5120
    got, want = (Database([c], bs=bs).batches[0] for c in
                 (one.expand(bs), one.expand(bs).contiguous()))
    assert torch.equal(got.ascii, want.ascii) and torch.equal(got.delim, want.delim)
