"""A search does not return hits chosen by a prefilter that gave up a wait
(host side: the count of failures is a stand-in)."""
import importlib

import pytest
import torch

from sseqs_b200 import conv

M = importlib.import_module("sseqs_b200.msa")


@pytest.fixture
def count(monkeypatch):
    """A settable stand-in for the device's count of failures."""
    box = {"n": 0}

    class Stream:
        def synchronize(self):
            box["waits"] = box.get("waits", 0) + 1

    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream())
    monkeypatch.setattr(conv, "_copy_failures", lambda: torch.tensor([box["n"]]), raising=False)
    monkeypatch.setattr(conv, "_failures_seen", {}, raising=False)
    monkeypatch.setattr(conv, "prefilter_luts", lambda *a, **k: None)
    return box


class _Db:
    device = "cpu"

    class _B:
        maxlen = 10

    batches = [_B(), _B()]


def _search(monkeypatch, on_batch, **kw):
    monkeypatch.setattr(M, "search_batch", lambda *a, **k: on_batch(a[3]))
    return M.search(["MKT"], _Db(), **kw)


def test_a_failed_prefilter_raises_once(count, monkeypatch):
    def fails(bi):
        count["n"] += bi
    with pytest.raises(RuntimeError, match="prefilter"):
        _search(monkeypatch, fails)
    assert _search(monkeypatch, lambda bi: None) == [[]]      # an older failure is not this one's
    with pytest.raises(RuntimeError, match="prefilter"):
        _search(monkeypatch, fails)


def test_the_count_is_read_only_after_a_wait(count, monkeypatch):
    """Hits that were read waited for the copy queued before them; a search
    without hits waits itself."""
    _search(monkeypatch, lambda bi: None)
    assert count["waits"] == 1
    monkeypatch.setattr(M, "rank_hits", lambda *a: [("hit",)])
    _search(monkeypatch, lambda bi: None)
    assert count["waits"] == 1


def test_without_a_prefilter_nothing_is_asked(count, monkeypatch):
    monkeypatch.setattr(conv, "_copy_failures", lambda: 1 / 0, raising=False)
    assert _search(monkeypatch, lambda bi: None, top_fft=1) == [[]]


def test_searches_at_the_same_time_all_see_a_failure(count):
    a, b = conv.FailureWatch(), conv.FailureWatch()
    count["n"] = 3
    for w in (b, a):
        w.queue()
        with pytest.raises(RuntimeError):
            w.check()
    w = conv.FailureWatch()
    w.queue()
    w.check()


@pytest.mark.gpu
def test_the_count_reads_the_same_around_a_search():
    from sseqs_b200 import dbtools
    from sseqs_b200.database import Database
    q = dbtools.random_query(200, 5)
    chunks = dbtools.synthetic_db([q], 4000, 0.01, (0.2, 0.95), seed=5, device="cuda",
                                  chunk_bytes=800_000).chunks
    db = Database(chunks[:1], bs=800_000)
    before = conv._copy_failures()
    rows = M.search(q, db, top_fft=20, top_sw=2)[0]
    after = conv._copy_failures()
    torch.cuda.synchronize()
    assert len(rows) > 0 and before.item() == after.item() == 0
