"""What the autotuner times (host side, with stand-ins for the launches)."""
import importlib
import types

import pytest
import torch

from sseqs_b200 import batched, select, tune

sw = importlib.import_module("sseqs_b200.sw")


class _Event:
    def __init__(self, **kw):
        pass

    def record(self):
        pass

    def elapsed_time(self, other):
        return 1.0


@pytest.fixture
def scans(monkeypatch):
    """Orders that the timed scans were given; no kernel runs, nothing is set."""
    seen = []

    def scan(*args, order=None, **kw):
        seen.append(order)

    monkeypatch.setattr(sw, "sw_scan", scan)
    monkeypatch.setattr(sw, "sw_scan_both", scan)
    monkeypatch.setattr(batched, "sw_scan_queries", scan)
    monkeypatch.setattr(select, "length_order",
                        lambda delim, n, good_idx=None, g0=0: ("order of", n, g0))
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    monkeypatch.setattr(tune, "set_variant", lambda *a: None)
    monkeypatch.setattr(tune, "get_variant", lambda *a: tune.BY_SIZE)
    monkeypatch.setattr(tune, "_keep", lambda *a: None)
    monkeypatch.setattr(tune, "set_query_pairing", lambda *a: None)
    monkeypatch.setattr(tune, "has_wide", lambda *a: True)
    monkeypatch.setattr(tune, "_chosen", {})
    return seen


def _batch(n, order="whole"):
    a = torch.zeros(1, dtype=torch.uint8)
    return types.SimpleNamespace(n_segments=n + 2, order=order, ascii=a, delim=a)


@pytest.mark.parametrize("run", [tune.autotune, tune.autotune_pairing])
@pytest.mark.parametrize("n,want", [(500, "whole"), (400, "whole"), (501, ("order of", 500, 1))])
def test_samples_are_scanned_in_the_order_of_a_search(run, n, want, scans):
    """A sample of a larger batch gets an order of its own, as the search of that
    batch takes its targets ordered too."""
    run([150], _batch(n), max_segments=500, reps=1)
    assert scans and all(o == want for o in scans)


@pytest.mark.parametrize("run", [tune.autotune, tune.autotune_pairing])
def test_a_batch_without_an_order_is_timed_without(run, scans):
    run([150], _batch(900, None), max_segments=500, reps=1)
    assert scans and all(o is None for o in scans)


def test_a_choice_holds_for_launches_like_its_sample(monkeypatch):
    """What a sample of n targets (of all queries) showed is kept for launches
    of at least n / 2, and nothing stays set for the others."""
    kept, unset = [], []
    L = types.SimpleNamespace(sseqs_sw_tune_variant=lambda *a: kept.append(a) or 0,
                              sseqs_sw_set_variant=lambda *a: unset.append(a) or 0)
    monkeypatch.setattr(tune, "lib", lambda: L)
    times = iter([2.0, 1.0, 1.0, 2.0, 3.0, 1.0])
    monkeypatch.setattr(tune, "_time", lambda *a: next(times))
    monkeypatch.setattr(tune, "has_wide", lambda *a: True)
    monkeypatch.setattr(tune, "_chosen", {})
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self: self)
    assert tune.autotune([150], _batch(1000)) == {("linear", 5): 1, ("affine", 5): 0,
                                                  ("both", 5): 1}
    assert kept == [(0, 5, 1, 500), (1, 5, 0, 500), (2, 5, 1, 500)]
    last = {m: w for m, t, w in unset}
    assert last == {0: tune.BY_SIZE, 1: tune.BY_SIZE, 2: tune.BY_SIZE}
