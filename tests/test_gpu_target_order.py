"""The order in which targets are taken: scores do not depend on it (exact)."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
AA = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", np.uint8)


def _batch(n, seed, lo=0, hi=700):
    rng = np.random.default_rng(seed)
    lens = rng.integers(lo, hi, n)
    lens[rng.integers(0, n, max(1, n // 20))] = 0          # empty windows
    buf = rng.choice(AA, int((lens + 1).sum()))
    buf[np.cumsum(lens + 1) - 1] = 64
    a = torch.from_numpy(buf).cuda()
    return a, torch.from_numpy((np.cumsum(lens + 1) - 1).astype(np.int32)).cuda(), lens


def _query(L, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, 20, (L,), generator=g, dtype=torch.uint8).cuda()


@pytest.mark.parametrize("n", [1, 2, 255, 256, 2047, 2049, 60_001])
@pytest.mark.parametrize("listed", [False, True])
def test_length_order_sorts(n, listed):
    from sseqs_b200 import select
    _, delim, lens = _batch(n + 3, n, hi=2500)
    idx = np.random.default_rng(n).permutation(n + 1)[:n].astype(np.int32) + 1 if listed else None
    t = torch.from_numpy(idx).cuda() if listed else None
    o = select.length_order(delim, n, good_idx=t, g0=1).cpu().numpy()
    np.testing.assert_array_equal(np.sort(o), np.arange(n))
    steps = np.minimum((lens[idx] if listed else lens[1:n + 1])[o] // 8, 255)
    assert (np.diff(steps) <= 0).all()


@pytest.mark.parametrize("Lq", [20, 33, 100, 129, 250, 257, 500, 700, 740, 1000, 1600])
def test_scans_do_not_depend_on_the_order(Lq):
    from sseqs_b200 import select
    sw = importlib.import_module("sseqs_b200.sw")
    batched = importlib.import_module("sseqs_b200.batched")
    tune = importlib.import_module("sseqs_b200.tune")
    n = 3000
    a, d, _ = _batch(n + 2, Lq)
    q = _query(Lq, Lq)
    rng = np.random.default_rng(Lq)
    orders = [select.length_order(d, n, g0=1),
              torch.from_numpy(rng.permutation(n).astype(np.int32)).cuda()]
    idx = torch.from_numpy((rng.permutation(n) + 1).astype(np.int32)).cuda()
    tpt = tune.tpt_of(Lq)
    qs = torch.zeros((3, 2048), dtype=torch.uint8, device="cuda")
    qs[:, :Lq] = torch.stack([_query(Lq, Lq + i) for i in range(3)])
    lens = torch.full((3,), Lq, dtype=torch.int32, device="cuda")
    for tgt in (dict(g0=1, n_targets=n), dict(good_idx=idx)):
        kw = dict(affine=True, skip=1, gap_a=11, gap_b=1, **tgt)
        lin = sw.sw_scan(q, a, d, affine=False, gap_a=-1, **tgt)
        aff = sw.sw_scan(q, a, d, **kw)
        many = batched.sw_scan_queries(qs, lens, tpt, a, d, **kw)
        old = [(m, tune.get_variant(m, tpt)) for m in range(4)]
        pair = tune.get_query_pairing(tpt)
        try:
            for o in orders:
                for wide in (0, 1):
                    for m in range(4):
                        tune.set_variant(m, tpt, wide)
                    assert torch.equal(sw.sw_scan(q, a, d, affine=False, gap_a=-1, order=o, **tgt),
                                       lin)
                    assert torch.equal(sw.sw_scan(q, a, d, order=o, **kw), aff)
                    both = sw.sw_scan_both(q, a, d, order=o, **tgt)
                    assert torch.equal(both[0], lin) and torch.equal(both[1], aff)
                    for on in (False, True):
                        tune.set_query_pairing(tpt, on)
                        got = batched.sw_scan_queries(qs, lens, tpt, a, d, order=o, **kw)
                        assert torch.equal(got[:, :n], many[:, :n])
        finally:
            for m, v in old:
                tune.set_variant(m, tpt, v)
            tune.set_query_pairing(tpt, pair)
    with pytest.raises(ValueError):
        sw.sw_scan(q, a, d, order=orders[0][:-1], **kw)


@pytest.mark.parametrize("Lq", [20, 60, 150, 300, 500, 860])
def test_few_targets_spread_over_blocks(Lq):
    """Launches around a warp's, a block's and an SM round's number of targets
    score as one launch over all of them does."""
    sw = importlib.import_module("sseqs_b200.sw")
    n = 9000
    a, d, _ = _batch(n + 2, Lq + 1, hi=60)
    q = _query(Lq, Lq)
    kw = dict(affine=True, skip=1, gap_a=11, gap_b=1, g0=1)
    aff = sw.sw_scan(q, a, d, n_targets=n, **kw)
    lin = sw.sw_scan(q, a, d, affine=False, gap_a=-1, g0=1, n_targets=n)
    for m in (1, 2, 3, 31, 33, 63, 65, 127, 129, 591, 593, 1183, 1185, 2367, 2369, 4737):
        assert torch.equal(sw.sw_scan(q, a, d, n_targets=m, **kw), aff[:m])
        both = sw.sw_scan_both(q, a, d, g0=1, n_targets=m)
        assert torch.equal(both[0], lin[:m]) and torch.equal(both[1], aff[:m])


@pytest.mark.parametrize("Lq", [20, 160, 250, 500, 700, 900])
@pytest.mark.parametrize("n", [300, 9000, 200_000])
def test_the_layout_by_size_scores_as_each_layout(Lq, n):
    """With none set, few targets, many and a number between (past eight
    lane groups' worth at 200000) score as both layouts do."""
    sw = importlib.import_module("sseqs_b200.sw")
    tune = importlib.import_module("sseqs_b200.tune")
    a, d, _ = _batch(n + 2, Lq + n, hi=30 if n > 9000 else 300)
    q = _query(Lq, Lq)
    tpt = tune.tpt_of(Lq)
    old = [tune.get_variant(m, tpt) for m in range(3)]
    got = []
    try:
        for wide in (tune.BY_SIZE, 0, 1):
            for m in range(3):
                tune.set_variant(m, tpt, wide)
            got.append((sw.sw_scan(q, a, d, affine=False, gap_a=-1, g0=1, n_targets=n),
                        sw.sw_scan(q, a, d, affine=True, skip=1, gap_a=11, gap_b=1, g0=1,
                                   n_targets=n), *sw.sw_scan_both(q, a, d, g0=1, n_targets=n)))
    finally:
        for m, v in enumerate(old):
            tune.set_variant(m, tpt, v)
    for other in got[1:]:
        for x, y in zip(got[0], other):
            assert torch.equal(x, y)


def test_a_tuned_layout_scores_the_same_on_both_sides_of_its_line():
    from sseqs_b200 import _lib
    sw = importlib.import_module("sseqs_b200.sw")
    tune = importlib.import_module("sseqs_b200.tune")
    a, d, _ = _batch(4002, 3)
    q = _query(150, 3)
    old = tune.get_variant(1, 5)
    kw = dict(affine=True, skip=1, gap_a=11, gap_b=1, g0=1)
    try:
        tune.set_variant(1, 5, 0)
        want = sw.sw_scan(q, a, d, n_targets=4000, **kw)
        tune.set_variant(1, 5, tune.BY_SIZE)
        for wide in (0, 1):
            _lib.check(_lib.lib().sseqs_sw_tune_variant(1, 5, wide, 2000))
            for n in (1999, 2000, 4000):
                assert torch.equal(sw.sw_scan(q, a, d, n_targets=n, **kw), want[:n])
    finally:
        _lib.check(_lib.lib().sseqs_sw_tune_variant(1, 5, tune.BY_SIZE, 0))
        tune.set_variant(1, 5, old)
