"""Top-k at the edges of its one-block and tiled forms (exact)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
SIZES = [2, 31, 33, 1023, 1024, 1025, 2049, 4097, 16383, 16384, 16385, 20_481, 70_001, 700_003]


def _check(v, k):
    from sseqs_b200 import select
    got = select.topk_indices(torch.from_numpy(v).cuda(), k).cpu().numpy()
    exp = np.sort(O.topk_canonical(v.astype(np.float64), k))
    np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["scores", "wide", "equal", "extremes", "half"])
def test_topk_sizes(n, kind):
    rng = np.random.default_rng(n)
    if kind == "scores":
        v = rng.integers(-1, 900, n).astype(np.int32)
    elif kind == "wide":
        v = rng.integers(-2 ** 31, 2 ** 31, n).astype(np.int32)
    elif kind == "equal":
        v = np.full(n, 7, np.int32)
    elif kind == "extremes":
        v = rng.choice(np.array([-2 ** 31, 2 ** 31 - 1, 0, -1], np.int64), n).astype(np.int32)
    else:
        v = (rng.standard_normal(n) * 30).astype(np.float16)
        v[rng.integers(0, n, max(1, n // 50))] = np.float16(np.inf)
        v[rng.integers(0, n, max(1, n // 50))] = np.float16(-np.inf)
    for k in sorted({1, n // 7, n // 2, n - 1} - {0}):
        _check(v, k)


@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1025, 5000, 8191, 8192])
def test_kth_largest_rows(n):
    from sseqs_b200 import _lib
    rng = np.random.default_rng(n)
    rows = np.stack([rng.standard_normal(n) * 100, rng.integers(-3, 4, n), np.full(n, -2.5),
                     np.where(rng.random(n) < 0.5, -np.inf, 1e30)]).astype(np.float32)
    x = torch.from_numpy(rows).cuda()
    out = torch.empty(4, dtype=torch.float32, device="cuda")
    for k in sorted({1, 2, n // 3, n // 2, n - 1, n} - {0, n + 1}):
        if k > n:
            continue
        _lib.check(_lib.lib().sseqs_kth_largest_rows(_lib.ptr(x), 4, n, k, _lib.ptr(out),
                                                     _lib.stream_ptr()))
        np.testing.assert_array_equal(out.cpu().numpy(), -np.sort(-rows, 1)[:, k - 1])
