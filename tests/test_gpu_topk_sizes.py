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
