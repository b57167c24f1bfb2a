"""The tensor-core prefilter at the edges of its groups, stages and passes.

Tolerance: both factors of every product are rounded to fp16 (2^-11 each), the
products are summed in fp32 (at most 4 * 2048 terms, 2^-24 each) and the score
is rounded to fp16, so a score may be off by (2^-10 + 2^-11) times the sum of
the products' magnitudes, plus 2^-11 of itself.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
AA = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", np.uint8)


def _segments(lens, rng, letters):
    parts = [rng.choice(letters, n) for n in lens]
    buf = np.concatenate([np.append(p, 64).astype(np.uint8) for p in parts])
    lens = np.asarray(lens, np.int64)
    return buf, np.cumsum(lens + 1) - (lens + 1), lens


def _scores(query, buf, off, lens, n, k, shift=0):
    from sseqs_b200 import conv
    dev = torch.from_numpy(np.concatenate([np.zeros(shift, np.uint8), buf])).cuda()[shift:]
    luts = conv.prefilter_luts(query, k)
    return conv.prefilter_scores(luts, dev, torch.from_numpy(off).cuda(),
                                 torch.from_numpy(lens.astype(np.int32)).cuda(), lens.size, n, k)


@pytest.mark.parametrize("n,Lq,k,count,shift", [
    (64, 1, 4, 3, 0), (64, 64, 4, 129, 1), (128, 33, 1, 128, 7), (256, 200, 2, 300, 31),
    (512, 512, 4, 140, 16), (1024, 16, 4, 127, 3), (1024, 497, 3, 260, 5), (1024, 1023, 4, 40, 9),
    (1024, 1024, 4, 30, 0), (2048, 60, 4, 20, 2), (2048, 1025, 4, 24, 11), (2048, 2048, 4, 16, 30),
])
def test_scores_at_group_edges(n, Lq, k, count, shift):
    rng = np.random.default_rng(n + Lq + k)
    edge = [0, 1, 2, 31, 32, 33, 63, n - 1, n, max(0, n - Lq), max(0, n - Lq + 1), n // 2]
    lens = (edge + list(rng.integers(0, n + 1, max(0, count - len(edge)))))[:count]
    letters = np.concatenate([AA, np.frombuffer(b"XBZ-*xa_", np.uint8), [200, 0, 63]]).astype(np.uint8)
    buf, off, lens = _segments(lens, rng, letters)
    query = rng.choice(AA, Lq).tobytes().decode()
    got = _scores(query, buf, off, lens, n, k, shift).float().cpu().numpy()
    A, B = O.prefilter_luts(query, k)
    exp = O.prefilter_scores(query, A, B, buf, off, lens, n, k)
    size = O.prefilter_scores(query, np.abs(A), np.abs(B), buf, off, lens, n, k)
    tol = (2.0 ** -10 + 2.0 ** -11) * np.abs(size) + 2.0 ** -11 * np.abs(exp) + 1e-6
    assert (np.abs(got - exp) <= tol).all(), np.max(np.abs(got - exp) / tol)


def test_scores_do_not_depend_on_the_grouping():
    """A call long enough for a second window of segments per CTA scores every
    segment as calls on parts of it do."""
    rng = np.random.default_rng(3)
    count = 148 * 4096 + 5000
    lens = rng.integers(0, 9, count)
    buf = rng.choice(AA, int((lens + 1).sum()))
    off = np.cumsum(lens + 1) - (lens + 1)
    buf[off + lens] = 64
    query = rng.choice(AA, 50).tobytes().decode()
    all_ = _scores(query, buf, off, lens, 64, 4).cpu().numpy()
    for lo, hi in ((0, 777), (300_000, 310_001), (count - 4999, count)):
        part = _scores(query, buf, off[lo:hi], lens[lo:hi], 64, 4).cpu().numpy()
        np.testing.assert_array_equal(all_[lo:hi].view(np.uint16), part.view(np.uint16))
