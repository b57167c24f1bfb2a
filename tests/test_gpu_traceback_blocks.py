"""The traceback at the edges of its row blocks, phases and sweeps (exact)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import rand_seq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lq", [1, 3, 4, 5, 127, 128, 129, 256, 257, 513, 1023, 1024, 1025, 1153,
                                2048])
def test_alignments_at_block_edges(Lq):
    from sseqs_b200.sw import backtrack
    rng = np.random.default_rng(Lq)
    query = rand_seq(rng, Lq)
    targets = [rand_seq(rng, n) for n in (1, 15, 16, 17, 31, 32, 33, 34, 63, 64, 65, 97, 129, 500)]
    # repeats of the query's pieces: ties of the best score, long gaps, both edges
    targets += [query, query + query, query[:64] * 3, query[Lq // 2:] + query[:Lq // 2],
                query[:Lq // 3] + rand_seq(rng, 40) + query[Lq // 3:], "W" * 70, "X" * 33, ""]
    for gaps in ((11, 1), (0, 0), (5, 2)):
        got = backtrack(query, targets, *gaps).to_dicts()
        _, exp = O.sw_affine_backtrack(query, targets, *gaps)
        assert got == exp, gaps


def test_matrix_at_block_edges():
    """M(i, j) = s(i, j) + H(i - 1, j - 1), from a plain restatement."""
    from sseqs_b200.sw import backtrack
    rng = np.random.default_rng(0)
    query = rand_seq(rng, 140)
    targets = [rand_seq(rng, 70), query[60:135]]
    M = backtrack(query, targets, with_matrix=True).m_full.cpu().numpy()
    for b, t in enumerate(targets):
        H = np.zeros((len(query) + 1, len(t) + 1), np.int64)
        X, Y = np.full_like(H, -16384), np.full_like(H, -16384)
        for i in range(1, len(query) + 1):
            for j in range(1, len(t) + 1):
                s = O.BLOSUM62[O.AA_MAP[query[i - 1]], O.AA_MAP[t[j - 1]]]
                m = s + H[i - 1, j - 1]
                X[i, j] = max(H[i - 1, j] - 11, X[i - 1, j] - 1)
                Y[i, j] = max(H[i, j - 1] - 11, Y[i, j - 1] - 1)
                H[i, j] = max(0, m, X[i, j], Y[i, j])
                assert M[b, i, j] == m


def _gotoh(query, target, go, ge):
    """Best score and alignment of one pair in 64 bits, row by row: the first best
    cell in query-major order, states in the order M, Ix, Iy."""
    n, m = len(query), len(target)
    H = np.zeros((n + 1, m + 1), np.int64)
    M, X, Y = (np.full((n + 1, m + 1), -16384, np.int64) for _ in range(3))
    for i in range(1, n + 1):
        for j in range(1, m + 1):
            s = O.BLOSUM62[O.AA_MAP[query[i - 1]], O.AA_MAP[target[j - 1]]]
            M[i, j] = s + H[i - 1, j - 1]
            X[i, j] = max(H[i - 1, j] - go, X[i - 1, j] - ge)
            Y[i, j] = max(H[i, j - 1] - go, Y[i, j - 1] - ge)
            H[i, j] = max(0, M[i, j], X[i, j], Y[i, j])
    best = int(H.max())
    i, j = np.unravel_index(int(H.argmax()), H.shape)
    qa, ta = [], []
    while i > 0 and j > 0 and H[i, j] > 0:
        if H[i, j] == M[i, j]:
            qa.append(query[i - 1])
            ta.append(target[j - 1])
            i, j = i - 1, j - 1
        elif H[i, j] == X[i, j]:
            qa.append(query[i - 1])
            ta.append("-")
            i -= 1
        else:
            qa.append("-")
            ta.append(target[j - 1])
            j -= 1
    return best, "".join(reversed(qa)), "".join(reversed(ta))


@pytest.mark.parametrize("gaps", [
    (-1, -1), (11, -40), (-300_000, 5), (-210_000, -1), (-240_000, -240_000),
    (-3_000_000, -3_000_000), (7, -3_000_000), (-3_000_000, 2), (1 << 27, -200_000),
    (1 << 30, -6_000_000), (1 << 27, 1 << 27), (1 << 30, 1 << 30), (-2_000_000, 1 << 30)])
def test_gap_costs_of_any_size_and_sign(gaps):
    """Gaps that are bonuses, up to sums near the 32-bit range, and costs past
    every score: each pair as a 64-bit restatement aligns it."""
    from sseqs_b200.sw import backtrack
    rng = np.random.default_rng(5)
    query = rand_seq(rng, 133)
    targets = [rand_seq(rng, 150), query[20:110], rand_seq(rng, 1), rand_seq(rng, 33) + query[:60]]
    res = backtrack(query, targets, *gaps)
    best = res.best.cpu().tolist()
    for t, b, got in zip(targets, best, res.to_dicts()):
        exp = _gotoh(query, t, *gaps)
        assert (b, got["q_aligned"], got["t_aligned"]) == exp
