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
