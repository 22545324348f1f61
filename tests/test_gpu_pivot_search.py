"""The blocked run's pivot search where its windows, lists and merges can go wrong:
many nonzero rows per window, one tile and many, pivots far behind the tiles of the W
pass, blocks narrower than 64, and a candidate set that does not span.  Against the
per-iteration form, which has no pivot search."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver
from minimumcyclebasis_gb300._native import MCBError

pytestmark = pytest.mark.gpu


def solver(N, rows):
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return Solver(N, np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32))


def same(s):
    s.run_plain()
    want, total = s.results()
    for _ in range(2):
        s.reset()
        s.run()
        got, tot = s.results()
        assert np.array_equal(got, want) and tot == total
    s.close()


@pytest.mark.parametrize("N,K,mean", [(63, 1025, 20), (64, 9000, 30), (128, 40000, 60), (190, 6000, 90)])
def test_dense_rows(N, K, mean):
    rng = np.random.default_rng(N + K)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(mean))) for _ in range(K)]
    same(solver(N, rows + [np.array([j]) for j in range(N)]))


@pytest.mark.parametrize("N,gap,every", [(100, 400000, 1), (130, 1500, 50), (260, 2000, 7), (65, 170000, 32)])
def test_pivots_far_apart(N, gap, every):
    # runs of `gap` candidates that are already spanned between every `every` new ones
    rng = np.random.default_rng(gap)
    order, rows = rng.permutation(N), []
    for i, j in enumerate(order):
        if i % every == every - 1 and (i // every) % 20 == 1:
            rows += [np.sort(order[[i - 1, max(i - 2, 0)]]) if i > 2 else order[[i - 1]]] * gap
        rows.append(np.unique(np.append(order[rng.integers(0, i + 1, 2)], j)))
    same(solver(N, rows))


def test_candidates_that_do_not_span():
    rows = [np.array([j]) for j in range(200) if j != 150] * 3
    s = solver(200, rows)
    s.run()
    with pytest.raises(MCBError):
        s.results()
    s.close()
