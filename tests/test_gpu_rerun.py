"""Blocked runs on one handle with no reset between: each starts from the unit vectors and
from empty lists, so it selects what the per-iteration form selects on a fresh handle,
with that total, behind short runs, whole ones, tuning and calls of the other form."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver

pytestmark = pytest.mark.gpu


def lists(N, K, mean, seed):
    rng = np.random.default_rng(seed)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(mean))) for _ in range(K)]
    rows += [np.array([j]) for j in rng.permutation(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("N,K,mean", [(1, 3, 1), (130, 300, 5), (200, 1500, 100), (512, 3000, 3), (512, 3000, 250)])
@pytest.mark.parametrize("first", [1, 64, 128, -1])
def test_a_run_behind_other_runs(N, K, mean, first):
    s = Solver(N, *lists(N, K, mean, N + K))
    s.run_plain()
    want, total = s.results()
    for _ in range(4):  # behind the other form, then behind its own
        s.run(first)
        got = s.results()[0] if first < 0 else s.results(min(first, N))[0]
        assert np.array_equal(got, want[:len(got)])
    s.run()
    got, tot = s.results()
    assert np.array_equal(got, want) and tot == total
    s.tune()
    s.run()
    got, tot = s.results()
    assert np.array_equal(got, want) and tot == total
    s.reset()
    for e in range(min(N, 3)):
        s.select(e)
        s.update(e)
    s.run()
    got, tot = s.results()
    assert np.array_equal(got, want) and tot == total
    s.run_graph(min(N, 70))
    s.run()
    got, tot = s.results()
    assert np.array_equal(got, want) and tot == total
    s.close()
