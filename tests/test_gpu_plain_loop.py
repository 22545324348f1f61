"""The whole per-iteration loop (one launch per iteration) against the per-iteration
calls: selections, support vectors and the state it hands over, for whole runs and
prefixes, candidate counts around a CTA's chunk of 256 and lists around the head of 8."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver
from minimumcyclebasis_gb300._native import MCBError

pytestmark = pytest.mark.gpu


def lists(N, K, mean, seed):
    rng = np.random.default_rng(seed)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(mean))) for _ in range(K)]
    rows += [np.array([j]) for j in rng.permutation(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("N,K,mean", [(1, 0, 1), (2, 254, 1), (64, 192, 7), (65, 192, 8), (130, 2000, 20), (257, 256, 3)])
@pytest.mark.parametrize("part", [1.0, 0.5])
def test_loop_equals_the_calls(N, K, mean, part):
    iters = max(1, int(N * part))
    s = Solver(N, *lists(N, K, mean, N + K))
    want = []
    for e in range(iters):
        want.append(s.select(e))
        s.update(e)
    rows = [s.support_vector(j) for j in range(N)]
    total = s.results(iters)[1]
    s.reset()
    s.run_plain(iters)
    got, tot = s.results(iters)
    assert got.tolist() == want and tot == total
    assert all(np.array_equal(s.support_vector(j), rows[j]) for j in range(N))
    if iters < N:  # the calls go on from where the loop stopped
        a = s.select(iters)
        s.update(iters)
        s.reset()
        s.run(iters + 1)
        assert s.results(iters + 1)[0][iters] == a
    s.close()


def test_no_candidate_is_reported():
    s = Solver(3, np.array([1, 2], np.int32), np.array([0, 1, 2], np.int64), np.array([0, 2], np.int32))
    s.run_plain()
    with pytest.raises(MCBError):
        s.results()
    s.close()
