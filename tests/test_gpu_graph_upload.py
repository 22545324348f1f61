"""The solve's CUDA graph behind an upload whose longest list outgrows the pair buffers the
graph was captured with (list total and counts as before): captured again, it selects
what the per-iteration form selects."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver

pytestmark = pytest.mark.gpu


def lists(N, lengths, seed):
    """One random list per length, then {j} for every coordinate."""
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(N, n, replace=False)) for n in lengths] + [np.array([j]) for j in rng.permutation(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("N,per", [(150, 4), (700, 60)])
def test_graph_behind_longer_lists(N, per):
    count = N
    short = [per] * count
    long = [2 * per] * (count // 2) + [0] * (count - 2 * (count // 2)) + [0] * (count // 2)
    long[-1] += sum(short) - sum(long)
    s = Solver(N, *lists(N, short, 1))
    for lengths, seed in ((short, 1), (long, 2), (short, 3)):  # longer, then shorter again
        w, off, co = lists(N, lengths, seed)
        s.upload(weight=w, offsets=off, coords=co)
        s.run_plain()
        want, total = s.results()
        for _ in range(2):
            s.run_graph()
            got, tot = s.results()
            assert np.array_equal(got, want) and tot == total
    s.close()
