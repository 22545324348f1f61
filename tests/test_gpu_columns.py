"""The group's W by the column index and by streaming the lists: the blocked run on
synthetic candidate lists (sparse ones, whose support vectors stay sparse, and dense
ones, whose do not; counts at the edges of tiles, blocks and groups) selects what the
per-iteration form selects, which uses neither."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver

pytestmark = pytest.mark.gpu


def lists(N, K, mean, seed):
    """K random ascending lists over [0, N), then one {j} per coordinate (they span)."""
    rng = np.random.default_rng(seed)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(mean))) for _ in range(K)]
    rows += [np.array([j]) for j in rng.permutation(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("N,K,mean", [(1, 0, 1), (64, 959, 1), (65, 960, 2), (129, 3000, 40), (200, 824, 1),
                                      (300, 700, 150), (700, 1349, 3), (1100, 5000, 2)])
def test_columns_and_streaming_select_alike(N, K, mean):
    w, off, co = lists(N, K, mean, 17 * N + K)
    s = Solver(N, w, off, co)
    s.run_plain()
    want, total = s.results()
    s.reset()
    s.run()
    got, tot = s.results()
    assert np.array_equal(got, want) and tot == total
    for _ in range(2):  # replayed: nothing of the previous solve is left in W or the lists
        s.run_graph()
        got, tot = s.results()
        assert np.array_equal(got, want) and tot == total
    s.close()


def test_a_second_upload_rebuilds_the_index():
    w, off, co = lists(257, 2000, 3, 1)
    # the same lists in another order: sizes as before, another index
    order = np.concatenate([np.random.default_rng(3).permutation(2000), np.arange(2000, 2257)])
    rows = [co[off[i]:off[i + 1]] for i in order]
    off2 = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    s = Solver(257, w, off, co)
    s.run()
    first = s.results()[0]
    s.upload(weight=w, offsets=off2, coords=np.concatenate(rows).astype(np.int32))
    s.run()
    got = s.results()[0]
    s.reset()
    s.run_plain()
    assert np.array_equal(got, s.results()[0]) and not np.array_equal(got, first)
    s.close()
