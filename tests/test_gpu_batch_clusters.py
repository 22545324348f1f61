"""The batched solver with one CTA per problem and with clusters of 2, 4 and 8: few long
problems among short ones, chunk and slice edges of the scan, dense lists whose rounds
overflow a slice, malformed lists and sets that do not span beside good problems.
Against the single-problem per-iteration form."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import BatchSolver, Problem, Solver, random_graph

pytestmark = pytest.mark.gpu


def lists(N, K, mean, seed):
    rng = np.random.default_rng(seed)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(mean))) for _ in range(K)]
    rows += [np.array([j]) for j in rng.permutation(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return N, np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32)


def check(items):
    b = BatchSolver(items)
    for _ in range(2):
        b.run()
        sels, tots = b.results()
    for i, it in enumerate(items):
        s = Solver(*it)
        s.run_plain()
        want, tot = s.results()
        assert np.array_equal(sels[i], want) and tots[i] == tot, i
        for j in {0, it[0] // 2, it[0] - 1}:
            assert np.array_equal(b.support_vector(i, j), s.support_vector(j)), (i, j)
        s.close()
    b.close()


# (N, K, mean list length) of the long problem; short ones beside it
@pytest.mark.parametrize("long", [(600, 1500, 3), (1025, 9000, 3), (2000, 17000, 4), (2100, 40000, 2), (4100, 33000, 6),
                                  (1300, 66000, 25)])
@pytest.mark.parametrize("short", [0, 5])
def test_long_problems_among_short_ones(long, short):
    items = [lists(*long, 1)] + [lists(40 + 60 * i, 500 * i, 3, i) for i in range(short)]
    check(items)


def test_graphs_of_very_different_sizes():
    items = []
    for n, seed in ((3000, 1), (2500, 2), (90, 3), (60, 4)):
        p = Problem.from_graph(random_graph(n, 2 * n, 1, 50, seed)).prepare()
        off, co = p.cycle_lists()
        items.append((p.N, p.candidates()[2], off, co))
    check(items)


def test_bad_problems_fail_alone():
    good, other = lists(1500, 20000, 3, 5), lists(300, 900, 3, 6)
    bad = lists(200, 900, 3, 7)
    co = bad[3].copy()
    co[bad[2][5]] = 200  # out of range
    few = (100, np.ones(50, np.int32), np.arange(51, dtype=np.int64), np.arange(50, dtype=np.int32))
    b = BatchSolver([good, (200, bad[1], bad[2], co), few, other])
    b.run()
    st = b.status()
    assert st[0] == 0 and st[3] == 0 and st[1] != 0 and st[2] != 0 and st[1] != st[2]
    b.close()
