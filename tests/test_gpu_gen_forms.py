"""Candidate generation where its forms meet: trees with distances in shared memory (up
to 53,248 vertices), with the near and far vertices alone there (up to 98,304), and
neither, with rows of more and of fewer arcs than the arc table's eight; the
candidate test in shared memory (up to 65,534 vertices) and over global memory.  A few
roots of each graph, against the host's heap searches and the numpy restatement of the
candidate test.  The lists' walks by rank and by tree."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import GpuGen, Problem, planar_chain_graph, prepare_on_device, random_graph
from minimumcyclebasis_gb300.devprep import generate_candidates
from test_two_stage_host import root_candidates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,lo,hi", [(lambda: random_graph(3000, 6000, 1, 1000, 1), 1, 53248),
                                        (lambda: planar_chain_graph(57500, seed=2), 1, 53248),
                                        (lambda: planar_chain_graph(60000, seed=3), 53249, 65534),
                                        (lambda: planar_chain_graph(73000, seed=4), 65535, 98304),
                                        (lambda: random_graph(125000, 250000, 1, 1000, 5), 98305, 1 << 21)])
def test_a_few_roots(make, lo, hi):
    p = Problem.from_graph(make()).prepare(structure_only=True)
    assert lo <= p.n <= hi
    rows, cols, w, rev, _ = p.reduced_graph()
    fa, roots = p.fvs()
    pairs = p.pairs()
    gen = GpuGen(p, chunk=5)
    for t0 in (0, p.F // 2, p.F - 5):
        tied = gen.trees(t0, 5)
        dist, ps = p.search_trees(np.arange(t0, t0 + 5))
        idx = np.nonzero(tied)[0]
        if len(idx):
            gen.put_trees(t0 + idx, dist[idx], ps[idx])
        pi, wi, counts = gen.candidates(5)
        at = 0
        for i in range(5):
            k, wk = root_candidates(int(roots[t0 + i]), dist[i], ps[i].astype(np.int64), rows, cols, w.astype(np.int64),
                                    rev, fa, pairs)
            assert counts[i] == len(k)
            assert np.array_equal(pi[at:at + len(k)], k) and np.array_equal(wi[at:at + len(k)], wk)
            at += len(k)
    gen.close()


def test_lists_walked_tree_by_tree():
    """9,000 planar points: over 64 MB of parent slots and hundreds per candidate, so the
    walks go tree by tree; the lists of all ranks and of half of them, against the host's."""
    g = planar_chain_graph(9000, seed=6)
    off, co = Problem.from_graph(g).prepare(cycle_lists=True).cycle_lists()
    d, gen = prepare_on_device(g, make_solver=False, keep_gen=True)
    p = d.problem
    assert 4 * p.F * p.n > 64 << 20 and p.F * p.n // d.K >= 64
    got = gen.fetch_lists()
    assert np.array_equal(got[0], off) and np.array_equal(got[1], co)
    gen.close()
    gen = GpuGen(p)
    _, edge, w, tree = p.candidates()
    generate_candidates(p, gen)
    half = np.sort(np.random.default_rng(1).permutation(d.K)[:d.K // 2])
    gen.lists(tree[half], edge[half], w[half])
    got = gen.fetch_lists()
    assert np.array_equal(got[0], np.concatenate([[0], np.cumsum(np.diff(off)[half])]))
    assert np.array_equal(got[1], np.concatenate([co[off[r]:off[r + 1]] for r in half]))
    gen.close()
