"""The tree kernel's forms where a round's list of vertices overflows: graphs with wide
frontiers (random, of mean degree 4 to 16; equal weights) around the sizes and degrees
where the form changes, a few roots each, against the host's searches."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import GpuGen, Problem, planar_chain_graph, random_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: random_graph(50000, 400000, 1, 1000, 1),   # distances in shared memory
                                  lambda: random_graph(72000, 144000, 1, 1000, 2),   # two bitmaps
                                  lambda: random_graph(66000, 198000, 1, 1000, 3),   # more arcs per vertex
                                  lambda: random_graph(66000, 528000, 1, 1000, 4),
                                  lambda: planar_chain_graph(86000, seed=5),          # the largest with two bitmaps
                                  lambda: planar_chain_graph(88000, seed=6),
                                  lambda: random_graph(96000, 192000, 1, 1000, 7),
                                  lambda: random_graph(150000, 600000, 1, 1000, 8),
                                  lambda: random_graph(250000, 500000, 1, 3, 9)])
def test_trees_of_wide_frontiers(make):
    p = Problem.from_graph(make()).prepare(structure_only=True)
    gen = GpuGen(p, chunk=6)
    for t0 in (0, p.F // 2, p.F - 6):
        tied = gen.trees(t0, 6)
        dist, ps = p.search_trees(np.arange(t0, t0 + 6))
        if len(np.nonzero(tied)[0]):
            gen.put_trees(t0 + np.nonzero(tied)[0], dist[tied != 0], ps[tied != 0])
        # the device's trees are the host's: the same candidates as with all of them put
        before = gen.candidates(6)
        gen.put_trees(np.arange(t0, t0 + 6), dist, ps)
        after = gen.candidates(6)
        assert all(np.array_equal(x, y) for x, y in zip(before, after))
    gen.close()
