"""Host-made parents that run in a cycle (of two, three and more vertices, some of them even)
are reported by the candidate test, in shared and in global memory, and the handle works
again once the tree is put right."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import GpuGen, Problem, planar_chain_graph, random_graph
from minimumcyclebasis_gb300._native import MCBError

pytestmark = pytest.mark.gpu


def cycles(root, ps, rows, cols, rev):
    """Cycles of slots that avoid the root, one per length: an edge both ways, then those
    that the edges outside the tree (parent slots ps) close, as lists of slots from one
    vertex of the cycle to the next."""
    out = {}

    def path(v):
        p = [v]
        while p[-1] != root:
            p.append(int(rows[ps[p[-1]]]))
        return p

    for o in range(len(rows)):
        a, b = int(rows[o]), int(cols[o])
        if a == root or b == root or a == b:
            continue
        out.setdefault(2, [o, int(rev[o])])
        if ps[b] == o or ps[a] == rev[o]:
            continue
        pa, pb = path(a), path(b)
        while len(pa) > 1 and len(pb) > 1 and pa[-2] == pb[-2]:
            pa.pop()
            pb.pop()
        if pa[-1] == root:
            continue
        # down from the meeting vertex to a, along o to b, back up to the meeting vertex
        slots = [int(ps[v]) for v in reversed(pa[:-1])] + [o] + [int(rev[ps[v]]) for v in pb[:-1]]
        out.setdefault(len(slots), slots)
        if len(out) >= 8 and 3 in out:
            break
    return out


@pytest.mark.parametrize("make,shared", [(lambda: random_graph(400, 1200, 1, 1000, 1), True),
                                         (lambda: planar_chain_graph(73000, seed=4), False)])
def test_parent_cycles_are_reported(make, shared):
    p = Problem.from_graph(make()).prepare(structure_only=True)
    assert (p.n <= 65534) == shared
    rows, cols, _, rev, _ = p.reduced_graph()
    _, roots = p.fvs()
    gen = GpuGen(p, chunk=2)
    gen.trees(0, 2)
    dist, ps = p.search_trees(np.arange(2))
    gen.put_trees(np.arange(2), dist, ps)
    want = gen.candidates(2)
    found = cycles(int(roots[1]), ps[1], rows, cols, rev)
    assert {2, 3} <= set(found) and any(k > 3 and k % 2 == 0 for k in found)
    for length, slots in sorted(found.items()):
        bad = ps[1:2].copy()
        for k in slots:
            bad[0, cols[k]] = k
        assert len({int(cols[k]) for k in slots}) == length
        gen.put_trees([1], dist[1:2], bad)
        with pytest.raises(MCBError):
            gen.candidates(2)
        gen.put_trees([1], dist[1:2], ps[1:2])
        got = gen.candidates(2)
        assert all(np.array_equal(x, y) for x, y in zip(got, want))
    gen.close()
