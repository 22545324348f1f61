"""List heads of 16-bit coordinates (up to 65,535 of them) and of 32-bit ones: lists that
end before, at and past either head's length, with the smallest and largest coordinates,
against elimination in rank order (the chosen cycles are the rank-first basis)."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver

pytestmark = pytest.mark.gpu


def rank_first_basis(rows):
    """Ranks of the rows not spanned by earlier ones; rows are Python ints (bit sets)."""
    basis, out = {}, []
    for r, v in enumerate(rows):
        while v and v.bit_length() in basis:
            v ^= basis[v.bit_length()]
        if v:
            basis[v.bit_length()] = v
            out.append(r)
    return out


@pytest.mark.parametrize("pad", [0, 65335, 65336])  # 200, 65,535 and 65,536 coordinates
def test_lists_around_the_heads_length(pad):
    rng = np.random.default_rng(pad + 1)
    n, sizes = 200, (1, 2, 7, 8, 9, 15, 16, 17, 24, 41)
    base = [np.sort(rng.choice(n, sizes[i % len(sizes)], replace=False)) for i in range(3000)]
    base += [np.array([j]) for j in rng.permutation(n)]
    want = rank_first_basis([sum(1 << int(c) for c in r) for r in base])
    # the first `pad` coordinates are cycles of their own, so that lists may hold them freely
    low = [np.unique(rng.integers(0, pad, i % 12)) if pad else np.zeros(0, int) for i in range(len(base))]
    rows = [np.array([c]) for c in range(pad)] + [np.concatenate([a, r + pad]) for a, r in zip(low, base)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    w = np.arange(1, len(rows) + 1, dtype=np.int32)
    s = Solver(n + pad, w, off, np.concatenate(rows).astype(np.int32))
    for run in (s.run, s.run_plain):
        s.reset()
        run()
        got = np.sort(s.results()[0])
        assert np.array_equal(got[:pad], np.arange(pad)) and np.array_equal(got[pad:] - pad, want)
    s.close()
