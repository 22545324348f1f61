"""The column index is made where a second W pass can use it: not for one group of blocks
(128 coordinates).  Both sides of that line against the per-iteration form."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,indexed", [(64, False), (127, False), (128, False), (129, True)])
def test_index_beyond_one_group(N, indexed):
    rng = np.random.default_rng(N)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(3))) for _ in range(40000)] + [np.array([j]) for j in range(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    s = Solver(N, np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32))
    # weights, offsets, lists, heads and two W's without it; 4 bytes per coordinate more with it
    K, nnz = len(rows), int(off[-1])
    assert (s.device_bytes > K * (4 + 8 + 32 + 16) + 8 * nnz) == indexed
    s.run_plain()
    want, total = s.results()
    s.run()
    got, tot = s.results()
    assert np.array_equal(got, want) and tot == total
    s.close()
