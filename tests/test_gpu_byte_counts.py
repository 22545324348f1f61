"""The byte counters of a run whose W come from the column index: one pair of blocks, whose
rows are still the unit vectors, so that every coordinate below 128 of every list is read
once (4 bytes) and adds to one W (16)."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(129, 3000), (300, 20000)])
def test_w_by_columns_and_its_zeroing_are_counted(N, K):
    rng = np.random.default_rng(N)
    rows = [np.unique(rng.integers(0, N, 1 + rng.poisson(4))) for _ in range(K)] + [np.array([j]) for j in range(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    co = np.concatenate(rows).astype(np.int32)
    s = Solver(N, np.arange(1, len(rows) + 1, dtype=np.int32), off, co)
    s.set_profiling(True)
    s.run(128)
    s.results(128)
    st = s.kernel_stats()
    nnz, tiles = int((co < 128).sum()), -(-len(rows) // 1024)
    # besides: per coordinate and warp that works on it, 12 bytes and its two words
    warps = 32 * 2 * 152
    assert 20 * nnz < st["blk_w"]["bytes"] <= 20 * nnz + 28 * max(warps, N)
    # the transposes of both blocks; at 64 columns of 8-byte words each, three times, they are
    # small beside the two W's of every candidate
    zeroed = 2 * 8 * 1024 * tiles
    assert zeroed < st["blk_transpose"]["bytes"] <= zeroed + 8 * 2 * 6 * 64 * 2
    s.close()
