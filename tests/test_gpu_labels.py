"""The label pass at the sizes where its forms meet: one position, a chain as deep as
the tree is large, more levels than a CTA has threads, the 16-bit and the 32-bit words
(2^15 positions), the largest tree in shared memory and the first of the level sweep,
against a sweep in numpy; parents that do not precede their children are flagged."""
import ctypes as C

import numpy as np
import pytest

from minimumcyclebasis_gb300 import GpuStruct
from minimumcyclebasis_gb300._native import gpu_lib

pytestmark = pytest.mark.gpu


def forest(n, F, width, edges, N, seed):
    """F trees of n positions in levels of up to `width`, random parents in the level above."""
    rng = np.random.default_rng(seed)
    levels = np.full((F, n + 1), n, np.uint32)
    parent = np.zeros((F, n), np.uint32)
    for t in range(F):
        at, k, prev = 1, 1, (0, 1)
        levels[t, 0] = 0
        while at < n:
            m = min(n - at, int(rng.integers(1, width + 1)))
            levels[t, k] = at
            parent[t, at:at + m] = rng.integers(prev[0], prev[1], m)
            prev, at, k = (at, at + m), at + m, k + 1
    edge = rng.integers(-1, edges, (F, n)).astype(np.int32)
    edge[:, 0] = -1
    return levels, parent, edge, rng.integers(-1, N, edges).astype(np.int32)


def expected(parent, edge, cmap, S):
    bits = np.unpackbits(S.view(np.uint8), bitorder="little")
    cols = np.where(edge >= 0, cmap[np.maximum(edge, 0)], -1)
    own = np.where(cols >= 0, bits[np.maximum(cols, 0)], 0).astype(np.uint32)
    lab = np.zeros_like(parent)
    for i in range(1, parent.shape[1]):  # parents precede children
        lab[:, i] = own[:, i] ^ lab[np.arange(len(lab)), parent[:, i]]
    return lab


@pytest.mark.parametrize("n,F,width", [(1, 3, 1), (2, 5, 1), (900, 7, 1), (3000, 5, 3), (12288, 3, 500), (12289, 3, 40),
                                       (32768, 3, 2000), (32769, 2, 100), (53248, 2, 300), (53249, 2, 300)])
def test_labels_equal_a_sweep(n, F, width):
    import torch
    edges, N = 777, 129
    levels, parent, edge, cmap = forest(n, F, width, edges, N, n + F)
    S = np.random.default_rng(n).integers(0, 2 ** 63, 3, dtype=np.int64).view(np.uint64)
    S[2] &= np.uint64(1)
    want = expected(parent, edge, cmap, S)
    gs = GpuStruct(edges, N, n, F, chunk_size=2)
    gs.initialize_memory(cmap, levels.reshape(-1), parent.reshape(-1), edge.reshape(-1))
    gs.copy_support_vector(S)
    assert np.array_equal(gs.process_shortest_path()[0], want)
    gs.close()
    dev = [torch.from_numpy(np.ascontiguousarray(a).view(np.int64 if a.dtype == np.uint64 else np.int32)).cuda()
           for a in (levels, parent, edge, cmap, S)]
    out = torch.full((F, n), 5, dtype=torch.int32, device="cuda")
    lv, pp, eo, mp, sv = (C.c_void_p(t.data_ptr()) for t in dev)
    assert gpu_lib().mcbgpu_label_forest_noalloc(lv, pp, eo, mp, edges, sv, N, F, n, C.c_void_p(out.data_ptr()), None) == 0
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)


def test_parent_after_child_is_flagged():
    levels, parent, edge, cmap = forest(40, 2, 4, 50, 64, 3)
    parent[1, 7] = 9
    gs = GpuStruct(50, 64, 40, 2)
    gs.initialize_memory(cmap, levels.reshape(-1), parent.reshape(-1), edge.reshape(-1))
    gs.copy_support_vector(np.array([5], np.uint64))
    assert gs.lib.mcbgpu_struct_process_shortest_path(gs._h, None, 0, None) != 0
    assert b"status 0x8" in gs.lib.mcbgpu_last_error()
    gs.close()
