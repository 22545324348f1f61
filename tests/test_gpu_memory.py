"""What is optional on the device gives way where the memory is short: a solver's column index
takes no more than a quarter of what is free, and makes room for an upload's pair buffers
and for the certificate's matrix; a generation's former lists make room for the next
ranking."""
import numpy as np
import pytest

from minimumcyclebasis_gb300 import GpuGen, Solver, prepare_on_device, random_graph
from minimumcyclebasis_gb300.devprep import generate_candidates

pytestmark = pytest.mark.gpu
MB = 1 << 20


class Squeeze:
    """Holds all of the GPU's free memory but `leave` bytes and at most 12 MB more."""

    def __init__(self, leave):
        import torch
        self.torch, self.held = torch, []
        torch.cuda.empty_cache()
        size = 1 << 36
        while size >= 10 * MB:
            if torch.cuda.mem_get_info()[0] >= leave + size:
                try:
                    self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                    continue
                except torch.cuda.OutOfMemoryError:
                    pass
            size = max(size // 2, 10 * MB) if size > 10 * MB else 0

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.held.clear()
        self.torch.cuda.empty_cache()


def lists(N, K, length, seed):
    """A list of all coordinates, K random ones of the given length, then {j} for every one."""
    rng = np.random.default_rng(seed)
    rows = [np.arange(N)] + [np.sort(rng.choice(N, length, replace=False)) for _ in range(K)]
    rows += [np.array([j]) for j in rng.permutation(N)]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    return np.arange(1, len(rows) + 1, dtype=np.int32), off, np.concatenate(rows).astype(np.int32)


@pytest.fixture(autouse=True)
def _loaded():
    """Every kernel loaded, and its local memory made, while there is room."""
    s = Solver(130, *lists(130, 400, 20, 1))
    s.run()
    s.results()
    s.verify()
    s.close()


def test_the_index_takes_a_quarter_at_most():
    nnz = 300_000_000
    args = np.ones(3, np.int32), np.array([0, 0, 0, nnz], np.int64), np.zeros(1, np.int32)  # the sizes alone
    s = Solver(500, *args, upload=False)
    full = s.device_bytes
    s.close()
    for times, taken in ((8, True), (3, False)):  # the lists take one part, the index another
        with Squeeze(times * 4 * nnz):
            s = Solver(500, *args, upload=False)
            assert (s.device_bytes == full) == taken and (full - s.device_bytes >= 4 * nnz) == (not taken)
            s.close()


def test_an_upload_takes_the_index_s_room():
    N = 50000
    args = lists(N, 700, 25000, 2)  # 70 MB of index; the pairs take 38 MB
    ref = Solver(N, *args)
    ref.run(64)
    want = ref.results(64)[0]
    ref.close()
    s = Solver(N, *args, upload=False)
    before = s.device_bytes
    with Squeeze(0):
        s.upload()
        assert s.device_bytes < before
        s.run(64)
        assert np.array_equal(s.results(64)[0], want)
    s.close()


def test_the_certificate_takes_the_index_s_room():
    N = 20000
    s = Solver(N, *lists(N, 2000, 10000, 3))  # 80 MB of index; the matrix takes 50 MB
    before = s.device_bytes
    s.run_graph()
    sel, total = s.results()
    with Squeeze(0):
        assert s.verify()["rank"] == N
        assert s.device_bytes < before  # a quarter of what is free now would not hold it
    s.run_graph()
    got, tot = s.results()
    assert np.array_equal(got, sel) and tot == total
    assert s.verify()["rank"] == N
    s.close()


def ranked(gen, p, which):
    """The lists of some of the ranks: offsets and coordinates."""
    _, edge, w, tree = p.candidates()
    gen.lists(tree[which], edge[which], w[which])
    return gen.fetch_lists()


def test_former_lists_make_room_for_a_ranking():
    d, gen = prepare_on_device(random_graph(30000, 60000, 1, 1000, 4), make_solver=False, keep_gen=True)
    p = d.problem
    off, co = gen.fetch_lists()
    gen.close()
    by_length = np.argsort(np.diff(off), kind="stable")
    short, long = np.sort(by_length[:3_700_000]), np.sort(by_length[-3_000_000:])
    # 24 bytes per rank and 4 per coordinate: the second ranking does not fit beside the first lists
    room = 24 * len(long) + 4 * int(np.diff(off)[long].sum())
    need = 24 * len(short) + 4 * int(np.diff(off)[short].sum())
    assert 24 * len(short) > 24 * len(long) + 12 * MB and need + 8 * MB < room
    gen = GpuGen(p)
    generate_candidates(p, gen)
    ranked(gen, p, long)
    with Squeeze(0):
        got = ranked(gen, p, short)
    assert np.array_equal(got[0], np.concatenate([[0], np.cumsum(np.diff(off)[short])]))
    at = np.repeat(off[short] - got[0][:-1], np.diff(got[0])) + np.arange(got[0][-1])
    assert np.array_equal(got[1], co[at])
    gen.close()
