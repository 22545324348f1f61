"""Rules of warp and barrier use that no run can show to be kept (a broken one goes wrong
once in a long while), read off the kernels' sources."""
import os
import re

from conftest import ROOT

GPU = os.path.join(ROOT, "minimumcyclebasis_gb300", "csrc", "gpu")


def kernel(file, name):
    """The body of a function of a source file, without comments."""
    text = open(os.path.join(GPU, file)).read()
    text = re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", text), flags=re.S)
    at = text.index("{", text.index(name + "("))
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError(name)


def test_far_rows_alternate_their_buffers_with_the_barrier():
    """Two warps share a group's partial sums through sD[par] and one barrier per group
    that has a row left.  A warp may pass the next barrier only after the other has
    arrived there, so a buffer is safe to write again two barriers on: par has to change
    with every barrier and with nothing else (a group without rows has no barrier)."""
    body = kernel("mcbgpu_solver.cu", "far_rows_kernel")
    changes = [m.start() for m in re.finditer(r"\bpar\s*(\^=|=(?!=)|\+\+|\+=)", body)]
    assert body[changes[0] - 4:changes[0]] == "int " and len(changes) == 2
    barrier = body.index("barrier.sync")
    assert "barrier.sync" not in body[barrier + 1:]
    between = body[barrier:changes[1]]
    assert changes[1] > barrier and "continue" not in between and "break" not in between
    # both in the block that the barrier's condition opens
    assert between.count("}") == between.count("{")


def test_a_word_that_others_change_decides_for_whole_warps():
    """A loop of warp collectives must not be left by each lane's own look at a word that
    other CTAs change meanwhile: lanes that saw different values part, and those that stay
    wait in the next collective for those that left.  Such a look is taken by one lane and
    handed to the others."""
    for file in sorted(os.listdir(GPU)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(GPU, file)).read())
        for m in re.finditer(r"\bif \(([^;{}]*volatile[^;{}]*)\)\s*\{?\s*(break|continue|return)\b", text):
            raise AssertionError((file, m.group(0)))
    body = kernel("mcbgpu_solver.cu", "plain_kernel")
    loop = body[body.index("for (long long r0"):]
    look = re.search(r"if \(lane == 0\) (\w+) = \*\(\(volatile unsigned long long \*\)&slot->best\);", loop)
    leave = re.search(r"if \(\(unsigned long long\)r0 > __shfl_sync\(0xffffffffu, (\w+), 0\)\) break;", loop)
    assert look and leave and look.group(1) == leave.group(1) and look.end() < leave.start()
    assert leave.end() < loop.index("__ballot_sync") and loop.count("slot->best") == 2  # the other: atomicMin


def test_a_warp_is_whole_before_it_reads_tensor_memory():
    """tcgen05.ld is a warp-aligned instruction and a thread leaves the mbarrier's polls by
    itself, so a barrier of the warp or of the CTA stands between."""
    for name in ("mlp_forward_kernel", "mlp_grads_kernel"):
        body = kernel("mcbgpu_mlp.cu", name)
        loop = body[body.index("for (int64_t tile"):]
        wait = loop.index("mbar_wait_bounded(")
        read = loop.index("tmem_ld", wait)
        assert re.search(r"__syncwarp\(\)|cta_sync(_and)?\(", loop[wait:read]), name
