"""Host memory running out while a candidate generation is created is an error code, not an
exception through the C entry (which would end the process).  In a child whose address
space leaves no room for the arc table (64 bytes per vertex); no GPU is needed."""
import subprocess
import sys

from conftest import ROOT

CHILD = """
import ctypes as C, resource
import numpy as np
from minimumcyclebasis_gb300._native import gpu_lib, ptr
lib = gpu_lib()
n = 2_000_000  # a ring: two slots per vertex
v = np.arange(n, dtype=np.int64)
ro = (2 * np.arange(n + 1)).astype(np.uint32)
rows = np.repeat(v, 2).astype(np.uint32)
cols = np.stack([(v - 1) % n, (v + 1) % n], 1).reshape(-1).astype(np.uint32)
rev = np.stack([2 * ((v - 1) % n) + 1, 2 * ((v + 1) % n)], 1).reshape(-1).astype(np.uint32)
w = np.ones(2 * n, np.int32)
ec = np.full(2 * n, -1, np.int32)
fa = np.full(n, -1, np.int32)
fa[0] = 0
fv = np.zeros(1, np.uint32)
pairs = np.flatnonzero(np.arange(2 * n) < rev).astype(np.uint32)
assert len(pairs) == n
h = C.c_void_p()
args = (C.byref(h), n, C.c_int64(2 * n), ptr(ro), ptr(rows), ptr(cols), ptr(w), ptr(rev), ptr(ec), 1, ptr(fa), ptr(fv), 1,
        ptr(pairs), 1)
lib.mcbgpu_gen_create(C.byref(h), 0, *args[2:])  # the first call's own needs
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (100 << 20), used + (100 << 20)))
rc = lib.mcbgpu_gen_create(*args)
print("rc", rc, (lib.mcbgpu_last_error() or b"").decode())
"""


def test_no_exception_leaves_the_entry():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    assert r.stdout.startswith("rc -") and "out of memory" in r.stdout, r.stdout
