"""Staged copies (upload.cpp) when the system gives no more threads: the calling thread does the
rest and the call succeeds, instead of an exception that ends the process."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import resource
import sys
import threading
sys.path.insert(0, %r)
import numpy as np
import rust_rank_b200 as rr
from rust_rank_b200 import synth
P, b, n = 2013265921, 16, 700_001
V = synth.random_vectors(b, n, P, 1)
dr, dc = synth.preconditioners(1, n, P, 2)
dm = rr.CsrMatrix.from_arrays(np.array([0, 1], np.int64), [0], [1], 1, n).to_device(P)
ks = rr.KrylovStream(dm, V, dr, dc, 0)
out = np.ones((b, n), np.uint32)
ks.get_curv(out)
out[:] = 1
# no room for the stacks of as many threads as the copy takes (a few are kept from the first call)
size = next(int(line.split()[1]) for line in open("/proc/self/status") if line.startswith("VmSize"))
resource.setrlimit(resource.RLIMIT_AS, (1024 * size + (1 << 20), resource.getrlimit(resource.RLIMIT_AS)[1]))
ks.get_curv(out)
go, started = threading.Event(), 0
try:
    for started in range(7):
        threading.Thread(target=go.wait).start()
except RuntimeError:
    pass
else:
    started = 7
go.set()
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
assert np.array_equal(out, V)
print("same" if started < 7 else "no limit")
"""


def test_staged_copy_without_threads():
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT], capture_output=True, text=True, timeout=120)
    if r.stdout.strip() == "no limit":
        pytest.skip("as many thread stacks as the copy takes fit all the same")
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr
