"""A long fetch on a device that has no room for its transposed copy of the terms: the terms are
reordered on the host instead of the call being refused."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys
sys.path.insert(0, %r)
import numpy as np
import torch
import rust_rank_b200 as rr
from rust_rank_b200 import synth
P, b, apps = 2013265921, 16, 60_000
rowptr, col, val, m, n = synth.incidence_fast(12, 9, 3, 10, 0, P, 4)
dr, dc = synth.preconditioners(m, n, P, 5)
V = synth.random_vectors(b, n, P, 6)
dm = rr.CsrMatrix.from_arrays(rowptr, col, val, m, n).to_device(P)
ks = rr.KrylovStream(dm, V, dr, dc, 0)
ks.step_device(apps)                       # 65 MB of terms
rr.default_context().synchronize()
rest = []
while torch.cuda.mem_get_info()[0] > 48 << 20:   # not all of the free memory can be had in one piece
    rest.append(torch.empty(max((torch.cuda.mem_get_info()[0] - (24 << 20)) * 7 // 8, 16 << 20), dtype=torch.uint8, device="cuda"))
seq = np.zeros((b * (b + 1) // 2, 2 * apps + 1), np.uint32)
ks.fetch(0, 2 * apps + 1, seq)
del rest
torch.cuda.empty_cache()
again = np.zeros_like(seq)
ks.fetch(0, 2 * apps + 1, again)           # transposed on the device
assert seq.any() and np.array_equal(seq, again)
print("same")
"""


def test_fetch_without_device_memory():
    r = subprocess.run([sys.executable, "-c", SCRIPT % ROOT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr
