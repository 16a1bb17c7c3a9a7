"""Stream capture of single calls with the library's own workspace.  The call in the
capture may be the first one of the process, when the workspace pool is made:
each case runs in a process of its own, captures its call before any other, and
the replay equals the oracle's result and a plain call's bit for bit."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import torch
from conftest import to_dev, to_host
from multifloats_b200 import _lib
from multifloats_b200 import workloads as W
from oracle import oracle as O

L, what, mode = _lib.lib(), {what!r}, {mode!r}
dev = torch.device("cuda:0")
m, k, n = 150, 200, 300
x = W.dd_uniform(30000, 1)
a, b = W.dd_rowcol_scaled(m, k, 8, "row", 2), W.dd_rowcol_scaled(k, n, 8, "col", 3)
if what[0] == "c":
    a = W.complex_from_parts(a, W.dd_rowcol_scaled(m, k, 8, "row", 4))
    b = W.complex_from_parts(b, W.dd_rowcol_scaled(k, n, 8, "col", 5))
fn = {{"split": (L.mfcuda_matmuldd_mm_split, O.split_gemm), "csplit": (L.mfcuda_cmatmuldd_mm_split, O.split_cgemm),
      "crt": (L.mfcuda_matmuldd_mm_crt, O.crt_gemm), "ccrt": (L.mfcuda_cmatmuldd_mm_crt, O.crt_cgemm)}}
want = O.reduce_blocked("dot", x, x) if what == "dot" else fn[what][1](a, b, m, k, n)
want = want[0] if isinstance(want, tuple) else want
dx, da, db = to_dev(x, dev), to_dev(a, dev), to_dev(b, dev)
out = torch.zeros(want.size, dtype=torch.float64, device=dev)


def call():
    s = torch.cuda.current_stream().cuda_stream
    if what == "dot":
        return L.mfcuda_dotdd(dx.data_ptr(), dx.data_ptr(), 30000, 8, out.data_ptr(), None, 0, s)
    return fn[what][0](da.data_ptr(), db.data_ptr(), out.data_ptr(), m, k, n, 0, 8.0, None, 0, None, s)


torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g, capture_error_mode=mode):
    rc = call()
for _ in range(2):
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert O.same_bits(to_host(out), want).all()
out.zero_()
assert rc == 0 and call() == 0
torch.cuda.synchronize()
assert O.same_bits(to_host(out), want).all()
print("equal")
"""


CASES = [(w, "global") for w in ("dot", "split", "crt", "csplit", "ccrt")] + [(w, "thread_local") for w in ("dot", "crt")]


@pytest.mark.parametrize("what,mode", CASES)
def test_first_call_in_a_capture(what, mode):
    proc = subprocess.run([sys.executable, "-c", _CHILD.format(root=ROOT, what=what, mode=mode)],
                          env=dict(os.environ), capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0 and proc.stdout.split()[-1:] == ["equal"], proc.stderr[-2000:]
