"""Staging memory of the host-pointer complex split calls.  The buffers are kept
for the life of the process, so a call takes no more than it uses, and a call
whose larger workspace cannot be allocated takes the smaller route."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

_HEAD = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import ctypes as C
import numpy as np
import torch
from multifloats_b200 import _lib
from multifloats_b200 import workloads as W
from oracle import oracle as O

L = _lib.lib()
p = lambda t: t.ctypes.data
"""

_HELD = _HEAD + """
def call(m, k, n):
    a, b, c = np.ones(4 * m * k), np.ones(4 * k * n), np.empty(4 * m * n)
    L.cmatmuldd_mm_crt(p(a), p(b), p(c), m, k, n, 0, None)
    assert L.mfcuda_last_error() == 0
torch.zeros(1, device="cuda")
call(20, 20, 20)
before = torch.cuda.mem_get_info()[0]
call(2700, 300, 2700)
torch.cuda.synchronize()
print((before - torch.cuda.mem_get_info()[0]) >> 20)
"""

_FAIL = _HEAD + """
m, k, n = 300, 200, 280
a = W.complex_from_parts(W.dd_rowcol_scaled(m, k, 8, "row", 1), W.dd_rowcol_scaled(m, k, 8, "row", 2))
b = W.complex_from_parts(W.dd_rowcol_scaled(k, n, 8, "col", 3), W.dd_rowcol_scaled(k, n, 8, "col", 4))
c = np.empty(4 * m * n)
bound = C.c_double()
L.cmatmuldd_mm_split(p(a), p(b), p(c), m, k, n, 0, C.byref(bound))
want = O.split_cgemm(a, b, m, k, n)[0]
print(L.mfcuda_last_error(), int(O.same_bits(c, want).all()))
"""


def _child(src, **env):
    proc = subprocess.run([sys.executable, "-c", src.format(root=ROOT)], env=dict(os.environ, **env),
                          capture_output=True, text=True, timeout=300)
    assert proc.returncode == 0, proc.stderr[-2000:]
    return [int(v) for v in proc.stdout.split()]


def test_crt_call_keeps_what_it_uses():
    # operands and result 285 MB, workspace of one product at a time 410 MB (of all four 1117)
    assert _child(_HELD)[-1] < 1000


def test_split_call_without_room_for_all_four():
    # the fourth allocation of the process is the workspace
    assert _child(_FAIL, MFCUDA_FAIL_ALLOC="4") == [0, 1]
    assert _child(_FAIL) == [0, 1]
