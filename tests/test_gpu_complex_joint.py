"""Complex products of the split forms whose four real products run as one product
of [Ar; Ai] with [Br | Bi]: sizes around the row (32) and column (4) alignment of
the second parts, one to several tiles, more than one K chunk.  Against the oracle
bit for bit, with the library's own workspace (all four at once) and with the
smallest workspace the call accepts (one product after the other)."""
import ctypes as C

import pytest

from conftest import to_dev, to_host
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (31, 40, 3), (32, 128, 4), (33, 129, 5), (64, 30, 127), (65, 200, 129), (96, 64, 260),
          (130, 300, 256), (257, 90, 515), (20, 9500, 6)]


@pytest.mark.parametrize("form", ["crt", "split"])
@pytest.mark.parametrize("shape", SHAPES)
def test_joint(cuda_lib, dev, form, shape):
    import torch

    m, k, n = shape
    A = W.complex_from_parts(W.dd_rowcol_scaled(m, k, 4, "row", 1), W.dd_rowcol_scaled(m, k, 4, "row", 2))
    B = W.complex_from_parts(W.dd_rowcol_scaled(k, n, 4, "col", 3), W.dd_rowcol_scaled(k, n, 4, "col", 4))
    want = (O.crt_cgemm if form == "crt" else O.split_cgemm)(A, B, m, k, n)
    want = want[0] if isinstance(want, tuple) else want
    fn = cuda_lib.mfcuda_cmatmuldd_mm_crt if form == "crt" else cuda_lib.mfcuda_cmatmuldd_mm_split
    a, b, c = to_dev(A, dev), to_dev(B, dev), torch.zeros(4 * m * n, dtype=torch.float64, device=dev)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call(ws, size):
        c.zero_()
        return fn(a.data_ptr(), b.data_ptr(), c.data_ptr(), m, k, n, 0, 8.0, ws, size, None, s)

    assert call(None, 0) == 0
    assert O.same_bits(to_host(c), want).all()
    full = (cuda_lib.mfcuda_ccrt_workspace_size(m, k, n, 0) if form == "crt"
            else cuda_lib.mfcuda_csplit_workspace_size(m, k, n))
    ws = torch.empty(full, dtype=torch.uint8, device=dev)
    lo, hi = 0, full  # lo refused, hi accepted
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if call(ws.data_ptr(), mid) == 0:
            hi = mid
        else:
            lo = mid
    for size in {hi, full}:
        assert call(ws.data_ptr(), size) == 0
        assert O.same_bits(to_host(c), want).all()
