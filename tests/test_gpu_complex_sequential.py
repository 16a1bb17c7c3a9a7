"""Complex products of the split forms with a workspace that holds one of the four
real products at a time: shapes whose joint layout is the larger one, so that the
smallest workspace the call accepts can only serve one product after the other;
one K chunk and two (the residues' fold, the recombination over chunks)."""
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# joint: 128 + 97 rows pad to 256 instead of 128, 132 + 130 columns to 512 instead of 256
@pytest.mark.parametrize("form,arg", [("crt", 20), ("split", 3)])
@pytest.mark.parametrize("shape", [(97, 200, 130), (97, 9500, 130)])
def test_one_after_the_other(cuda_lib, dev, form, arg, shape):
    import torch

    m, k, n = shape
    A = W.complex_from_parts(W.dd_rowcol_scaled(m, k, 4, "row", 1), W.dd_rowcol_scaled(m, k, 4, "row", 2))
    B = W.complex_from_parts(W.dd_rowcol_scaled(k, n, 4, "col", 3), W.dd_rowcol_scaled(k, n, 4, "col", 4))
    want = (O.crt_cgemm if form == "crt" else O.split_cgemm)(A, B, m, k, n, arg)
    want = want[0] if isinstance(want, tuple) else want
    fn = getattr(cuda_lib, f"mfcuda_cmatmuldd_mm_{form}")
    full = (cuda_lib.mfcuda_ccrt_workspace_size(m, k, n, arg) if form == "crt"
            else cuda_lib.mfcuda_csplit_workspace_size(m, k, n))
    a, b, c = to_dev(A, dev), to_dev(B, dev), torch.zeros(4 * m * n, dtype=torch.float64, device=dev)
    ws = torch.empty(full, dtype=torch.uint8, device=dev)
    s = torch.cuda.current_stream().cuda_stream

    def call(size):
        c.zero_()
        return fn(a.data_ptr(), b.data_ptr(), c.data_ptr(), m, k, n, arg, 8.0, ws.data_ptr(), size, None, s)

    lo, hi = 0, full  # lo refused, hi accepted
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if call(mid) == 0 else (mid, hi)
    assert full - hi >= 500_000  # the diagonals or residues of three products
    for size in (hi, full):
        assert call(size) == 0
        assert O.same_bits(to_host(c), want).all(), size
