"""Memory that the workspace pool keeps between calls: kept below its limit, and
given back to the device by release_workspace (other processes can have it then)."""
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _free(dev):
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(dev)[0]


def test_kept_then_released(dev):
    import torch

    n = 4096  # a workspace of 1.6 GB
    a = torch.ones(2 * n * n, dtype=torch.float64, device=dev)
    c = torch.empty_like(a)
    a[1::2] = 0.0
    api.release_workspace()
    api.sum_dd(a[:200])  # modules loaded, pool made
    api.matmuldd_mm_crt(a[:200], a[:200], 10, 10, 10)
    api.release_workspace()
    before = _free(dev)
    for _ in range(2):  # the second call reuses what the first one left
        api.matmuldd_mm_crt(a, a, n, n, n, out=c)
        held = before - _free(dev)
        assert 1 << 30 <= held <= (2 << 30), held
    api.release_workspace()
    assert before - _free(dev) < 64 << 20
    # and the library goes on working
    m, k, q = 100, 90, 80
    x, y = W.dd_rowcol_scaled(m, k, 8, "row", 1), W.dd_rowcol_scaled(k, q, 8, "col", 2)
    got = to_host(api.matmuldd_mm_crt(to_dev(x, dev), to_dev(y, dev), m, k, q)[0])
    assert O.same_bits(got, O.crt_gemm(x, y, m, k, q)[0]).all()
    assert float(c[0]) == n
