"""One workspace, sized for the largest of several shapes, serves all of them: real
and complex, both split forms, also with fewer bits than it was sized for.
Outputs equal those of calls with the library's own workspace."""
import pytest

pytestmark = pytest.mark.gpu

LARGEST = (1309, 512, 666)
SHAPES = [LARGEST, (1028, 97, 591), (1281, 512, 513), (1100, 512, 513), (1100, 300, 600), (257, 40, 515), (129, 512, 666),
          (100, 512, 600), (1309, 1, 1)]


def _rand(n, dev, seed):
    import torch

    g = torch.Generator(device=dev).manual_seed(seed)
    h = torch.rand(n, generator=g, device=dev, dtype=torch.float64) * 2 - 1
    return torch.stack((h, h * 2.0 ** -54), -1).reshape(-1).contiguous()


@pytest.mark.parametrize("sym,size,args", [
    ("mfcuda_matmuldd_mm_split", "mfcuda_split_workspace_size", (0, 9)),
    ("mfcuda_matmuldd_mm_crt", "mfcuda_crt_workspace_size", (0, 60)),
    ("mfcuda_cmatmuldd_mm_split", "mfcuda_csplit_workspace_size", (0, 9)),
    ("mfcuda_cmatmuldd_mm_crt", "mfcuda_ccrt_workspace_size", (0, 60))])
def test_sized_for_the_largest(cuda_lib, dev, sym, size, args):
    import torch

    w = 2 if sym.startswith("mfcuda_c") else 1
    fn = getattr(cuda_lib, sym)
    need = getattr(cuda_lib, size)(*LARGEST, *((0,) if "crt" in size else ()))
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    s = torch.cuda.current_stream().cuda_stream
    for i, (m, k, n) in enumerate(SHAPES):
        a, b = _rand(w * m * k, dev, 2 * i), _rand(w * k * n, dev, 2 * i + 1)
        for arg in args:
            c, d = (torch.full((2 * w * m * n,), 7.0, dtype=torch.float64, device=dev) for _ in range(2))
            assert fn(a.data_ptr(), b.data_ptr(), c.data_ptr(), m, k, n, arg, 8.0, ws.data_ptr(), need, None, s) == 0, (m, k, n, arg)
            assert fn(a.data_ptr(), b.data_ptr(), d.data_ptr(), m, k, n, arg, 8.0, None, 0, None, s) == 0
            assert torch.equal(c.view(torch.int64), d.view(torch.int64)), (m, k, n, arg)
