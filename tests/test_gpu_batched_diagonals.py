"""Digit-sliced batches on both sides of the line between items of one diagonal and of
two (five single ones per SM): the same problems alone and among so many others that
they are paired, with odd and even slice counts, several tiles and K chunks.  Every
result equals the oracle bit for bit, and the item count follows the rule."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (130, 600, 190), (64, 129, 65)]


@pytest.mark.parametrize("slices", [0, 2, 5])
@pytest.mark.parametrize("more", [0, 400])
@pytest.mark.parametrize("cplx", [False, True])
def test_diagonals(dev, slices, more, cplx):
    import torch

    w = 2 if cplx else 1

    def operand(rows, cols, per, seed):
        parts = [W.dd_rowcol_scaled(rows, cols, 4, per, seed + 100 * p) for p in range(w)]
        return W.complex_from_parts(*parts) if cplx else parts[0]

    host = [(operand(m, k, "row", i), operand(k, n, "col", i + 50)) for i, (m, k, n) in enumerate(SHAPES)]
    probs = [(to_dev(a, dev), to_dev(b, dev), to_dev(np.full(2 * w * m * n, 7.0), dev), m, k, n)
             for (a, b), (m, k, n) in zip(host, SHAPES)]
    one = torch.ones(2 * w, dtype=torch.float64, device=dev)
    probs += [(one, one, torch.empty_like(one), 1, 1, 1) for _ in range(more)]
    with api.GemmBatch(probs, form="split", slices=slices, complex_=cplx) as plan:
        for _ in range(2):
            plan.run()
        assert plan.status() == 0
        out = [to_host(p[2]) for p in probs[:len(SHAPES)]]
        kc = api.lib().mfcuda_batch_kchunk(plan._plan)
        items = api.lib().mfcuda_batch_work_items(plan._plan)
        width = [api.lib().mfcuda_batch_config(plan._plan, i) for i in range(len(probs))]
    # groups of diagonals over the 14 slices there may be: 14 of one, 7 of two
    tiles = (4 if cplx else 1) * sum(-(-m // 128) * -(-n // width[i]) * -(-k // kc)
                                     for i, (_, _, _, m, k, n) in enumerate(probs))
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    assert items == tiles * (14 if tiles * (slices or 14) <= 5 * sms else 7)
    for (m, k, n), (a, b), got in zip(SHAPES, host, out):
        want = (O.split_cgemm if cplx else O.split_gemm)(a, b, m, k, n, slices=slices, kc=kc)
        assert O.same_bits(got, want[0]).all(), (m, k, n)
