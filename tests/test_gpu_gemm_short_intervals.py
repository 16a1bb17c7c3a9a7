"""Plain products with renormalisation intervals of a few steps, which run kernels of
their own up to three: every kind of tile (64, 32, 16, mixed; complex 32, 16), depths
that end on a group of eight, one step before and after it, aligned operands or not,
single products and batches.  Every output equals the oracle bit for bit."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

INTERVALS = [1, 2, 3, 4]
REAL = [(1, 1, 1), (17, 8, 15), (250, 41, 300), (381, 33, 384), (960, 9, 639), (3899, 17, 185), (64 * 37, 15, 256)]
CPLX = [(3, 5, 2), (130, 33, 70), (480, 9, 319), (1184, 16, 128)]


def _dev(x, dev, off):
    return to_dev(np.concatenate([np.zeros(off), x]), dev)[off:]


@pytest.mark.parametrize("ri", INTERVALS)
@pytest.mark.parametrize("off", [0, 1])
def test_single(dev, ri, off):
    for m, k, n in REAL:
        a, b = W.dd_uniform(m * k, seed=m + k), W.dd_uniform(k * n, seed=n + 7)
        got = to_host(api.matmuldd_mm(_dev(a, dev, off), _dev(b, dev, off), m, k, n, ri))
        assert O.same_bits(got, O.matmul_mm(a, b, m, k, n, ri)).all(), (m, k, n)
    for m, k, n in CPLX:
        a, b = W.dd_uniform(2 * m * k, seed=m), W.dd_uniform(2 * k * n, seed=n)
        got = to_host(api.cmatmuldd_mm(_dev(a, dev, off), _dev(b, dev, off), m, k, n, ri))
        assert O.same_bits(got, O.cmatmul_mm(a, b, m, k, n, ri)).all(), (m, k, n)


@pytest.mark.parametrize("ri", INTERVALS)
@pytest.mark.parametrize("cplx", [False, True])
def test_batch(dev, ri, cplx):
    shapes, w = [(1, 1, 1), (17, 40, 30), (65, 8, 33), (40, 300, 25), (150, 31, 97), (5, 0, 9)], 2 if cplx else 1
    host = [(W.dd_uniform(w * m * k, seed=i), W.dd_uniform(w * k * n, seed=i + 50)) for i, (m, k, n) in enumerate(shapes)]
    probs = [(to_dev(a, dev), to_dev(b, dev), to_dev(np.full(2 * w * m * n, 7.0), dev), m, k, n)
             for (a, b), (m, k, n) in zip(host, shapes)]
    with api.GemmBatch(probs, form="plain", renorm_interval=ri, complex_=cplx) as plan:
        plan.run()
        out = [to_host(p[2]) for p in probs]
    for (m, k, n), (a, b), got in zip(shapes, host, out):
        want = (O.cmatmul_mm if cplx else O.matmul_mm)(a, b, m, k, n, ri) if k else np.zeros_like(got)
        assert O.same_bits(got, want).all(), (m, k, n)
