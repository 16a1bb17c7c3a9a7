"""GPU parity of the plain products at the sizes where the tile choice changes:
uniform tiles of 16 and 32, whole tiles of 64 with the rest cut into 4 or 16
(complex: 32 and 16), depths that end inside a group of eight steps or a stage,
and renormalisation intervals that are or are not a multiple of the group.
Every output equals the oracle bit for bit."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# m, k, n and the tiles a 148-SM device cuts them into
REAL = [
    (1, 1, 1),         # one 16 x 16 tile, one step
    (15, 7, 17),       # edges below and above 16, no full group
    (250, 40, 300),    # 304 tiles of 16
    (381, 33, 384),    # 144 tiles of 32, one step past a 16-deep stage
    (960, 9, 639),     # 148 tiles of 64 and 2 cut into 16
    (3899, 24, 185),   # 148 tiles of 64 and 35 cut into 4
    (64 * 37, 8, 256),  # 148 whole tiles
]
CPLX = [(3, 5, 2), (130, 17, 70), (480, 9, 319), (1184, 16, 128)]


@pytest.mark.parametrize("shape", REAL)
@pytest.mark.parametrize("ri", [8, 0, 5, 24])
def test_real_tiles(dev, shape, ri):
    m, k, n = shape
    a, b = W.dd_uniform(m * k, seed=m + k), W.dd_uniform(k * n, seed=n + 7)
    got = to_host(api.matmuldd_mm(to_dev(a, dev), to_dev(b, dev), m, k, n, ri))
    assert O.same_bits(got, O.matmul_mm(a, b, m, k, n, ri)).all()


@pytest.mark.parametrize("shape", CPLX)
@pytest.mark.parametrize("ri", [8, 3])
def test_complex_tiles(dev, shape, ri):
    m, k, n = shape
    a, b = W.dd_uniform(2 * m * k, seed=m), W.dd_uniform(2 * k * n, seed=n)
    got = to_host(api.cmatmuldd_mm(to_dev(a, dev), to_dev(b, dev), m, k, n, ri))
    assert O.same_bits(got, O.cmatmul_mm(a, b, m, k, n, ri)).all()


@pytest.mark.parametrize("shape", [(250, 40, 300), (381, 33, 384), (960, 9, 639)])
def test_real_tiles_unaligned(dev, shape):
    m, k, n = shape
    a, b = W.dd_uniform(m * k, seed=1), W.dd_uniform(k * n, seed=2)
    da, db = (to_dev(np.concatenate([[0.0], x]), dev)[1:] for x in (a, b))
    got = to_host(api.matmuldd_mm(da, db, m, k, n, 8))
    assert O.same_bits(got, O.matmul_mm(a, b, m, k, n, 8)).all()


MATVEC = [(1, 1), (31, 7), (33, 32), (40, 33), (65, 64), (130, 259), (148 * 32, 65), (148 * 32 + 5, 97),
          (70, 8 * 32), (70, 16 * 32 + 1)]


@pytest.mark.parametrize("shape", MATVEC)  # one wave of CTAs up to 148 * 32 outputs, two CTAs per SM beyond
@pytest.mark.parametrize("ri", [8, 0, 5, 24])
@pytest.mark.parametrize("off", [0, 1])
def test_matvec_stages(dev, shape, ri, off):
    m, k = shape
    a, x = W.dd_uniform(m * k, seed=m), W.dd_uniform(k, seed=k + 3)
    da, dx = (to_dev(np.concatenate([np.zeros(off), v]), dev)[off:] for v in (a, x))
    assert O.same_bits(to_host(api.matmuldd_mv(da, dx, m, k, ri)), O.matmul_mv(a, x, m, k, ri)).all()
    assert O.same_bits(to_host(api.matmuldd_vm(dx, da, k, m, ri)), O.matmul_vm(x, a, k, m, ri)).all()
