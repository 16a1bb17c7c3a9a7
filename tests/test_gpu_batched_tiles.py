"""GPU parity of split batches where the grouped tensor-core kernels can go wrong:
edges of the tiles (64, 128, 256 columns, 128 rows), even and odd slice counts
(the digit form takes two diagonals per item), several K blocks and K chunks,
more items than CTAs, empty products.  Every result equals the oracle bit for
bit."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (127, 129, 63), (128, 128, 64), (129, 1, 65), (33, 300, 127), (200, 127, 128), (17, 257, 129),
          (130, 64, 255), (140, 385, 257), (256, 40, 513), (0, 5, 7), (5, 0, 9)]


def _run(dev, shapes, form, slices, R=0):
    import torch

    host, probs = [], []
    for i, (m, k, n) in enumerate(shapes):
        if R:
            a, b = W.dd_rowcol_scaled(m, k, R, "row", i), W.dd_rowcol_scaled(k, n, R, "col", i + 99)
        else:
            a, b = W.dd_uniform(m * k, seed=i), W.dd_uniform(k * n, seed=i + 99)
        host.append((a, b))
        c = torch.full((2 * m * n,), 7.0, dtype=torch.float64, device=dev)
        probs.append((to_dev(a, dev), to_dev(b, dev), c, m, k, n))
    with api.GemmBatch(probs, form=form, slices=slices) as plan:
        kc = api.lib().mfcuda_batch_kchunk(plan._plan)
        for _ in range(2):  # the item counter starts again
            plan.run()
        assert plan.status() == 0
        out = [to_host(p[2]) for p in probs]
    return host, out, kc


@pytest.mark.parametrize("extra", [[], [(900, 5, 1000)] * 12])  # alone, and beside short-k work for every SM
def test_plain_tiles(dev, extra):
    shapes = SHAPES + [(40, 700, 30), (23, 9, 60)] + extra
    host, out, _ = _run(dev, shapes, "plain", 0)
    for (m, k, n), (a, b), got in zip(shapes, host, out):
        assert O.same_bits(got, O.matmul_mm(a, b, m, k, n, 8)).all(), (m, k, n)


@pytest.mark.parametrize("slices", [0, 2, 3, 13])
def test_digit_tiles(dev, slices):
    host, out, kc = _run(dev, SHAPES, "split", slices)
    for (m, k, n), (a, b), got in zip(SHAPES, host, out):
        if m * n and k:
            want, _ = O.split_gemm(a, b, m, k, n, slices=slices, kc=kc)
            assert O.same_bits(got, want).all(), (m, k, n)
        else:
            assert not got.any()


@pytest.mark.parametrize("bits", [0, 40])
def test_crt_tiles(dev, bits):
    host, out, _ = _run(dev, SHAPES, "crt", bits, R=8)
    for (m, k, n), (a, b), got in zip(SHAPES, host, out):
        if m * n and k:
            want, _ = O.crt_gemm(a, b, m, k, n, bits=bits)
            assert O.same_bits(got, want).all(), (m, k, n)
        else:
            assert not got.any()


def test_many_items(dev):
    rng = np.random.default_rng(3)
    shapes = [tuple(int(v) for v in rng.integers(1, 150, 3)) for _ in range(400)]
    host, out, kc = _run(dev, shapes, "split", 0)
    for (m, k, n), (a, b), got in list(zip(shapes, host, out))[::7]:
        want, _ = O.split_gemm(a, b, m, k, n, kc=kc)
        assert O.same_bits(got, want).all(), (m, k, n)


# where loads, MMAs and drain stop: rows 32 / 64, columns 32 / 64 of a tile, K steps
# of 32 of the last block; large problems first, so that the rings hold their tiles
TRIM = [(200, 300, 300), (31, 31, 31), (32, 32, 32), (33, 33, 33), (64, 96, 64), (65, 97, 65), (63, 129, 95),
        (96, 160, 96), (97, 161, 97), (128, 64, 160), (129, 65, 161), (160, 128, 288), (161, 95, 289), (192, 1, 193)]


@pytest.mark.parametrize("form", ["split", "crt"])
def test_trimmed_tiles(dev, form):
    host, out, kc = _run(dev, TRIM, form, 0, R=3)
    for (m, k, n), (a, b), got in zip(TRIM, host, out):
        want, _ = O.split_gemm(a, b, m, k, n, kc=kc) if form == "split" else O.crt_gemm(a, b, m, k, n)
        assert O.same_bits(got, want).all(), (m, k, n)
