"""GPU parity of the elementwise maps where their kernels change form: operands
whose reduced argument leaves the range the polynomials' fast form is valid for
(low limbs that are not small, |x| up to 2^55), results next to the overflow and
underflow limits, the borders of the log intervals, zeros of either sign and
non-finite limbs.  Every output equals the oracle bit for bit."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _interleave(hi, lo):
    out = np.empty(2 * hi.size)
    out[0::2], out[1::2] = hi, lo
    return out


def _inputs(op):
    r = np.random.default_rng(11)
    n = 4000
    lo_rel = r.uniform(-1, 1, n) * 2.0 ** -53
    parts = []

    def add(hi, lo=None):
        hi = np.asarray(hi, dtype=np.float64)
        parts.append(_interleave(hi, hi * lo_rel[: hi.size] if lo is None else np.broadcast_to(lo, hi.shape)))

    core = {"exp": 700.0, "exp2": 1000.0, "sin": 1e6, "cos": 1e6}.get(op)
    x = r.uniform(-core, core, n) if core else np.exp2(r.uniform(-1000, 1000, n))
    add(x)
    # unnormalised: the low limb up to the size of the high one, or far above it
    add(x[:500], x[:500] * r.uniform(-1, 1, 500))
    add(x[:500], x[:500] * np.exp2(r.uniform(-52, 3, 500)))
    if op not in ("exp", "exp2"):  # there the reference converts an out-of-range double to int: undefined in C
        add(x[:50], 1e10)
    add(x[:20], np.inf)
    add(x[:20], np.nan)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2e-308, -2.2e-308,
                        1.7976931348623157e308, -1.7976931348623157e308])
    for lo in (0.0, -0.0, 5e-324):
        add(special, lo)
    if op in ("exp", "exp2"):
        c = 1.0 if op == "exp2" else np.log(2)
        for edge in (1024.0, -1021.0, -1022.0, -1060.0, -1074.0, -1075.0):
            add(edge * c + r.uniform(-1.5, 1.5, 400))
        add((np.arange(-300, 300) + 0.5) / 256 * c)  # ties of the table index
    elif op in ("sin", "cos"):
        add(np.exp2(r.uniform(30, 55.2, 1000)) * r.choice([-1.0, 1.0], 1000))
        add((np.arange(-200, 200) * (np.pi / 8)) + r.uniform(-1e-15, 1e-15, 400))
        add(np.exp2(r.uniform(-1060, -20, 300)))
    else:
        for edge in (15 / 16, 17 / 16, 1.0):
            add(edge + r.uniform(-1e-3, 1e-3, 400))
            add(np.nextafter(edge, [0.0, 2.0]))
        add(1 + np.arange(0, 33) / 32)
        add(np.exp2(r.uniform(-1074, -1022, 300)))
        add(-np.abs(x[:20]))
    return np.concatenate(parts)


@pytest.mark.parametrize("op", ["exp", "log", "sin", "cos", "sqrt", "exp2", "log2", "log10"])
def test_edges(dev, op):
    x = _inputs(op)
    got = to_host(api.unary(op, to_dev(x, dev)))
    same = O.same_bits(got, O.unary(op, x))
    assert same.all(), x.reshape(-1, 2)[~same][:8]


def test_pair_edges(dev):
    x = _inputs("sin")
    s, c = api.sincos(to_dev(x, dev))
    assert O.same_bits(to_host(s), O.unary("sin", x)).all()
    assert O.same_bits(to_host(c), O.unary("cos", x)).all()


# sizes around a warp, a block and one pass of the grid (148 SMs x 16 blocks of
# 256); shares of arguments next to one from none to all, so that both queues of
# a warp fill, overflow and are emptied with 1 to 31 arguments left
@pytest.mark.parametrize("op", ["log", "log2", "log10"])
@pytest.mark.parametrize("n, share", [(1, 1.0), (31, 0.5), (33, 0.5), (257, 0.03), (4099, 0.97), (1300001, 0.0),
                                      (1300001, 0.1), (1300001, 0.6), (1300001, 1.0)])
def test_log_mixed(cuda_lib, dev, op, n, share):
    import ctypes as C

    import torch

    r = np.random.default_rng(n)
    hi = np.where(r.uniform(size=n) < share, r.uniform(0.94, 1.06, n), np.exp2(r.uniform(-40, 40, n)))
    x = _interleave(hi, hi * r.uniform(-1, 1, n) * 2.0 ** -53)
    want = O.unary(op, x)
    assert O.same_bits(to_host(api.unary(op, to_dev(x, dev))), want).all()
    off = to_dev(np.concatenate([[0.0], x]), dev)[1:]  # 8-byte aligned
    assert O.same_bits(to_host(api.unary(op, off)), want).all()
    if op == "log":  # ragged: pieces of 0 to 1000 elements of the same array
        d, y = to_dev(x, dev), torch.zeros(2 * n, dtype=torch.float64, device=dev)
        cuts = np.unique(np.concatenate([[0, n], r.integers(0, n + 1, 1 + n // 500)]))
        lens = np.diff(cuts).tolist()
        cnt = len(lens)
        X = (C.c_void_p * cnt)(*[d.data_ptr() + 16 * int(c) for c in cuts[:-1]])
        Y = (C.c_void_p * cnt)(*[y.data_ptr() + 16 * int(c) for c in cuts[:-1]])
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert cuda_lib.mfcuda_unary_dd_ragged(1, X, Y, (C.c_int64 * cnt)(*lens), cnt, s) == 0
        assert O.same_bits(to_host(y), want).all()
