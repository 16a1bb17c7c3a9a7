"""The library's workspace pool: calls of several threads on their own streams
share it and keep their results, and what it holds after a synchronisation is
bounded (4 GiB)."""
import threading

import pytest

from conftest import to_dev, to_host
from multifloats_b200 import api
from multifloats_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_threads_and_streams(dev):
    import torch

    shapes = [(300, 200, 520), (257, 700, 300), (96, 130, 64), (600, 128, 130)]
    jobs, want, got = [], [], [None] * len(shapes)
    for i, (m, k, n) in enumerate(shapes):
        a, b = W.dd_rowcol_scaled(m, k, 8, "row", i), W.dd_rowcol_scaled(k, n, 8, "col", i + 50)
        jobs.append((to_dev(a, dev), to_dev(b, dev), m, k, n))
        want.append(O.crt_gemm(a, b, m, k, n)[0])
    torch.cuda.synchronize()

    def work(i):
        s = torch.cuda.Stream(device=dev)
        with torch.cuda.stream(s):
            outs = [api.matmuldd_mm_crt(*jobs[i])[0] for _ in range(6)]
            d = api.dot_product(jobs[i][0], jobs[i][0])
            s.synchronize()
            got[i] = [to_host(o) for o in outs], to_host(d)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, (outs, d) in enumerate(got):
        assert all(O.same_bits(o, want[i]).all() for o in outs), i
        a = to_host(jobs[i][0])
        assert O.same_bits(d, O.reduce_blocked("dot", a, a)).all(), i


def test_held_memory_is_bounded(dev):
    import torch

    n = 7168  # a workspace of more than 4 GiB
    a = torch.ones(2 * n * n, dtype=torch.float64, device=dev)
    c = torch.empty_like(a)
    a[1::2] = 0.0
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(dev)[0]
    api.matmuldd_mm_crt(a, a, n, n, n, out=c)
    torch.cuda.synchronize()
    api.sum_dd(a[:20000])  # a small workspace, and the synchronisation after it
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info(dev)[0]
    assert held <= (4 << 30) + (256 << 20), held
    assert float(c[0]) == n
