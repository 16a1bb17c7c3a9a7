"""Workspace sizes of the split forms: pure arithmetic (no device is asked), and a
workspace for one shape is large enough for every shape that is no larger in any
extent, also where the width of the tiles differs between the two."""
import random

import pytest

SHAPES = [(1309, 97, 666), (1281, 512, 513), (1500, 2500, 700), (2048, 2048, 2048), (4096, 128, 900), (600, 20000, 600),
          (130, 300, 5000)]
SMALLER = [(1028, 97, 591), (1100, 512, 513), (1100, 2500, 600), (1800, 2000, 1700), (3000, 100, 800), (520, 9000, 520),
           (129, 300, 4700)]


@pytest.mark.parametrize("large,small", list(zip(SHAPES, SMALLER)))
def test_known_shapes(cuda_lib, large, small):
    assert cuda_lib.mfcuda_split_workspace_size(*small) <= cuda_lib.mfcuda_split_workspace_size(*large)
    for bits in (0, 60, 92):
        assert (cuda_lib.mfcuda_crt_workspace_size(*small, bits) <= cuda_lib.mfcuda_crt_workspace_size(*large, bits)
                <= cuda_lib.mfcuda_crt_workspace_size(*large, 0))


def test_monotone_in_every_extent(cuda_lib):
    rng = random.Random(7)
    fns = [cuda_lib.mfcuda_split_workspace_size] + [
        lambda m, k, n, b=b: cuda_lib.mfcuda_crt_workspace_size(m, k, n, b) for b in (0, 8, 77, 110)]
    for _ in range(3000):
        big = [int(round(2 ** rng.uniform(0, 13))) for _ in range(3)]
        small = [rng.randint(v - v // 4, v) for v in big]
        for fn in fns:
            assert fn(*small) <= fn(*big), (small, big)
