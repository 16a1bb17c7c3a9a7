"""Cache of the batch autotuner: winners are read back by another process, and those
that were timed on former kernels (entries without the generation number) decide
nothing.  Each plan is made in a process of its own, as the cache is read once."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

_CHILD = r"""
import sys
sys.path[:0] = [{root!r}]
import torch
from multifloats_b200 import api
m, k, n, count = {shape!r}
t = lambda e: torch.ones(2 * e, dtype=torch.float64, device="cuda")
probs = [(t(m * k), t(k * n), t(m * n), m, k, n) for _ in range(count)]
with api.GemmBatch(probs, form={form!r}, tune={tune!r}) as plan:
    print({{api.lib().mfcuda_batch_config(plan._plan, i) for i in range(count)}}.pop())
"""


def _config(path, form, shape, tune=False):
    proc = subprocess.run([sys.executable, "-c", _CHILD.format(root=ROOT, shape=shape, form=form, tune=tune)],
                          env=dict(os.environ, MFCUDA_AUTOTUNE_CACHE=str(path)), capture_output=True, text=True,
                          timeout=300)
    assert proc.returncode == 0, proc.stderr[-2000:]
    return int(proc.stdout.split()[-1])


def _entries(path):
    return dict(line.split() for line in path.read_text().splitlines())


# (form, shape, a configuration that the heuristic does not choose: as stored, as reported)
CASES = [("plain", (300, 40, 300, 40), "0", 64), ("split", (100, 100, 300, 4), "64", 64), ("crt", (100, 100, 300, 4), "64", 64)]


@pytest.mark.parametrize("form,shape,stored,reported", CASES)
def test_former_winners_are_ignored(dev, tmp_path, form, shape, stored, reported):
    fresh, planted = tmp_path / "fresh.txt", tmp_path / "planted.txt"
    heuristic = _config(tmp_path / "none.txt", form, shape)
    assert heuristic != reported
    _config(fresh, form, shape, tune=True)
    (key, _), = _entries(fresh).items()
    planted.write_text(f"{key} {stored}\n")  # a winner of these kernels is used
    assert _config(planted, form, shape) == reported
    former = key.rsplit(":", 1)[0]  # one from before is not
    assert former.count(":") == 4
    planted.write_text(f"{former} {stored}\n")
    assert _config(planted, form, shape) == heuristic
    _config(planted, form, shape, tune=True)
    assert set(_entries(planted)) == {key, former}


@pytest.mark.parametrize("stored", ["0", "1"])
def test_winner_whose_tiles_outlast_the_batch(dev, tmp_path, stored):
    """Two products of 100 x 2000 x 100: a tile of 64 or 32 runs its k loop alone
    when the SMs have long finished the rest, whatever won for the bucket."""
    fresh, planted = tmp_path / "fresh.txt", tmp_path / "planted.txt"
    shape = (100, 2000, 100, 2)
    _config(fresh, "plain", shape, tune=True)
    (key, _), = _entries(fresh).items()
    planted.write_text(f"{key} {stored}\n")
    assert _config(planted, "plain", shape) == _config(tmp_path / "none.txt", "plain", shape) == 16
