"""Prepared batches on the fused kernel: every instantiation, the autotuner and
its cache file, against the two kernels that batches run by default.  The
launches of a run tell which kernels it is: one for the fused kernel, two or
more for the others, after the frame kernels."""
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import synthetic  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ARGS = (21, [3, 5, 7], [1, 3])
SHAPES = [(70, 40), (129, 257), (32, 33)]


@pytest.fixture(scope="module")
def stats():
    return dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), *ARGS[1:])


@pytest.fixture(scope="module")
def scenes():
    return [tuple(torch.from_numpy(x).cuda() for x in synthetic.insar_scene(h, w, 50 + i))
            for i, (h, w) in enumerate(SHAPES)]


def _run(b):
    out = [o.cpu().numpy() for scene in b.run() for o in scene]
    torch.cuda.synchronize()
    return out


@pytest.fixture(scope="module")
def want(scenes, stats):
    b = dcl.NlsarBatch(scenes, *ARGS, stats, graph=False, autotune=False)
    assert not b.fused and b.launches >= len(SHAPES) * 3 + 2
    out = _run(b)
    b.close()
    return out


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("variant,autotune", [(0, False), (1, False), (2, False), (0, True)])
def test_fused_batches_equal_the_two_kernels(graph, variant, autotune, scenes, stats, want):
    b = dcl.NlsarBatch(scenes, *ARGS, stats, graph=graph, autotune=autotune, variant=variant)
    assert b.fused and b.launches == len(SHAPES) * 3 + 1
    assert b.variant in (0, 1, 2) if autotune else b.variant == variant
    for _ in range(2):
        for g, w in zip(_run(b), want):
            np.testing.assert_array_equal(g, w)
    b.close()


PROGRAM = """
import torch
import despeckcl_b200 as dcl
from despeckcl_b200 import synthetic

st = dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), [3, 5, 7], [1, 3])
a = [torch.from_numpy(x).cuda() for x in synthetic.insar_scene(90, 118, 1)]
b = dcl.NlsarBatch([tuple(a)], 21, [3, 5, 7], [1, 3], st, graph=True, autotune=True, variant=0)
out = b.run()[0]
one = dcl.nlsar_insar_device(*a, 21, [3, 5, 7], [1, 3], st, select_mode="argmax_enl")
torch.cuda.synchronize()
print(b.fused, b.variant, all(torch.equal(x, y) for x, y in zip(out, one)))
"""


def test_autotuner_cache_file(tmp_path):
    path = tmp_path / "tune.txt"

    def run():
        out = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, cwd=ROOT, timeout=300,
                             env=dict(os.environ, DESPECKCL_B200_TUNE_CACHE=str(path)))
        assert out.returncode == 0, out.stdout + out.stderr
        fused, variant, same = out.stdout.split()
        assert fused == same == "True"
        return int(variant)

    first = run()  # times the instantiations and writes the choice
    key, kept = path.read_text().split()
    assert int(kept) == first
    for planted in (0, 1, 2):  # a later process takes what the file says
        path.write_text(f"{key} {planted}\n")
        assert run() == planted
