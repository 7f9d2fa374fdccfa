"""A kernel whose grid the device refuses fails its call: in a process's first
calls too, where shared-memory limits are set between a call's launches (which
clears the thread's last error)."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# frames of more than 8 * 65535 rows exceed the grid of the kernels that fill them
PROGRAM = """
import sys
import torch
import despeckcl_b200 as dcl
from despeckcl_b200 import synthetic

st = dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), [3, 5], [1])
a = [torch.from_numpy(x).cuda() for x in synthetic.insar_scene(600000, 1, 3)]
calls = {
    "device 21": lambda: dcl.nlsar_insar_device(*a, 21, [3], [1], {k: v for k, v in st.items() if k == (3, 1)}),
    "device 5": lambda: dcl.nlsar_insar_device(*a, 5, [3, 5], [1], st, select_mode="argmax_enl"),
    "batch": lambda: dcl.nlsar_insar_batch_device([tuple(a)], 3, [3], [1], st),
    "prepared": lambda: dcl.NlsarBatch([tuple(a)], 21, [3], [1], st, graph=True, autotune=False),
}
try:
    calls[sys.argv[1]]()
except dcl.DespeckclError as e:
    assert e.code == (-4 if sys.argv[1] != "prepared" else -1) and "invalid configuration" in str(e), e
    print("refused")
# the refused call leaves the next one as it was
out = dcl.nlsar_insar_device(*[x[:300] for x in a], 21, [3], [1], st)
torch.cuda.synchronize()
assert bool(torch.isfinite(out[0]).all())
"""


@pytest.mark.parametrize("call", ["device 21", "device 5", "batch", "prepared"])
def test_refused_grids_fail_the_call(call):
    out = subprocess.run([sys.executable, "-c", PROGRAM, call], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "refused"
