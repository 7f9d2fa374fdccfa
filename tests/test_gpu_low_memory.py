"""Calls whose usual scratch cannot be had: with the device's stream-ordered pool
limited in size (in a process of its own) NL-SAR takes smaller volumes of weight
codes, then the fused kernel, and NL-InSAR evaluates its similarities in every
pass; the results are the same bits."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes
import numpy as np
import torch
import despeckcl_b200 as dcl
from despeckcl_b200 import api, synthetic

cu = ctypes.CDLL("libcuda.so.1")


class Props(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("locationType", ctypes.c_int),
                ("locationId", ctypes.c_int), ("win32", ctypes.c_void_p), ("maxSize", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


def use_pool(mib):
    pool, dev = ctypes.c_void_p(), torch.cuda.current_device()
    props = Props(1, 0, 1, dev, None, mib << 20, 0)
    assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
    assert cu.cuDeviceSetMemPool(dev, pool) == 0
    return pool


BENCH = ([3, 5, 7], [1, 3])
a = synthetic.insar_scene(500, 601, 3)
d = [torch.from_numpy(x).cuda() for x in a]
small = [x[:150, :170].contiguous() for x in d]
st = dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), *BENCH)
rng = np.random.default_rng(1)
z = rng.normal(size=(3, 180, 290)) + 1j * rng.normal(size=(3, 180, 290))
cov = (z[:, None] * z[None].conj()).astype(np.complex64)
st3 = dcl.nlsar_train(cov[:, :, :64, :64], *BENCH)


def launches(call):
    ms, groups, n = ctypes.c_double(), ctypes.c_long(), ctypes.c_long()
    api.lib().dcl_profile_begin()
    out = [np.asarray(o.cpu()) if hasattr(o, "cpu") else np.asarray(o) for o in call()]
    torch.cuda.synchronize()
    api._check(api.lib().dcl_profile_end(ctypes.byref(ms), ctypes.byref(groups), ctypes.byref(n)))
    return out, n.value


calls = {
    "device": lambda: dcl.nlsar_insar_device(*d, 21, *BENCH, st, select_mode="argmax_enl"),
    "host": lambda: dcl.nlsar_insar(*a, 21, *BENCH, st, select_mode="argmax_enl"),
    "general": lambda: dcl.nlsar_insar_device(*d, 15, *BENCH, st, select_mode="argmax_enl"),
    "3x3": lambda: [dcl.nlsar(cov, 21, *BENCH, st3, select_mode="argmax_enl").view(np.float32)],
    "nlinsar": lambda: dcl.nlinsar_device(*small, 21, 7, 3, 10),
}
for name, caps in (("device", (448, 160, 64, 32)), ("host", (480, 192, 64, 32)), ("general", (288, 160, 64, 32)),
                   ("3x3", (416, 160, 96, 32)), ("nlinsar", (128,))):
    default = ctypes.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(default), torch.cuda.current_device()) == 0
    assert cu.cuDeviceSetMemPool(torch.cuda.current_device(), default) == 0
    want, n = launches(calls[name])
    counts = [n]
    for mib in caps:
        pool = use_pool(mib)
        got, n = launches(calls[name])
        counts.append(n)
        for g, w in zip(got, want):
            assert np.array_equal(g, w, equal_nan=True), (name, mib)
        assert cu.cuDeviceSetMemPool(torch.cuda.current_device(), default) == 0
        torch.cuda.synchronize()
        assert cu.cuMemPoolDestroy(pool) == 0
    print(name, *counts)
"""


def test_smaller_scratch_gives_the_same_bits():
    out = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    counts = {line.split()[0]: [int(x) for x in line.split()[1:]] for line in out.stdout.splitlines()}
    assert len(counts) == 5
    for name, n in counts.items():
        if name != "nlinsar":
            assert max(n) > n[0], (name, n)   # several segments
            assert min(n) < n[0], (name, n)   # the fused or general kernel
