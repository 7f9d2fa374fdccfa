"""Host-pointer calls whose planes go through pinned slots (pageable memory, 8
MiB or more in all) against the device entry point: the same bits, with planes
that end inside a slot, planes of several slots and calls from two threads."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import synthetic  # noqa: E402


@pytest.fixture(scope="module")
def stats():
    return dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), [3], [1])


def _check(shape, seed, stats, got=None):
    a = synthetic.insar_scene(*shape, seed)
    host = dcl.nlsar_insar(*a, 21, [3], [1], stats)
    dev = dcl.nlsar_insar_device(*[torch.from_numpy(x).cuda() for x in a], 21, [3], [1], stats)
    torch.cuda.synchronize()
    for h, d in zip(host, dev):
        np.testing.assert_array_equal(h, d.cpu().numpy())
    if got is not None:
        got.append(seed)


@pytest.mark.parametrize("shape", [(600, 583), (349526, 1), (1024, 2100), (1500, 1601)])
def test_staged_planes_equal_device_entry_point(shape, stats):
    _check(shape, 3, stats)


def test_staged_calls_from_two_threads(stats):
    got = []
    t = [threading.Thread(target=_check, args=((700, 701 + i), 10 + i, stats, got)) for i in range(2)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert sorted(got) == [10, 11]
