"""Host-pointer calls staged through pinned blocks (pageable planes, 8 MiB or
more in all) against the device entry point: the same bits with planes that end
on and next to a slot's end, 8-plane covariances, a thread per call, and more
calls at the same time than there are blocks."""
import ctypes
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import api, synthetic  # noqa: E402

ARGS = (21, [3], [1])


@pytest.fixture(scope="module")
def stats():
    return dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), *ARGS[1:])


def _pair(shape, seed, stats):
    a = synthetic.insar_scene(*shape, seed)
    want = dcl.nlsar_insar_device(*[torch.from_numpy(x).cuda() for x in a], *ARGS, stats)
    torch.cuda.synchronize()
    return a, [w.cpu().numpy() for w in want]


def _same(got, want):
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


# a plane is one slot (4 MiB), one row more, a little less, and several slots
@pytest.mark.parametrize("shape", [(1024, 1024), (1024, 1025), (1025, 1021), (500001, 3), (2100, 1801)])
def test_planes_around_a_slot(shape, stats):
    a, want = _pair(shape, 3, stats)
    _same(dcl.nlsar_insar(*a, *ARGS, stats), want)


def test_eight_planes(stats):
    a1, a2, ph = synthetic.insar_scene(520, 611, 4)
    z = a1 * a2 * np.exp(1j * ph)
    cov = np.array([[a1 * a1, z], [z.conj(), a2 * a2]]).astype(np.complex64)
    planes = np.stack([cov.real, cov.imag], 2).reshape(8, *a1.shape)
    c = torch.from_numpy(np.ascontiguousarray(planes)).cuda()
    out = torch.empty_like(c)
    pk, pp, npn = api._ints(ARGS[1])
    sk, sp, nsn = api._ints(ARGS[2])
    arr, n, keep = api._entries(stats)
    api._check(api.lib().dcl_nlsar_covmat_device(api._dptr(c), api._dptr(out), *a1.shape, 2, ARGS[0], pp, npn, sp, nsn,
                                                 arr, n, ctypes.c_float(15.0), ctypes.c_float(49.0), 0,
                                                 api._stream(None)))
    torch.cuda.synchronize()
    host = dcl.nlsar(cov, *ARGS, stats)
    np.testing.assert_array_equal(np.stack([host.real, host.imag], 2).reshape(planes.shape), out.cpu().numpy())


def test_threads_one_after_another_and_together(stats):
    jobs = [_pair((900 + i, 901), 10 + i, stats) for i in range(6)]
    done = []

    def call(a, want):
        for _ in range(2):
            _same(dcl.nlsar_insar(*a, *ARGS, stats), want)
        done.append(1)

    for a, want in jobs:
        t = threading.Thread(target=call, args=(a, want))
        t.start()
        t.join()
    ts = [threading.Thread(target=call, args=j) for j in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert len(done) == 2 * len(jobs)
