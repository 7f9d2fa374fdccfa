"""The two-kernel NL-SAR path of the settings with a specialised fused kernel
(search window 21) against that kernel, which filters where no memory is given
to weight codes: the same bits for every pass shape, InSAR and 8-plane input,
on scenes with zero, tiny, huge, infinite and NaN pixels.  The launches of a call
tell which kernels filtered."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import api, synthetic  # noqa: E402

CAP = "DESPECKCL_B200_VOLUME_MIB"
_STATS = {}


def _stats(patches, scales):
    key = (tuple(patches), tuple(scales))
    if key not in _STATS:
        _STATS[key] = dcl.nlsar_train_insar(*synthetic.training_area(128, seed=7), patches, scales)
    return _STATS[key]


def _scene(h, w, seed, kind):
    a1, a2, ph = (x.copy() for x in synthetic.insar_scene(h, w, seed))
    y, x = h // 2, w // 2
    if kind == "zeros":
        a1[y:y + 9, x:x + 14] = 0
        a2[y:y + 9, x:x + 14] = 0
        a1[0, :5] = 0
        a2[-1, -1] = 0
    elif kind == "range":
        a1[y, x] = 1e-30
        a2[y, x] = 1e-30
        a1[y // 2, x // 2] = 1e19  # its square is finite, the product of two is not
        a2[y // 2, x // 2] = 3e19  # its square is not
        a1[-1, 0] = 1e-45
    elif kind == "inf":
        a1[y, x] = np.inf
        a2[1, 0] = np.inf
    elif kind == "nan":
        a1[y, x] = np.nan
        a2[0, -1] = np.nan
        ph[-1, x] = np.nan
    return a1, a2, ph


def _launches(call):
    ms, groups, n = ctypes.c_double(), ctypes.c_long(), ctypes.c_long()
    api.lib().dcl_profile_begin()
    out = call()
    torch.cuda.synchronize()
    api._check(api.lib().dcl_profile_end(ctypes.byref(ms), ctypes.byref(groups), ctypes.byref(n)))
    return out, n.value


def _both(call, monkeypatch):
    monkeypatch.delenv(CAP, raising=False)
    got, n = _launches(call)
    monkeypatch.setenv(CAP, "0")
    want, fused = _launches(call)
    assert n > fused
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


SETS = [([3, 5, 7], [1, 3]), ([3, 5, 7, 9, 11], [1, 3, 5]), ([3], [3]), ([5], [1, 3]), ([7], [1]), ([9], [3]),
        ([11], [1, 5])]
KINDS = ["plain", "zeros", "range", "inf", "nan"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("patches,scales", SETS)
def test_insar(patches, scales, kind, monkeypatch):
    st = _stats(patches, scales)
    args = (21, patches, scales, st)
    for shape in ((33, 33), (71, 131), (131, 70)):
        s = _scene(*shape, 5, kind)
        dev = [torch.from_numpy(x).cuda() for x in s]
        for mode in ("argmax_enl", "reference"):
            _both(lambda: [o.cpu().numpy() for o in dcl.nlsar_insar_device(*dev, *args, select_mode=mode)], monkeypatch)
    monkeypatch.setenv("DESPECKCL_B200_BANDS", "3")
    _both(lambda: list(dcl.nlsar_insar(*s, *args, select_mode="argmax_enl")), monkeypatch)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("patches,scales", SETS)
def test_eight_planes(patches, scales, kind, monkeypatch):
    st = _stats(patches, scales)
    for shape in ((33, 33), (71, 131), (131, 70)):
        a1, a2, ph = _scene(*shape, 6, kind)
        with np.errstate(all="ignore"):
            re, im, z = a1 * a2 * np.cos(ph), a1 * a2 * np.sin(ph), np.zeros_like(a1)
            planes = np.stack([a1 * a1, z, re, im, re, -im, a2 * a2, z])
        c = torch.from_numpy(planes).cuda()
        pk, pp, npn = api._ints(patches)
        sk, sp, nsn = api._ints(scales)
        arr, n, keep = api._entries(st)

        def call(mode):
            out = torch.empty_like(c)
            api._check(api.lib().dcl_nlsar_covmat_device(api._dptr(c), api._dptr(out), *shape, 2, 21, pp, npn, sp, nsn,
                                                         arr, n, ctypes.c_float(15.0), ctypes.c_float(49.0), mode,
                                                         api._stream(None)))
            return [out.cpu().numpy()]

        for mode in (0, 1):
            _both(lambda: call(mode), monkeypatch)


# 3x3: [3,5,7] and single sizes have a specialised kernel, [3,5] the general one
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("search,patches,scales", [(21, [3, 5, 7], [1, 3]), (21, [5], [3]), (21, [3, 5], [1, 3]),
                                                   (7, [3, 5, 7], [1])])
def test_3x3(search, patches, scales, kind, monkeypatch):
    def cov(h, w, seed):
        rng = np.random.default_rng(seed)
        z = rng.normal(size=(3, 5)) + 1j * rng.normal(size=(3, 5))
        x = rng.normal(size=(3, h * w)) + 1j * rng.normal(size=(3, h * w))
        k = (np.linalg.cholesky(z @ z.conj().T) @ x).reshape(3, h, w) * np.linspace(1, 2, w)
        return (k[:, None] * k[None, :].conj()).astype(np.complex64)

    key = ("3x3", tuple(patches), tuple(scales))
    if key not in _STATS:
        _STATS[key] = dcl.nlsar_train(cov(64, 64, 1), patches, scales)
    pk, pp, npn = api._ints(patches)
    sk, sp, nsn = api._ints(scales)
    arr, n, keep = api._entries(_STATS[key])
    for shape in ((33, 33), (71, 131)):
        x = cov(*shape, 2).reshape(9, *shape)
        planes = np.stack([x.real, x.imag], 1).reshape(18, *shape)
        v = {"plain": None, "zeros": 0.0, "range": 1e30, "inf": np.inf, "nan": np.nan}[kind]
        if v is not None:
            planes[:, shape[0] // 2, shape[1] // 2] = v
            planes[0, 0, 0] = v
            planes[16, -1, 3] = v
            planes[5, 7, -1] = v
        if kind == "zeros":
            planes[:, 3:9, 4:20] = 0
        c = torch.from_numpy(planes).cuda()

        def call(mode):
            out = torch.empty_like(c)
            api._check(api.lib().dcl_nlsar_covmat_device(api._dptr(c), api._dptr(out), *shape, 3, search, pp, npn, sp,
                                                         nsn, arr, n, ctypes.c_float(15.0), ctypes.c_float(49.0), mode,
                                                         api._stream(None)))
            return [out.cpu().numpy()]

        for mode in (0, 1):
            _both(lambda: call(mode), monkeypatch)
