"""The volume of weight codes that NL-SAR calls hold: never more than its bound,
also where one row of tiles of a wide scene exceeds it, and the same results
where it is cut in rows and columns (DESPECKCL_B200_VOLUME_MIB caps it) or not
used at all."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import api, synthetic  # noqa: E402

CAP = "DESPECKCL_B200_VOLUME_MIB"
EXAMPLE = ([3, 5, 7, 9, 11], [1, 3, 5])
BENCH = ([3, 5, 7], [1, 3])
_STATS = {}


def _polsar(h, w, seed):
    rng = np.random.default_rng(seed)
    z = rng.normal(size=(3, 5)) + 1j * rng.normal(size=(3, 5))
    x = rng.normal(size=(3, h * w)) + 1j * rng.normal(size=(3, h * w))
    k = (np.linalg.cholesky(z @ z.conj().T) @ x).reshape(3, h, w) * np.linspace(1, 2, w)
    return (k[:, None] * k[None, :].conj()).astype(np.complex64)


def _stats(patches, scales, dim=2):
    key = (dim, tuple(patches), tuple(scales))
    if key not in _STATS:
        _STATS[key] = (dcl.nlsar_train_insar(*synthetic.training_area(128, seed=7), patches, scales) if dim == 2 else
                       dcl.nlsar_train(_polsar(64, 64, 1), patches, scales))
    return _STATS[key]


def _covmat_device(cov, search, patches, scales, st, mode):
    d, _, h, w = cov.shape
    planes = np.stack([cov.real, cov.imag], 2).reshape(2 * d * d, h, w)
    c = torch.from_numpy(np.ascontiguousarray(planes)).cuda()
    out = torch.empty_like(c)
    pk, pp, npn = api._ints(patches)
    sk, sp, nsn = api._ints(scales)
    arr, n, keep = api._entries(st)
    api._check(api.lib().dcl_nlsar_covmat_device(api._dptr(c), api._dptr(out), h, w, d, search, pp, npn, sp, nsn, arr,
                                                 n, ctypes.c_float(15.0), ctypes.c_float(49.0), api._mode(mode),
                                                 api._stream(None)))
    return out


class _PoolHigh:
    """Most memory in use at once in the device's stream-ordered pool."""

    HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH

    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), torch.cuda.current_device()) == 0
        zero = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, self.HIGH, ctypes.byref(zero)) == 0

    def read(self):
        v = ctypes.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, self.HIGH, ctypes.byref(v)) == 0
        return v.value


# one row of tiles is 2.6 GiB (example settings, InSAR), 2.6 GiB (8 planes) and
# 3.5 GiB (3x3); the frames take less than 0.45 GiB
@pytest.mark.parametrize("kind,shape,setting", [("insar", (24, 17000), EXAMPLE), ("cov2", (4, 17000), EXAMPLE),
                                                ("cov3", (8, 40000), BENCH)])
def test_wide_scenes_stay_within_the_volume(kind, shape, setting):
    st = _stats(*setting, dim=3 if kind == "cov3" else 2)
    if kind == "insar":
        a = [torch.from_numpy(x).cuda() for x in synthetic.insar_scene(*shape, 3)]
    elif kind == "cov2":
        a1, a2, ph = synthetic.insar_scene(*shape, 3)
        z = a1 * a2 * np.exp(1j * ph)
        c = np.array([[a1 * a1, z], [z.conj(), a2 * a2]]).astype(np.complex64)
    else:
        c = _polsar(*shape, 2)
    torch.cuda.synchronize()
    high = _PoolHigh()
    if kind == "insar":
        dcl.nlsar_insar_device(*a, 21, *setting, st, select_mode="argmax_enl")
    else:
        _covmat_device(c, 21, *setting, st, "argmax_enl")
    torch.cuda.synchronize()
    assert high.read() <= (2 << 30) + (460 << 20)


def _launches(call):
    ms, groups, n = ctypes.c_double(), ctypes.c_long(), ctypes.c_long()
    api.lib().dcl_profile_begin()
    out = call()
    torch.cuda.synchronize()
    api._check(api.lib().dcl_profile_end(ctypes.byref(ms), ctypes.byref(groups), ctypes.byref(n)))
    return out, n.value


# MiB of one tile and of the rows of tiles at these settings lie between the
# caps: 1 has no room for a tile (the fused or general kernel filters), 5 to 9
# cut rows of tiles in columns, 64 cuts the scene in rows; 3x3: 5 has no room
@pytest.mark.parametrize("search,patches,scales", [(21, *BENCH), (21, *EXAMPLE), (21, [5], [1]), (15, *BENCH),
                                                   (21, [3, 5], [1, 3])])
@pytest.mark.parametrize("shape", [(1, 700), (75, 601), (170, 333)])
def test_cut_volumes_give_the_same_bits(search, patches, scales, shape, monkeypatch):
    st = _stats(patches, scales)
    a = synthetic.insar_scene(*shape, 9)
    dev = [torch.from_numpy(x).cuda() for x in a]
    z = a[0] * a[1] * np.exp(1j * a[2])
    cov = np.array([[a[0] * a[0], z], [z.conj(), a[1] * a[1]]]).astype(np.complex64)

    def everything(mode):
        args = (search, patches, scales, st)
        out, n = _launches(lambda: list(dcl.nlsar_insar_device(*dev, *args, select_mode=mode)))
        out += [_covmat_device(cov, *args, mode)]
        out += dcl.nlsar_insar(*a, *args, select_mode=mode)
        b = dcl.NlsarBatch([tuple(dev), tuple(x[: shape[0] // 2 + 1].contiguous() for x in dev)], *args,
                           select_mode=mode, graph=False, autotune=False)
        out += [o for scene in b.run() for o in scene]
        torch.cuda.synchronize()
        out = [o.cpu().numpy() if hasattr(o, "cpu") else o for o in out]
        b.close()
        return out, n

    for mode in ("argmax_enl", "reference"):
        monkeypatch.delenv(CAP, raising=False)
        want, full = everything(mode)
        seen = set()
        for mib in (0, 1, 5, 9, 64):
            monkeypatch.setenv(CAP, str(mib))
            got, n = everything(mode)
            seen.add(n)
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g, w)
        assert min(seen) < full  # the kernels without a volume
        assert max(seen) > full or shape[0] == 1 or len(patches) == 1  # several segments


@pytest.mark.parametrize("search,patches,scales", [(21, *BENCH), (15, *BENCH), (21, [5], [1, 3])])
def test_cut_3x3_volumes_give_the_same_bits(search, patches, scales, monkeypatch):
    st = _stats(patches, scales, dim=3)
    c = _polsar(77, 260, 4)
    for mode in ("argmax_enl", "reference"):
        monkeypatch.delenv(CAP, raising=False)
        want, full = _launches(lambda: _covmat_device(c, search, patches, scales, st, mode).cpu().numpy())
        seen = set()
        for mib in (0, 5, 13, 50):
            monkeypatch.setenv(CAP, str(mib))
            got, n = _launches(lambda: _covmat_device(c, search, patches, scales, st, mode).cpu().numpy())
            seen.add(n)
            np.testing.assert_array_equal(got, want)
            host = dcl.nlsar(c, search, patches, scales, st, select_mode=mode)
            planes = np.stack([host.real, host.imag], 2).reshape(want.shape)
            np.testing.assert_array_equal(planes, want)
        assert min(seen) < full < max(seen)
