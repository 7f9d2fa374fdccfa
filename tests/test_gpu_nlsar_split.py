"""The two-kernel NL-SAR path (weight indices, then means) against the fused
tile kernel, which a prepared batch runs when one of its instantiations is
asked for: the same bits, at the edges of both kernels' tiles (blocks of at
most 45 x 120 weights, 16 x 32 means) and where a scene is filtered in several
segments of rows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import synthetic  # noqa: E402

_STATS = {}


def _stats(patches, scales):
    key = (tuple(patches), tuple(scales))
    if key not in _STATS:
        _STATS[key] = dcl.nlsar_train_insar(*synthetic.training_area(64, seed=7), patches, scales)
    return _STATS[key]


# one wide and one tall scene exceed the volume of a segment (2 GiB)
@pytest.mark.parametrize("shape", [(1, 1), (1, 40), (33, 1), (2, 17), (16, 32), (17, 33), (32, 107), (36, 88),
                                   (45, 120), (109, 141), (4300, 310), (150, 9001)])
@pytest.mark.parametrize("patches,scales", [([3, 5, 7], [1, 3]), ([7], [1]), ([3], [3])])
def test_two_kernel_path_equals_fused_kernel(shape, patches, scales):
    st = _stats(patches, scales)
    a = [torch.from_numpy(x).cuda() for x in synthetic.insar_scene(*shape, 77)]
    for mode in ("argmax_enl", "reference"):
        got = dcl.nlsar_insar_device(*a, 21, patches, scales, st, select_mode=mode)
        b = dcl.NlsarBatch([tuple(a)], 21, patches, scales, st, select_mode=mode, graph=False, autotune=False,
                           variant=1)
        want = b.run()[0]
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())
        b.close()


@pytest.mark.parametrize("shape", [(1, 1), (1, 33), (12, 18), (13, 32), (25, 107), (49, 131)])
@pytest.mark.parametrize("patches,scales", [([3, 5, 7], [1, 3]), ([3, 5, 7, 9, 11], [1, 3]), ([5], [1, 3])])
def test_two_kernel_3x3_path_equals_fused_kernel(shape, patches, scales, monkeypatch):
    # the staging switch of the timeout tests keeps calls on the fused kernels;
    # the 3x3 one has no staging copies to withhold
    def cov(h, w, seed):
        rng = np.random.default_rng(seed)
        z = rng.normal(size=(3, 5)) + 1j * rng.normal(size=(3, 5))
        x = rng.normal(size=(3, h * w)) + 1j * rng.normal(size=(3, h * w))
        k = (np.linalg.cholesky(z @ z.conj().T) @ x).reshape(3, h, w) * np.linspace(1, 2, w)
        return (k[:, None] * k[None, :].conj()).astype(np.complex64)

    key = ("3x3", tuple(patches), tuple(scales))
    if key not in _STATS:
        _STATS[key] = dcl.nlsar_train(cov(40, 40, 1), patches, scales)
    c = cov(*shape, 2)
    for mode in ("argmax_enl", "reference"):
        monkeypatch.delenv("DESPECKCL_B200_TEST_WITHHOLD_STAGING", raising=False)
        got = dcl.nlsar(c, 21, patches, scales, _STATS[key], select_mode=mode)
        monkeypatch.setenv("DESPECKCL_B200_TEST_WITHHOLD_STAGING", "1")
        want = dcl.nlsar(c, 21, patches, scales, _STATS[key], select_mode=mode)
        np.testing.assert_array_equal(got.view(np.float32), want.view(np.float32))


# one byte per weight: more than 2^30 of them in 2 GiB, so segments are cut by
# the 32-bit word offsets instead
@pytest.mark.parametrize("shape", [(2300, 2301), (5003, 1100)])
def test_segments_cut_by_word_offsets(shape):
    st = _stats([3, 5, 7], [1, 3])
    a = [torch.from_numpy(x).cuda() for x in synthetic.insar_scene(*shape, 78)]
    got = dcl.nlsar_insar_device(*a, 21, [3, 5, 7], [1, 3], st, select_mode="reference")
    b = dcl.NlsarBatch([tuple(a)], 21, [3, 5, 7], [1, 3], st, select_mode="reference", graph=False, autotune=False,
                       variant=1)
    want = b.run()[0]
    torch.cuda.synchronize()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy(), w.cpu().numpy())
    b.close()


# settings without a specialised fused kernel: other windows, patches {3,5};
# the staging switch keeps them on the general kernel, which has no staging
# copies to withhold.  Statistics of a larger patch than the call's make the
# reference's selection fall back to its first combination with alpha 0.
@pytest.mark.parametrize("search", [3, 5, 15, 21, 23, 39])
@pytest.mark.parametrize("patches,scales,trained", [([3, 5], [1, 3], [3, 5]), ([3, 5, 7], [1, 3], [3, 5, 7]),
                                                    ([5], [1, 3], [5]), ([3, 5, 7, 9, 11], [3], [3, 5, 7, 9, 11]),
                                                    ([3, 5], [3], [3, 5, 7]), ([9], [1], [9]), ([11], [3], [11])])
def test_other_settings_equal_general_kernel(search, patches, scales, trained, monkeypatch):
    st = _stats(trained, scales)
    shapes = [(1, 1), (2, 40), (33, 17), (71, 131)]
    scenes = [synthetic.insar_scene(*s, 5) for s in shapes]
    scenes[2][0][3:9, 2:12] = 0
    scenes[2][1][3:9, 2:12] = 0
    scenes[3][0][20, 30] = np.inf
    scenes[3][1][50, 100] = np.nan
    dev = [tuple(torch.from_numpy(x).cuda() for x in s) for s in scenes]
    covs = []
    for a1, a2, ph in scenes:
        z = a1 * a2 * np.exp(1j * ph)
        covs.append(np.array([[a1 * a1, z], [z.conj(), a2 * a2]]).astype(np.complex64))
    for mode in ("argmax_enl", "reference"):
        if search == 21 and (patches != [3, 5] or mode == "reference"):
            continue  # the specialised kernel's

        def attempt(call):
            try:
                return [np.asarray(o.cpu() if hasattr(o, "cpu") else o) for o in call()]
            except dcl.DespeckclError as e:  # the largest windows and patches have no room, either way
                assert "too large for shared memory" in str(e)
                return [np.zeros(0)]

        def run():
            args = (search, patches, scales, st)
            out = []
            for a in dev:
                out += attempt(lambda: dcl.nlsar_insar_device(*a, *args, select_mode=mode))
            out += attempt(lambda: [o for scene in dcl.nlsar_insar_batch_device(dev, *args, select_mode=mode)
                                    for o in scene])
            for s in scenes:
                out += attempt(lambda: dcl.nlsar_insar(*s, *args, select_mode=mode))
            for c in covs:
                out += attempt(lambda: [dcl.nlsar(c, *args, select_mode=mode).view(np.float32)])
            return out

        monkeypatch.delenv("DESPECKCL_B200_TEST_WITHHOLD_STAGING", raising=False)
        got = run()
        monkeypatch.setenv("DESPECKCL_B200_TEST_WITHHOLD_STAGING", "1")
        want = run()
        assert len(got) == len(want)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("search", [3, 5, 15, 21, 25])
@pytest.mark.parametrize("patches,scales", [([3, 5], [1, 3]), ([3, 5, 7], [1, 3]), ([9], [1]), ([3, 5, 7, 9, 11], [3])])
def test_other_3x3_settings_equal_general_kernel(search, patches, scales, monkeypatch):
    def cov(h, w, seed):
        rng = np.random.default_rng(seed)
        z = rng.normal(size=(3, 5)) + 1j * rng.normal(size=(3, 5))
        x = rng.normal(size=(3, h * w)) + 1j * rng.normal(size=(3, h * w))
        k = (np.linalg.cholesky(z @ z.conj().T) @ x).reshape(3, h, w) * np.linspace(1, 2, w)
        return (k[:, None] * k[None, :].conj()).astype(np.complex64)

    key = ("3x3", tuple(patches), tuple(scales))
    if key not in _STATS:
        _STATS[key] = dcl.nlsar_train(cov(40, 40, 1), patches, scales)
    for shape in ((1, 1), (2, 40), (33, 17), (71, 131) if search > 3 else (250, 270)):
        c = cov(*shape, 2)
        c[:, :, shape[0] // 2:, : shape[1] // 8] = 0
        for mode in ("argmax_enl", "reference"):
            out = []
            for switch in (False, True):
                if switch:
                    monkeypatch.setenv("DESPECKCL_B200_TEST_WITHHOLD_STAGING", "1")
                else:
                    monkeypatch.delenv("DESPECKCL_B200_TEST_WITHHOLD_STAGING", raising=False)
                try:
                    out.append(dcl.nlsar(c, search, patches, scales, _STATS[key], select_mode=mode).view(np.float32))
                except dcl.DespeckclError as e:  # the largest windows and patches have no room, either way
                    assert "too large for shared memory" in str(e)
                    out.append(np.zeros(0))
            np.testing.assert_array_equal(*out)
