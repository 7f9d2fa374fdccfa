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
