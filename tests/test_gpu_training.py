"""Edges of the training kernels against the oracle: few and many patches (one
block to several in each direction), patches clamped at the far edges, and
pixels whose dissimilarities are not finite, which the LUT drops.

Tolerances as for the 128 x 128 area: extremes within 1e-5 relative, a LUT
entry within five pairs of the oracle's (a value within rounding of a
threshold may count on either side)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import synthetic  # noqa: E402


@pytest.mark.parametrize("size,patches,scales", [(4, [3], [1]), (12, [3], [9]), (33, [1, 15], [7]), (35, [3, 11], [1, 5]),
                                                 (130, [3], [3])])
@pytest.mark.parametrize("broken", [False, True])
def test_training_edges_match_oracle(oracle, size, patches, scales, broken):
    a = [x.copy() for x in synthetic.training_area(size, seed=size)]
    if broken:
        a[0][size // 2, size // 3] = np.inf
        a[2][size - 1, 0] = np.nan
    mine = dcl.nlsar_train_insar(*a, patches, scales)
    ref = oracle.training_insar(*a, patches, scales)
    assert sorted(mine.keys()) == sorted(ref.keys())
    for k in ref:
        x, y = mine[k], ref[k]
        n = size - k[1] + 1
        patches_n = (-(-n // k[0])) ** 2
        npairs = patches_n * (patches_n - 1) // 2
        assert x.dissims_min == pytest.approx(y.dissims_min, rel=1e-5, abs=1e-5)
        assert x.dissims_max == pytest.approx(y.dissims_max, rel=1e-5)
        assert np.abs(x.quantilles - y.quantilles).max() <= 5.0 / npairs + 1e-7
        np.testing.assert_array_equal(x.chi2cdf_inv, y.chi2cdf_inv)
