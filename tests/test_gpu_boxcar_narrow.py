"""Which kernel takes a large scene: the walk's strips of 120 columns do not fit
narrow scenes, where it took four to six times the tiles' time.  A narrow scene
may take longer per pixel than a wide one, but not by that much; widths on both
sides of the rule's lines give the bits of the same columns in a wide scene."""
import pytest
import torch

import despeckcl_b200 as dcl

pytestmark = pytest.mark.gpu


def _planes(h, w, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    p = [torch.rand(h, w, generator=gen, device="cuda") for _ in range(3)]
    p[2].mul_(6.28).sub_(3.14)
    return p


def _best_ms(planes, window):
    out = tuple(torch.empty_like(p) for p in planes)
    best = float("inf")
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        for _ in range(4):
            dcl.boxcar_device(*planes, window, out=out)
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]) / 4)
    return best


# 12 Mpx each: with tiles 0.09 to 0.13 ms, walked 0.46 (40 columns) and 0.38 ms (118)
@pytest.mark.parametrize("h,w,window", [(314573, 40, 3), (314573, 40, 7), (106635, 118, 7)])
def test_narrow_scenes_are_not_walked(h, w, window):
    wide = _best_ms(_planes(4195, 3000, 1), window)
    narrow = _best_ms(_planes(h, w, 2), window)
    assert narrow < 2.5 * wide


@pytest.mark.parametrize("w", [476, 480, 1196, 1200, 1797, 2880, 2884])
def test_widths_around_the_rule(w):
    planes = _planes(5300000 // w + 1, 2884, w)
    cut = [p[:, :w].contiguous() for p in planes]
    for window in (3, 7):
        whole = dcl.boxcar_device(*planes, window)
        got = dcl.boxcar_device(*cut, window)
        cols = w - window if w < 2884 else w  # windows that do not see the cut
        for g, p in zip(got, whole):
            assert torch.equal(g[:, :cols].contiguous().view(torch.int32), p[:, :cols].contiguous().view(torch.int32))
