"""The boxcar filter on large scenes against the same filter on pieces of them.

Large scenes with windows up to 7 x 7 are walked by warps, small ones go
through staged tiles.  Both add a window's values in the same order, counted
from columns and rows that are multiples of four, so a piece cut at such an
origin has to give the same bits wherever its windows see no cut edge.
"""
import pytest
import torch

import despeckcl_b200 as dcl

pytestmark = pytest.mark.gpu


def _spans(n, piece, r):
    """(start, stop, first valid, last valid + 1) of pieces that cover n."""
    a = 0
    while True:
        b = min(n, a + piece)
        yield a, b, (a if a == 0 else a + r), (n if b == n else b - r - 1)
        if b == n:
            return
        a = b - 4 * ((2 * r + 8) // 4 + 1) & ~3


# rows of whole vectors and not, a single warp of columns, fewer rows than a walk's
@pytest.mark.parametrize("h,w,offset", [(2304, 2292, 0), (2304, 2292, 1), (2291, 2293, 0), (3, 1800000, 0), (60001, 92, 0),
                                        (1400009, 4, 0), (41, 131201, 0)])
def test_walk_matches_tiles(h, w, offset):
    gen = torch.Generator(device="cuda").manual_seed(h)
    flat = torch.rand(3 * h * w + offset, generator=gen, device="cuda")
    planes = [flat[offset + k * h * w:offset + (k + 1) * h * w].view(h, w) for k in range(3)]
    planes[2].mul_(6.28).sub_(3.14)
    planes[0][h // 2, w // 2] = float("inf")
    planes[1][h // 3, w // 3] = float("nan")
    planes[0][:2, :3] = 0
    planes[1][:2, :3] = 0
    for window in (3, 5, 7):
        r = window // 2
        got = dcl.boxcar_device(*planes, window)
        for y0, y1, ya, yb in _spans(h, 1200, r):
            for x0, x1, xa, xb in _spans(w, 1600, r):
                part = dcl.boxcar_device(*(p[y0:y1, x0:x1].contiguous() for p in planes), window)
                for g, p in zip(got, part):
                    g, p = g[ya:yb, xa:xb], p[ya - y0:yb - y0, xa - x0:xb - x0]
                    assert torch.equal(g.contiguous().view(torch.int32), p.contiguous().view(torch.int32)) or \
                        bool(((g == p) | (g.isnan() & p.isnan())).all()), (window, y0, x0)
