"""The chain passes at the sizes where their parts change over: label counts at
and around the shapes' widths (8 or 16 label pairs per lane, one or two units
per lane in the winner kernel), ranges of one chunk, of several, wider than the
shared-memory vectors and moving by any shift, and the diagonal left-right
check, each with byte terms and with u16 sums. Whole numbers: equal to the
oracle's on the emulator and on the GPU."""

from __future__ import annotations

import numpy as np
import pytest

from images import Rng, Texture, mismatch_report, random_image, render_pair, same_disparities
from regard3d_mvs_b200.types import LabelRanges, StereoOptions

BUILDS = ["simt_matcher", pytest.param("gpu_matcher", marks=pytest.mark.gpu)]


@pytest.mark.parametrize("build", BUILDS)
@pytest.mark.parametrize("p2", [180, 4000])
@pytest.mark.parametrize("nd", [16, 32, 48, 64, 80, 128, 144, 272, 512, 528, 768])
def test_full_range_volume(request, oracle, build, nd, p2):
    m = request.getfixturevalue(build)
    left, right, _ = render_pair(Texture(41), 37, 9, lambda x, y: 6.0 + 0.2 * x)
    right = right ^ (random_image(37, 9, nd) & 0x0700)
    o = StereoOptions(p1=25, p2=p2, p2_adapt=7 if p2 < 256 else 0, invalid_cost=35)
    assert np.array_equal(m.sgm_cost_volume(left, right, -4, nd, o), oracle.sgm_cost_volume(left, right, -4, nd, o))


def _ranges(w, h, nd, kind, seed):
    r = Rng(seed)
    if kind == "narrow":  # one unit, the same range along most of every chain, then small and large shifts
        num = np.full((h, w), 16, np.uint16)
        lo = np.full((h, w), nd // 2, np.uint16)
        lo[:, w // 3:] += 1
        lo[h // 2:, :] -= 3
        lo[h // 3, w // 2] = 0
        lo[2 * h // 3, w // 4] = nd - 16
    elif kind == "pairs":  # two units with a band of wide pixels through them
        num = np.full((h, w), 32, np.uint16)
        lo = np.full((h, w), nd // 4, np.uint16)
        num[:, w // 2:w // 2 + 4] = 112
        lo[:, w // 2:w // 2 + 4] = nd // 4 - 16
        num[h // 2, :w // 3] = 16
    else:  # anything, at random
        num = np.array([[16 * r.uniform_int(1, nd // 16) for _ in range(w)] for _ in range(h)], np.uint16)
        lo = np.array([[r.uniform_int(0, nd - int(n)) for n in row] for row in num], np.uint16)
    return LabelRanges(lo, num)


@pytest.mark.parametrize("build", BUILDS)
@pytest.mark.parametrize("p2", [180, 4000])
@pytest.mark.parametrize("w,h,nd,kind", [(70, 35, 160, "narrow"), (70, 35, 160, "pairs"), (37, 11, 160, "random"),
                                         (5, 3, 32, "random"), (1, 40, 48, "random"), (40, 1, 48, "random"),
                                         (9, 4, 640, "random")])
def test_ranged_volume(request, oracle, build, w, h, nd, kind, p2):
    m = request.getfixturevalue(build)
    left, right, _ = render_pair(Texture(43), w, h, lambda x, y: 9.0 + 0.3 * x - 0.1 * y)
    rg = _ranges(w, h, nd, kind, 47)
    o = StereoOptions(p1=25, p2=p2, p2_adapt=7 if p2 < 256 else 0)
    assert np.array_equal(m.sgm_cost_volume(left, right, 1, nd, o, rg),
                          oracle.sgm_cost_volume(left, right, 1, nd, o, (rg.lo, rg.num)))


@pytest.mark.parametrize("build", BUILDS)
@pytest.mark.parametrize("p2", [180, 4000])
@pytest.mark.parametrize("nd,levels", [(16, 0), (48, 0), (144, 0), (48, 1)])
def test_diagonal_check(request, oracle, build, nd, levels, p2):
    m = request.getfixturevalue(build)
    left, right, _ = render_pair(Texture(53), 75, 33, lambda x, y: np.where(x < 40, 5.0, 11.5))
    mask = np.full(left.shape, 255, np.uint8)
    mask[:, :4] = 0
    mask[9, :] = 0
    o = StereoOptions(p1=25, p2=p2, p2_adapt=0, levels=levels, lr_full_match=False, uniqueness=0.03, tile_size=32,
                      tile_margin=4, tile_blend=4, range_radius=1)
    a = m.match_stereo(left, right, mask, None, 0, nd, o)
    b = oracle.match_stereo(left, right, mask, None, 0, nd, o)
    assert same_disparities(a.disparity, b.disparity), mismatch_report(a.disparity, b.disparity)
    assert np.array_equal(a.confidence, b.confidence) and a.cells == b.cells
