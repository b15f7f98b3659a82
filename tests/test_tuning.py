"""The autotuner's table reaches the launches: entries given through
R3DGPU_TUNING set the band rows of the ranged kernel and the shape of the
full-range kernel (seen in the library's per-launch profile), results stay
identical, and environment overrides take precedence."""

from __future__ import annotations

import collections
import ctypes
import json

import numpy as np

from images import Texture, render_pair
from regard3d_mvs_b200.types import CProfile, LabelRanges, StereoOptions


def _launches(m, run):
    lib = m.lib
    lib.r3dgpu_profile_enable(1)
    prof = CProfile()
    lib.r3dgpu_profile_take(ctypes.byref(prof))
    out = run()
    lib.r3dgpu_profile_take(ctypes.byref(prof))
    lib.r3dgpu_profile_enable(0)
    n = lib.r3dgpu_profile_launches(None, 0)
    buf = ctypes.create_string_buffer(int(n) + 1)
    lib.r3dgpu_profile_launches(buf, n + 1)
    return out, [e for e in json.loads(buf.value.decode() or "[]") if e["kernel"] != "sgm_round"]


def pass_shapes(m, run):
    """The result of run() and the shapes ("GxK/modeM") of its chain passes."""
    out, launches = _launches(m, run)
    return out, {e["shape"] for e in launches if e.get("pass")}


def match_kernels(m, run):
    """The result of run() and the names of its matches' SGM kernels."""
    out, launches = _launches(m, run)
    return out, {e["kernel"] for e in launches}


def test_default_kernels_are_the_chain_passes(simt_matcher):
    """Full-range and ranged tiles go to the chain-pass kernels by default."""
    tex = Texture(61)
    left, right, _ = render_pair(tex, 40, 30, lambda x, y: 6.0 + 0.1 * x)
    pairs = [dict(left=left, right=right, disparity_min=0, num_disparities=32, options=StereoOptions(levels=0)),
             dict(left=left, right=right, disparity_min=0, num_disparities=32, options=StereoOptions(levels=1))]
    _, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    kinds = {e["kernel"] for e in launches}
    assert kinds == {"sgm_path_kernel", "sgm_path_ranged_kernel"}, kinds


def test_table_from_environment(simt_matcher, monkeypatch):
    """The table drives the one-CTA-per-tile kernels (selected by the environment)."""
    monkeypatch.setenv("R3DGPU_FULL_KERNEL", "wavefront")
    monkeypatch.setenv("R3DGPU_RANGED_KERNEL", "ranged")
    tex = Texture(61)
    left, right, _ = render_pair(tex, 40, 30, lambda x, y: 6.0 + 0.1 * x)
    pairs = [dict(left=left, right=right, disparity_min=0, num_disparities=32, options=StereoOptions(levels=0))]
    monkeypatch.setenv("R3DGPU_TUNING", "#")
    ref, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert [e["shape"] for e in launches] == ["8x4/nd32"]
    monkeypatch.setenv("R3DGPU_TUNING", "full 32 16 4 6; ranged 32 8")
    got, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert [(e["shape"], e["rows"]) for e in launches] == [("16x4/nd32", 6)]
    assert np.array_equal(np.nan_to_num(got[0].disparity, posinf=-1), np.nan_to_num(ref[0].disparity, posinf=-1))
    # Ranged kernel rows, and an environment override that wins over the table.
    lo = np.full((30, 40), 4, np.uint16)
    num = np.full((30, 40), 16, np.uint16)
    _, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    monkeypatch.setenv("R3DGPU_FULL_ROWS", "2")
    _, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert [(e["shape"], e["rows"]) for e in launches] == [("16x4/nd32", 2)]
    vol = simt_matcher.sgm_cost_volume(left, right, 0, 32, StereoOptions(), LabelRanges(lo, num))
    assert vol.size == 16 * 40 * 30


def test_path_shape_from_table(simt_matcher, monkeypatch):
    """A `path` entry sets the chain passes' shape for its label count (seen
    in the per-pass profile), R3DGPU_PATH_SHAPE overrides it, and the maps
    stay identical."""
    tex = Texture(62)
    left, right, _ = render_pair(tex, 40, 30, lambda x, y: 6.0 + 0.1 * x)
    pairs = [dict(left=left, right=right, disparity_min=0, num_disparities=64, options=StereoOptions(levels=0))]

    def shapes(launches):
        return {e["shape"].split("/")[0] for e in launches if e.get("pass")}

    monkeypatch.setenv("R3DGPU_TUNING", "#")
    ref, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert shapes(launches) == {"4x8"}
    monkeypatch.setenv("R3DGPU_TUNING", "path 64 2 16")
    got, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert shapes(launches) == {"2x16"}
    assert np.array_equal(np.nan_to_num(got[0].disparity, posinf=-1), np.nan_to_num(ref[0].disparity, posinf=-1))
    monkeypatch.setenv("R3DGPU_PATH_SHAPE", "8,8")
    got, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert shapes(launches) == {"8x8"}
    assert np.array_equal(np.nan_to_num(got[0].disparity, posinf=-1), np.nan_to_num(ref[0].disparity, posinf=-1))


def test_shapes_of_one_width_in_a_batch(simt_matcher, monkeypatch):
    """Two shapes of the same label width (8x16 for 256 labels, 16x8 from the
    table for 192) in turn over a batch of more pairs than a wave has block
    counters for: tiles are grouped by the shape itself, one term launch each,
    and the maps are those of the built-in shapes."""
    pairs = []
    for i in range(34):
        left, right, _ = render_pair(Texture(63 + i), 18, 4, lambda x, y: 5.0 + 0.1 * x)
        pairs.append(dict(left=left, right=right, disparity_min=0, num_disparities=192 if i % 2 else 256,
                          options=StereoOptions(levels=0, lr_full_match=False)))
    monkeypatch.setenv("R3DGPU_TUNING", "#")
    ref = simt_matcher.match_stereo_batch(pairs)
    monkeypatch.setenv("R3DGPU_TUNING", "path 192 16 8")
    got, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
    assert sorted(e["shape"].split("/")[0] for e in launches if e.get("pass")) == ["16x8", "8x16"]
    for a, b in zip(got, ref):
        assert np.array_equal(a.disparity, b.disparity) and np.array_equal(a.confidence, b.confidence)


def test_default_shapes_by_mode(simt_matcher):
    """Byte terms take 16 label pairs per lane above 64 labels; u16 sums, one
    direction at a time, 8 up to 512 labels."""
    left, right, _ = render_pair(Texture(75), 12, 4, lambda x, y: 4.0 + 0.1 * x)
    for nd, terms, sums in ((64, "4x8", "4x8"), (80, "4x16", "8x8"), (128, "4x16", "8x8"), (256, "8x16", "16x8"),
                            (272, "16x16", "32x8"), (512, "16x16", "32x8"), (528, "32x16", "32x16")):
        for p2, want in ((200, {f"{terms}/mode3"}), (400, {f"{sums}/mode0", f"{sums}/mode1"})):
            _, shapes = pass_shapes(simt_matcher,
                                    lambda: simt_matcher.sgm_cost_volume(left, right, 0, nd, StereoOptions(p2=p2)))
            assert shapes == want, (nd, p2)


def _scratch_budget(m, n):
    """Sets the SGM scratch budget of this thread, as a server worker does (0: the default)."""
    m.lib._ZN6r3dgpu25set_thread_scratch_budgetEm(ctypes.c_size_t(n))


def test_pass_mode_by_tile(simt_matcher):
    """The pass mode is each tile's own: a tile whose byte terms (9 bytes a
    label) pass the scratch budget takes u16 sums (two volumes, 5 bytes, two
    directions a launch, or one, 3 bytes), as a pair with a P2 above 255 does,
    and the batch's other pairs keep byte terms."""
    def pair(seed, w, h, nd, **kw):
        left, right, _ = render_pair(Texture(seed), w, h, lambda x, y: 5.0 + 0.1 * x)
        return dict(left=left, right=right, disparity_min=0, num_disparities=nd, options=StereoOptions(**kw))

    def modes(pairs, budget):
        _scratch_budget(simt_matcher, budget)
        try:
            out, launches = _launches(simt_matcher, lambda: simt_matcher.match_stereo_batch(pairs))
            return out, collections.Counter(e["shape"] for e in launches if e.get("pass"))
        finally:
            _scratch_budget(simt_matcher, 0)

    # 60 x 24 x 64 labels: 829 kB with terms, 461 and 276 kB with sums (a wave for each of its two matches).
    pairs = [pair(71, 60, 24, 64, levels=0), pair(72, 24, 12, 32, levels=0), pair(73, 20, 10, 16, levels=0, p2=400)]
    ref, shapes = modes(pairs, 0)
    assert shapes == {"4x8/mode3": 1, "2x8/mode3": 1, "1x8/mode0": 1, "1x8/mode1": 3}
    for budget, adding in ((500_000, 3), (300_000, 7)):
        got, shapes = modes(pairs, budget)
        assert set(shapes) == {"4x8/mode0", "4x8/mode1", "2x8/mode3", "1x8/mode0", "1x8/mode1"}
        assert (shapes["4x8/mode0"], shapes["4x8/mode1"]) == (2, 2 * adding)
        for a, b in zip(got, ref):
            assert np.array_equal(a.disparity, b.disparity) and np.array_equal(a.confidence, b.confidence)
    # Ranged tiles, the finer level of a hierarchy: 46 k labels a match at 9, 5 or 3 bytes, 23 kB of records, and in
    # one of the two matches 230 kB for the vectors of wide pixels.
    for p2, budget, want in ((200, 0, {"1x8/mode3": 1}), (200, 600_000, {"1x8/mode3": 1, "1x8/mode0": 1, "1x8/mode1": 3}),
                             (200, 250_000, {"1x8/mode0": 2, "1x8/mode1": 14}), (400, 0, {"1x8/mode0": 1, "1x8/mode1": 3})):
        pairs = [pair(74, 72, 40, 48, levels=1, range_radius=0, range_margin=2, range_fill=0, p2=p2)]
        got, shapes = modes(pairs, budget)
        assert {q: n for q, n in shapes.items() if q.startswith("1x8/")} == want, (p2, budget)
        if p2 == 200:
            ref = got if budget == 0 else ref
            assert np.array_equal(got[0].disparity, ref[0].disparity)
