"""Warps whose frames take different launch forms, in one call.

Maps whose tiles' footprints fit a staged box at 64, 48 and 16 rows or not at
all, projective ones, with and without the clamp, in an order that no launch
keeps; widths that TMA can and cannot describe; more frames than spare slots.

Bar (that of the other warp tests): within 1e-5 relative plus 3e-6 of the largest
sample; validity exact.  Nearest decides by the float32 offset, which is the tie
itself for positions within 2^-25 of one (1 of 2.8 million here): those may take
either sample.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import warp as owarp

pytestmark = pytest.mark.gpu

NAMES = {0: "nearest", 1: "bilinear", 3: "lanczos3"}


def _maps(h, w):
    def similarity(scale, deg, dx, dy):
        c, s = scale * np.cos(np.deg2rad(deg)), scale * np.sin(np.deg2rad(deg))
        cx, cy = w / 2, h / 2
        return [[c, -s, cx - c * cx + s * cy + dx], [s, c, cy - s * cx - c * cy + dy], [0, 0, 1]]

    return np.array([similarity(1, 30.0, 0.3, 0.2), similarity(1, 0.3, 5.2, -7.9), similarity(1.9, 3.0, 0.2, 0.1),
                     similarity(1, 7.0, 1.1, 2.3), [[1.0, 0.001, 2.0], [0.002, 1.0, -1.0], [1e-6, -2e-6, 1.0]],
                     similarity(1, 90.0, 0.3, 0.4), similarity(0.5, 1.0, 0.2, 0.3), similarity(1, 180.2, 0.4, -0.3),
                     similarity(1, -135.0, 0.7, 0.1), similarity(0.85, 4.0, 0.3, 0.6), similarity(1, 8.0, -0.4, 0.7)])


@pytest.mark.parametrize("interp,clamp", [(0, -1.0), (1, -1.0), (3, -1.0), (3, 0.3)])
@pytest.mark.parametrize("h,w", [(200, 260), (131, 257), (49, 64), (400, 1028)])
def test_maps_of_all_forms_in_one_call(native, h, w, interp, clamp):
    rng = np.random.default_rng(h + interp)
    maps = _maps(h, w)
    n = len(maps)
    frames = (1000.0 + 30.0 * rng.standard_normal((n, h, w))).astype(np.float32)
    frames[1, h // 2, w // 2] = np.nan
    frames[8, h // 2, w // 2 : w // 2 + 3] = np.nan
    s = native.ResidentCalibratedStack(n, h, w)
    for k in range(n):
        s.upload_calibrated_frame(k, frames[k])
    s.reset_warp_coverage()
    s.warp_frames_async(np.arange(n), maps, interp, np.nan, clamp, True)
    coverage = np.zeros((h, w), np.float32)
    for k in range(n):
        want, cov = owarp.warp_matrix(frames[k], maps[k], NAMES[interp], np.nan, clamp)
        got = s.download_frame(k)
        coverage += cov
        np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want), err_msg=f"map {k}")
        ok = np.isfinite(want)
        valid = ok.sum()
        if interp == 0:
            for c in owarp.source_coordinates(maps[k], h, w):
                ok &= np.abs(c - np.floor(c) - 0.5) > 2.0 ** -25
        np.testing.assert_allclose(got[ok], want[ok], rtol=1e-5, atol=3e-6 * np.nanmax(np.abs(frames[k])),
                                   err_msg=f"map {k}")
        assert s.frame_global_stats(k)["nonfinite_pixels"] == h * w - valid
    np.testing.assert_array_equal(s.warp_coverage_map(), coverage)
    s.close()


def test_more_frames_than_spare_slots(native):
    """17 frames over 2 GiB have 16 spare slots: two groups, each of several forms."""
    h, w, n = 4600, 7040, 17
    maps = _maps(h, w)[[0, 1, 2, 3, 4]]
    base = np.random.default_rng(5).normal(1000.0, 30.0, (h, w)).astype(np.float32)
    one = native.ResidentCalibratedStack(1, h, w)
    want = []
    for m in maps:
        one.upload_calibrated_frame(0, base)
        one.warp_frames_async([0], m[None], 1, 0.0)
        want.append(one.download_frame(0))
    one.close()
    s = native.ResidentCalibratedStack(n, h, w)
    order = np.random.default_rng(6).integers(0, len(maps), n)
    for k in range(n):
        s.upload_calibrated_frame(k, base)
    s.warp_frames_async(np.arange(n), maps[order], 1, 0.0)
    for k in range(n):
        np.testing.assert_array_equal(s.download_frame(k), want[order[k]], err_msg=f"frame {k}")
    s.close()
