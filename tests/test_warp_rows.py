"""The straight-line rows of the warp tiles against the general path.

A matrix times two is the same map, but no affine one to the library: it takes
the general path, with a division by a power of two that is exact.  The arithmetic of the samples is the same;
the coordinates (fixed point here, float-float there) agree to about 2^-34
pixels, so a sample's offset now and then rounds to the neighbouring float32:
the frames are equal but for few samples, and those within the slope of the
kernel (at most 6 per pixel) times 2^-24 of the largest sample, plus its
rounding.  Widths that TMA can and cannot describe, footprints that fit the
staged box and that do not, maps whose windows move by other than one source row
per output row, and sizes on both sides of a tile.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _maps(rng, h, w):
    def similarity(scale, deg, dx, dy):
        c, s = scale * np.cos(np.deg2rad(deg)), scale * np.sin(np.deg2rad(deg))
        cx, cy = w / 2, h / 2
        return [[c, -s, cx - c * cx + s * cy + dx], [s, c, cy - s * cx - c * cy + dy], [0, 0, 1]]

    return np.array([np.eye(3), similarity(1, 0, 3, -2), similarity(1, 0, 0.375, 0.6), similarity(1, 0.3, 5.2, -7.9),
                     similarity(1, -0.5, -11.7, 4.4), similarity(1.004, 0.1, 0.3, 0.8), similarity(0.93, -2.0, 1.0, 2.0),
                     similarity(1.3, 20.0, 0.0, 0.0), similarity(0.5, 3.0, 0.2, 0.1),
                     [[1.001, 2e-4, 0.4], [-3e-4, 0.998, 1.7], [0, 0, 1]],
                     [[1.0, 0.001, 2.0], [0.002, 1.0, -1.0], [1e-6, -2e-6, 1.0]]])


@pytest.mark.parametrize("interp", [1, 3])
@pytest.mark.parametrize("h,w", [(64, 64), (65, 68), (200, 264), (203, 257), (193, 130), (448, 511), (5, 131), (70, 4), (3, 3)])
def test_interior_rows_equal_general_path(native, interp, h, w):
    rng = np.random.default_rng(h * w + interp)
    maps = _maps(rng, h, w)
    n = len(maps)
    frames = (1000.0 + 30.0 * rng.standard_normal((n, h, w))).astype(np.float32)
    frames[rng.random(frames.shape) < 1e-3] += 30000.0
    frames[4, h // 2, w // 2] = np.inf
    frames[5, h // 3, w // 2] = np.nan
    frames[2, -1, -1] = np.nan
    frames[1, h // 2, : w // 2 : 3] = -np.inf
    stacks = []
    for scale, track in ((1.0, False), (2.0, True), (1.0, True)):
        s = native.ResidentCalibratedStack(n, h, w)
        for k in range(n):
            s.upload_calibrated_frame(k, frames[k])
        s.warp_frames_async(np.arange(n), scale * maps, interp, np.nan, -1.0, track)
        stacks.append(s)
    for k in range(n):
        a, b, c = (s.download_frame(k) for s in stacks)
        np.testing.assert_array_equal(a, c, err_msg=f"map {k}, coverage tracked")
        np.testing.assert_array_equal(np.isfinite(a), np.isfinite(b), err_msg=f"map {k}")
        ok = np.isfinite(a)
        limit = 8.0 * 2.0**-24 * np.abs(frames[k][np.isfinite(frames[k])]).max()
        assert np.abs(a[ok] - b[ok]).max(initial=0.0) <= limit, f"map {k}"
        assert np.mean(a[ok] != b[ok]) <= 0.01 if ok.any() else True, f"map {k}"
        # the counters of non-finite samples choose the integrator's formulas
        counts = {s.frame_global_stats(k)["nonfinite_pixels"] for s in stacks}
        assert counts == {a.size - ok.sum()}
    np.testing.assert_array_equal(stacks[1].warp_coverage_map(), stacks[2].warp_coverage_map())
    for s in stacks:
        s.close()
