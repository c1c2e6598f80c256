"""A frame that is listed more than once in one host calibration call.

The entries are calibrated in order: the last one is the frame's content, and
its non-finite count is the frame's, wherever the entries fall in the groups of
four that a call uploads together.  Sizes with and without pixels past the
last group of eight, one NaN per frame from the flat.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle.calibration import calibrate_light

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(1, 1), (7, 9), (33, 41), (64, 64)])
@pytest.mark.parametrize("order", [[2, 2], [0, 2, 2, 1], [1, 2, 0, 2, 2, 0], [2] * 9, [0, 1, 2, 0, 1, 2, 1, 1]])
def test_last_entry_of_a_host_call_wins(native, h, w, order):
    rng = np.random.default_rng(h * w + len(order))
    raw = rng.integers(0, 65536, (len(order), h, w), dtype=np.uint16)
    bias, dark = (rng.normal(m, 3.0, (h, w)).astype(np.float32) for m in (500.0, 20.0))
    flat = rng.uniform(0.5, 1.5, (h, w)).astype(np.float32)
    flat[h // 2, w // 3] = np.nan
    s = native.ResidentCalibratedStack(3, h, w)
    s.set_calibration_masters(bias, dark, flat)
    for _ in range(20):
        s.calibrate_frames_u16(order, raw, 1.0, 1.0)
        for k in set(order):
            light = raw[len(order) - 1 - order[::-1].index(k)]
            np.testing.assert_array_equal(s.download_frame(k), calibrate_light(light, bias, dark, flat, 1.0, 1.0))
            assert s.frame_global_stats(k)["nonfinite_pixels"] == 1
    if min(h, w) > 16:
        # the published count decides how a warp samples: around the NaN, or through it
        s.calibrate_frames_u16([0, 0, 1, 1, 2, 2], raw[[0] * 6], 1.0, 1.0)
        half = np.tile(np.array([[1.0, 0.0, 0.5], [0.0, 1.0, 0.5], [0.0, 0.0, 1.0]]), (3, 1, 1))
        s.warp_frames_async([0, 1, 2], half, 3, 0.0)
        for k in range(3):
            assert np.isfinite(s.download_frame(k)).all()
    s.close()
