"""Fused warp + integration in bands of rows: stacks above 2 GiB have 16 spare
slots, so several frames share one and the image is done band by band.

The maps and the geometric coverage must be those of warping the frames in
place and integrating them (the frames themselves stay as they are).
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 40 frames: three to a spare slot, three bands with a partial last tile row.
# 512 frames two rows high: the spare slots hold less than a row of each.
@pytest.mark.parametrize("n,h,w,interp", [(40, 3703, 3652, "lanczos3"), (40, 3652, 3703, "bilinear"),
                                          (512, 2, 600000, "bilinear")])
def test_bands_equal_warp_then_integrate(native, n, h, w, interp):
    rng = np.random.default_rng(n + h)
    base = (900.0 + 20.0 * rng.standard_normal((3, h, w))).astype(np.float32)
    base[rng.random(base.shape) < 1e-3] += 9000.0
    base[1, h // 2, w // 3 : w // 3 + 40] = np.nan
    # shifts by eighths of a pixel: every source coordinate is exact, so both
    # forms agree on it to the last bit
    mats = np.tile(np.eye(3), (n, 1, 1))
    mats[1:, 0, 2] = rng.integers(-240, 241, n - 1) / 8.0
    mats[1:, 1, 2] = rng.integers(-240, 241, n - 1) / 8.0 if h > 2 else 0.25
    weights = rng.uniform(0.5, 2.0, n).astype(np.float32)
    s = native.ResidentCalibratedStack(n, h, w)
    try:
        for k in range(n):
            s.upload_calibrated_frame(k, base[k % 3])
        fused = s.integrate_matrix_warped_sigma_clip(mats, weights, interp, -1.0, 3.0, 3.0, True)
        np.testing.assert_array_equal(s.download_frame(1), base[1])
        s.reset_warp_coverage()
        s.warp_frames_async(np.arange(n), mats, 1 if interp == "bilinear" else 3, np.nan, -1.0, True)
        geo = s.warp_coverage_map()
        two = s.integrate_sigma_clip(weights, 3.0, 3.0, True)
    finally:
        s.close()
    np.testing.assert_array_equal(fused[5], geo)
    for a, b, name in zip(fused[:5], two, ("master", "weight", "coverage", "low", "high")):
        # whole shifts: the fused form takes the Lanczos3 sum at offset 0 where
        # the warp takes the sample itself
        np.testing.assert_allclose(a, b, rtol=3e-7 if name == "master" else 0, atol=0, err_msg=name)
