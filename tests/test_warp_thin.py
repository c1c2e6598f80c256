"""Bilinear warps of frames of one or two rows or columns.

Positions outside such a frame are sampled at a clamped place before the mask
drops them, and that place may be the frame's last sample.  Maps that put
positions before the first and behind the last row and column, frames of a
stack and single images.

Bar (that of the other warp tests): within 1e-5 relative plus 3e-6 of the largest
sample, validity exact.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import warp as owarp

pytestmark = pytest.mark.gpu

MAPS = np.array([[[1, 0, 0.5], [0, 1, 0.25], [0, 0, 1]], [[1, 0, -0.25], [0, 1, -0.5], [0, 0, 1]],
                 [[1, 0, 3.0], [0, 1, 0.0], [0, 0, 1]], [[1, 0, 0.0], [0, 1, 70.5], [0, 0, 1]],
                 [[1, 0, -40.0], [0, 1, 0.0], [0, 0, 1]], [[-1, 0, 0.25], [0, 1, 0.0], [0, 0, 1]]], dtype=np.float64)


@pytest.mark.parametrize("h,w", [(1, 1), (1, 2), (1, 7), (1, 130), (1, 4096), (5, 1), (200, 1), (2, 2), (2, 64), (130, 2)])
@pytest.mark.parametrize("interp", [1, 3])
def test_thin_frames(native, h, w, interp):
    from glass_gb300.adjoint import warp_affine

    import torch

    rng = np.random.default_rng(h + w)
    n = len(MAPS)
    frames = rng.normal(1000.0, 30.0, (n, h, w)).astype(np.float32)
    s = native.ResidentCalibratedStack(n, h, w)
    for k in range(n):
        s.upload_calibrated_frame(k, frames[k])
    s.warp_frames_async(np.arange(n), MAPS, interp, np.nan)
    name = {1: "bilinear", 3: "lanczos3"}[interp]
    for k in range(n):
        want, _ = owarp.warp_matrix(frames[k], MAPS[k], name, np.nan)
        theta = torch.from_numpy(np.linalg.inv(MAPS[k])[:2].reshape(-1).copy())
        image = warp_affine(torch.from_numpy(frames[k]).cuda(), theta, name, float("nan"), True).cpu().numpy()
        for got in (s.download_frame(k), image):
            np.testing.assert_array_equal(np.isfinite(got), np.isfinite(want), err_msg=f"map {k}")
            ok = np.isfinite(want)
            np.testing.assert_allclose(got[ok], want[ok], rtol=1e-5, atol=3e-6 * 1200.0, err_msg=f"map {k}")
    s.close()
