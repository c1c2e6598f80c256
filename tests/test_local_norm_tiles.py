"""Local normalisation at widths around the kernels' vectors and thread counts:
every alignment of a row's start, tiles that end inside a vector, tiles smaller
and larger than a block, samples that are not finite.  The bar is that of the
other local normalisation tests: scale and offset within one float32 ulp, pixels
within two."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import local_norm as oln
from tests.test_local_norm import _ulps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (37, 255), (33, 256), (35, 257), (70, 1025), (129, 1030)])
@pytest.mark.parametrize("tile", [1, 7, 64, 300])
def test_normalised_frames_match_oracle(native, shape, tile):
    if tile == 1 and shape[0] * shape[1] > 10000:
        pytest.skip("one tile per pixel: the small shapes cover it")
    rng = np.random.default_rng(shape[1] * 31 + tile)
    frames = (1000.0 + 20.0 * rng.standard_normal((3, *shape))).astype(np.float32)
    frames[1] = frames[1] * np.float32(1.07) + np.float32(40.0)
    frames[rng.random(frames.shape) < 0.02] = np.nan
    frames[2][rng.random(shape) < 0.01] = np.inf
    s = native.ResidentCalibratedStack(3, *shape)
    try:
        for k in range(3):
            s.upload_calibrated_frame(k, frames[k])
        s.local_normalize_grid(0, [1, 2], tile=tile)
        got = [s.download_frame(k) for k in range(3)]
    finally:
        s.close()
    with np.errstate(invalid="ignore"):
        exp, _ = oln.normalize_frames(frames, 0, np.ones(3, np.float32), tile=tile)
    for k in range(3):
        np.testing.assert_array_equal(np.isfinite(got[k]), np.isfinite(exp[k]), err_msg=f"frame {k}")
        fin = np.isfinite(exp[k])
        assert not fin.any() or _ulps(got[k][fin], exp[k][fin]).max() <= 2
