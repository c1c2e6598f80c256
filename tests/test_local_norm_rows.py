"""Grid normalisation of narrow frames, whose rows share a thread block.

Widths on both sides of every number of threads that a row gets (8 to 256), rows
that start at every place of a 16-byte vector, heights that leave a block partly
empty.  The kernel multiplies and adds, each rounded once: equal to NumPy's
float32 to the last bit.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1, 4, 29, 30, 61, 62, 63, 125, 126, 253, 254, 509, 510, 1021, 1022, 2051])
@pytest.mark.parametrize("h", [1, 7, 33, 70])
def test_rows_of_any_width(native, h, w):
    rng = np.random.default_rng(w * 100 + h)
    n, tile = 3, 16
    frames = rng.normal(1000.0, 30.0, (n, h, w)).astype(np.float32)
    frames[1, h // 2, w // 2] = np.nan
    rows, cols = -(-h // tile), -(-w // tile)
    scales = rng.uniform(0.5, 1.5, (2, rows, cols)).astype(np.float32)
    offsets = rng.normal(0.0, 50.0, (2, rows, cols)).astype(np.float32)
    s = native.ResidentCalibratedStack(n, h, w)
    for k in range(n):
        s.upload_calibrated_frame(k, frames[k])
    s.apply_grid_normalization_frames([2, 1], scales, offsets, tile, tile)
    ty, tx = np.minimum(np.arange(h) // tile, rows - 1), np.minimum(np.arange(w) // tile, cols - 1)
    np.testing.assert_array_equal(s.download_frame(0), frames[0])
    for k, q in ((2, 0), (1, 1)):
        want = frames[k] * scales[q][ty][:, tx] + offsets[q][ty][:, tx]
        np.testing.assert_array_equal(s.download_frame(k), want.astype(np.float32))
    s.close()
