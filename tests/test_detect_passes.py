"""The passes of the star detector at the sizes where their work splits change:
the order statistics are exact order statistics, so they equal np.median bit
for bit, and the star lists equal the oracle's (order and count exactly, float64
sums within 1e-9 relative as for the detector's other tests)."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import stars as ostars


def _values(kind, n, rng):
    if kind == "sky":
        return 1000.0 + 30.0 * rng.standard_normal(n)
    if kind == "ties":  # whole numbers around the middle
        return np.round(1000.0 + 2.0 * rng.standard_normal(n))
    if kind == "constant":
        return np.full(n, 7.25)
    if kind == "wide":  # every exponent, both signs
        return rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(-126.0, 126.0, n))
    v = 5.0 * rng.standard_normal(n)  # "holes": hardly any finite sample, infinities of both signs
    v[rng.random(n) < 0.97] = np.nan
    v[rng.random(n) < 0.2] = np.inf
    v[rng.random(n) < 0.2] = -np.inf
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["sky", "ties", "constant", "wide", "holes"])
@pytest.mark.parametrize("shape", [(1, 1), (1, 2), (31, 33), (64, 64), (127, 129), (181, 181), (182, 181),
                                   (256, 256), (257, 1021), (1201, 1003)])
def test_gpu_order_statistics_exact(native, shape, kind):
    rng = np.random.default_rng(shape[0] * 10000 + shape[1])
    frames = [_values(kind, shape[0] * shape[1], rng).astype(np.float32).reshape(shape) for _ in range(2)]
    s = native.ResidentCalibratedStack(2, *shape)
    try:
        for k, f in enumerate(frames):
            s.upload_calibrated_frame(k, f)
        for _ in range(2):  # the scratch of one call serves the next
            _, info = s.detect_stars([1, 0], threshold_sigma=1.0e38, max_stars=4, with_info=True)
            for got, f in zip(info, frames[::-1]):
                v = f[np.isfinite(f)]
                assert got["valid_pixels"] == v.size
                if v.size == 0:
                    continue
                with np.errstate(over="ignore"):
                    med = np.median(v)
                    mad = np.median(np.abs(v - med))
                assert got["median"] == med
                assert got["mad"] == mad
    finally:
        s.close()
