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


FIELDS = ("x", "y", "flux", "peak", "fwhm", "eccentricity", "snr", "sharpness", "npix")


def _compare(native, images, **params):
    h, w = images[0].shape
    s = native.ResidentCalibratedStack(len(images), h, w)
    try:
        for k, f in enumerate(images):
            s.upload_calibrated_frame(k, f)
        found = s.detect_stars(range(len(images)), **params)
    finally:
        s.close()
    for got, image in zip(found, images):
        exp = ostars.detect_stars(image, **params)
        assert got.size == len(exp)
        for i, field in enumerate(FIELDS):
            want = np.asarray([np.nan if e[i] is None else e[i] for e in exp], dtype=np.float64)
            np.testing.assert_allclose(got[field].astype(np.float64), want, rtol=1e-9, atol=1e-12, err_msg=field)
    return sum(got.size for got in found)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 3), (4, 4), (3, 700), (700, 3), (40, 129), (33, 511), (33, 512), (33, 513),
                                   (31, 1025), (130, 2047)])
def test_gpu_detection_at_chunk_edges(native, shape):
    """Widths around the columns of one chunk, every alignment of a row's start;
    peaks up to the border, holes beside them."""
    h, w = shape
    rng = np.random.default_rng(h * 4096 + w)
    images = []
    for _ in range(2):
        img = 100.0 + rng.standard_normal((h, w))
        n = max(4, h * w // 60)
        np.add.at(img, (rng.integers(0, h, n), rng.integers(0, w, n)), rng.uniform(50.0, 5000.0, n))
        img[rng.random((h, w)) < 0.01] = np.nan
        images.append(img.astype(np.float32))
    _compare(native, images, threshold_sigma=4.0, max_stars=300, window_radius=3)


@pytest.mark.gpu
@pytest.mark.parametrize("min_separation_px,radius,max_stars", [(0.0, 4, 4096), (2.9, 1, 4096), (5.7, 4, 7),
                                                                (39.3, 2, 50), (1.0e9, 3, 10)])
def test_gpu_detection_of_crowds_and_plateaus(native, min_separation_px, radius, max_stars):
    """More brighter neighbours than a list holds, equal fluxes (raster order
    decides, also at the last place) and plateaus on which every pixel is a
    candidate; whole-number pixels, so every flux is exact on both sides."""
    rng = np.random.default_rng(5)
    h, w = 150, 260
    crowd = np.zeros((h, w))
    crowd[rng.random((h, w)) < 0.08] = 1.0
    crowd *= rng.integers(1, 900, (h, w))
    equal = np.zeros((h, w))
    equal[5:-5:9, 6:-6:11] = 64.0
    plateau = np.zeros((h, w))
    plateau[40:60, 17:150] = 5000.0
    images = [f.astype(np.float32) for f in (crowd, equal, plateau)]
    assert _compare(native, images, threshold_sigma=0.5, max_stars=max_stars, window_radius=radius,
                    min_separation_px=min_separation_px, background=0.0, noise=2.0) > 0
