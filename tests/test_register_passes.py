"""The passes of the catalog registration at the sizes where their work splits
change: descriptor counts around a warp, catalogs of every size up to 80, more
matches than the list holds, crowds in which stars have several partners within
the tolerance.  Pair sets and counts are exact, matrices and rms within the
bounds of the estimator's other tests."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import registration as oreg


def _catalogs(n, seed, crowded=False):
    rng = np.random.default_rng(seed)
    ref = rng.uniform(20.0, 900.0, (n, 2))
    if crowded:  # half the stars beside another one
        ref[n // 2 :] = ref[: n - n // 2] + rng.uniform(-2.5, 2.5, (n - n // 2, 2))
    angle = 0.01 * rng.standard_normal()
    lin = np.array([[np.cos(angle), -np.sin(angle)], [np.sin(angle), np.cos(angle)]])
    mov = ref @ lin.T + rng.uniform(-15.0, 15.0, 2) + 0.05 * rng.standard_normal((n, 2))
    return ref, mov[rng.permutation(n)]


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["similarity", "affine"])
@pytest.mark.parametrize("crowded", [False, True])
@pytest.mark.parametrize("n", [2, 4, 7, 12, 31, 32, 33, 64, 80])
def test_gpu_estimator_of_every_size(native, n, crowded, model):
    ref, mov = _catalogs(n, 100 + n, crowded)
    params = dict(min_inliers=3, tolerance_px=3.0, max_candidates=600)
    if n == 33:  # 64-bit selection over more matches than the list holds
        params.update(descriptor_radius=1.0e6, neighbors=6)
    got = native.estimate_triangle_asterism_transform(ref, mov, transform_model=model, **params)
    exp = oreg.estimate_triangle_asterism_transform(ref, mov, transform_model=model, **params)
    assert got["inliers"] == exp["inliers"]
    assert got["status"] == exp["status"]
    assert sorted(got["pairs"]) == sorted(tuple(p) for p in exp["pairs"])
    if exp["inliers"]:
        np.testing.assert_allclose(got["matrix"], exp["matrix"], rtol=0, atol=1e-8)
        np.testing.assert_allclose(got["rms_px"], exp["rms_px"], rtol=1e-9, atol=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("side,neighbors", [(2, 3), (3, 5), (5, 6), (8, 5), (9, 6)])
def test_gpu_descriptors_of_a_lattice(native, side, neighbors):
    """Equal distances and equal areas everywhere: index order decides."""
    y, x = np.mgrid[0:side, 0:side].reshape(2, -1).astype(np.float64) * 16.0
    x, y = x[:80], y[:80]
    got = native.triangle_asterism_descriptors_f32(x, y, 80, neighbors, 5000)
    exp = oreg.local_triangle_descriptors(np.stack([x, y], 1), 80, neighbors, 5000)
    assert got["count"] == len(exp)
    np.testing.assert_array_equal(got["indices"], np.asarray([d[1] for d in exp], np.int32).reshape(-1, 3))
    np.testing.assert_array_equal(got["descriptors"],
                                  np.asarray([d[0] for d in exp], np.float64).reshape(-1, 2).astype(np.float32))
