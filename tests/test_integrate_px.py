"""Thread-per-pixel integration of 33 to 256 frames against the oracle.

Frame counts on both sides of every list length of the dispatch, a pixel count
that leaves a partial last tile of 32, and columns that take each path of the
statistics: exact deviations from the median (sky), deviations that round
(values around zero), ties and constant columns, samples that are not finite,
columns with one or no sample, frames without weight.

Bar (that of the other integration kernels): rejection and coverage maps exact,
master and weight within one float32 ulp.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import integration as oint
from tests.test_gpu_integrate import MODES, _stack_from, assert_within_ulp

pytestmark = pytest.mark.gpu

EDGES = [33, 40, 41, 48, 49, 64, 65, 80, 81, 96, 97, 128, 129, 160, 161, 192, 193, 200, 208, 209, 255, 256]


def _columns(kind, rng, n, shape):
    if kind == "sky":
        v = 1000.0 + 30.0 * rng.standard_normal((n, *shape))
        v[rng.random(v.shape) < 0.02] += 20000.0
    elif kind == "zero":
        v = 3.0 * rng.standard_normal((n, *shape)) + rng.choice([0.0, 1e-3, -2.0, 7.0], shape)
        v[rng.random(v.shape) < 0.02] -= 500.0
    else:
        v = np.round(50.0 + 2.0 * rng.standard_normal((n, *shape)))
        v[:, 0, :5] = 50.0
        v[: n // 8, 0, 2] = 90.0
    v = v.astype(np.float32)
    if kind == "holes":
        v = (1000.0 + 30.0 * rng.standard_normal((n, *shape))).astype(np.float32)
        bad = rng.random(v.shape)
        v[bad < 0.06] = np.nan
        v[(bad > 0.06) & (bad < 0.08)] = np.inf
        v[(bad > 0.08) & (bad < 0.10)] = -np.inf
        v[:, 1, 1] = np.nan
        v[1:, 1, 2] = np.nan
        v[: n - 2, 1, 3] = np.nan
    return v


@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("kind", ["sky", "zero", "ties", "holes"])
def test_columns_match_oracle(native, kind, n):
    rng = np.random.default_rng(7 * n + len(kind))
    stack = _columns(kind, rng, n, (9, 39))
    weights = rng.uniform(0.5, 2.0, n).astype(np.float32)
    dropped = weights.copy()
    dropped[[0, n // 2]] = 0.0
    dropped[n - 1] = np.nan
    s = _stack_from(native, stack)
    for tag, w in (("unit", None), ("weights", weights), ("dropped", dropped)):
        for rej in ("winsorized_sigma", "sigma_clip", "none"):
            s.integrate_async(w, MODES[rej], 2.5, 3.0, 3, 0.4, count_map_dtype="float32")
            master, weight, cov, low, high, dq = s.download_maps("full")
            em, ew, ec, el, eh = oint.weighted_integrate_stack(stack, w, rej, 2.5, 3.0, 3, 0.4)
            what = f"{kind} n={n} {tag} {rej}"
            np.testing.assert_array_equal(cov, ec, err_msg=what)
            np.testing.assert_array_equal(low, el, err_msg=what)
            np.testing.assert_array_equal(high, eh, err_msg=what)
            assert_within_ulp(weight, ew, 1, what + " weight")
            assert_within_ulp(master, em, 1, what + " master")
            np.testing.assert_array_equal(dq, oint.dq_map(master, weight, cov, low, high), err_msg=what)
    s.close()


def test_most_frames_without_weight(native):
    """Lists that are mostly padding: 4 of 200 frames count."""
    rng = np.random.default_rng(3)
    stack = _columns("sky", rng, 200, (5, 33))
    weights = np.zeros(200, np.float32)
    weights[[1, 77, 150, 199]] = (1.0, 0.5, 2.0, 1.5)
    s = _stack_from(native, stack)
    for w in (weights, np.zeros(200, np.float32)):
        for rej in ("winsorized_sigma", "sigma_clip", "none"):
            s.integrate_async(w, MODES[rej], 3.0, 3.0, 3, 0.5, count_map_dtype="float32")
            master, weight, cov, low, high, _ = s.download_maps("full")
            em, ew, ec, el, eh = oint.weighted_integrate_stack(stack, w, rej, 3.0, 3.0, 3, 0.5)
            np.testing.assert_array_equal(cov, ec, err_msg=rej)
            np.testing.assert_array_equal(low, el, err_msg=rej)
            np.testing.assert_array_equal(high, eh, err_msg=rej)
            assert_within_ulp(weight, ew, 1, rej)
            assert_within_ulp(master, em, 1, rej)
    s.close()
