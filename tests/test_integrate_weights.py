"""Thread-per-pixel integration with frame weights far apart.

A pixel's weight is the frames' total minus what does not count only where
every partial sum of that is exact; else the weights that count are added up.
Weights over up to ten decades with rows that the lightest frames alone cover,
weights on both sides of the line between the two forms, with the bits that
make the low parts' sums as long as they get, weights near the ends of the
float32 range.

Bar (that of the other integration kernels): coverage and rejection maps
exact, master and weight within one float32 ulp.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import integration as oint
from tests.test_gpu_integrate import MODES, _stack_from, assert_within_ulp

pytestmark = pytest.mark.gpu


def _check(native, frames, weights, repeat=1, rejections=("winsorized_sigma", "sigma_clip", "none")):
    s = _stack_from(native, np.tile(frames, (1, 1, repeat)))
    for rej in rejections:
        s.integrate_async(weights, MODES[rej], 3.0, 3.0, 3, 0.5, count_map_dtype="float32")
        master, weight, cov, low, high, _ = s.download_maps("full")
        em, ew, ec, el, eh = (np.tile(m, (1, repeat)) for m in
                              oint.weighted_integrate_stack(frames, weights, rej, 3.0, 3.0, 3, 0.5))
        np.testing.assert_array_equal(cov, ec, err_msg=rej)
        np.testing.assert_array_equal(low, el, err_msg=rej)
        np.testing.assert_array_equal(high, eh, err_msg=rej)
        assert np.isfinite(em).all() and np.isfinite(master).all() and np.isfinite(weight).all()
        assert_within_ulp(weight, ew, 1, rej + " weight")
        assert_within_ulp(master, em, 1, rej + " master")
    s.close()


def _frames(rng, n, weights):
    """Sky; rows 3 to 5 hold the lightest tenth of the frames only, one pixel the lightest frame."""
    frames = (1000.0 + 30.0 * rng.standard_normal((n, 9, 39))).astype(np.float32)
    order = np.argsort(weights, kind="stable")
    frames[order[max(4, n // 10):], 3:6] = np.nan
    frames[order[1:], 6, 5] = np.nan
    return frames


@pytest.mark.parametrize("n", [24, 33, 64, 100, 200, 256])
@pytest.mark.parametrize("decades", [0.5, 1, 2, 3, 4, 6, 10])
def test_weights_over_decades(native, n, decades):
    rng = np.random.default_rng(n)
    weights = (10.0 ** rng.uniform(0, decades, n)).astype(np.float32)
    # 24 frames are on this path above 2^22 samples
    _check(native, _frames(rng, n, weights), weights, 1 if n > 32 else (1 << 22) // (n * 351) + 1)


@pytest.mark.parametrize("n", [33, 64, 65, 128, 256])
@pytest.mark.parametrize("bits", [1, 2, 3, 4, 5, 6])
def test_both_sides_of_the_split(native, n, bits):
    """Heavy frames whose low parts are all the largest there are, and light ones
    `bits` binary places down whose last bit is set."""
    rng = np.random.default_rng(bits)
    heavy = np.float32(1.0 + 2.0 ** -9 - 2.0 ** -23)
    light = np.float32(2.0 ** -bits * (1.0 + 2.0 ** -23))
    weights = np.where(np.arange(n) % 8 == 3, light, heavy).astype(np.float32)
    _check(native, _frames(rng, n, weights), weights)


@pytest.mark.parametrize("scale", [1e-30, 1e33, 1e34, 1e36])
def test_weights_of_any_size(native, scale):
    rng = np.random.default_rng(4)
    n = 40
    frames = (1.0 + 0.03 * rng.standard_normal((n, 9, 39))).astype(np.float32)
    frames[rng.random(frames.shape) < 0.02] = np.nan
    _check(native, frames, (scale * rng.uniform(0.5, 1.5, n)).astype(np.float32))
