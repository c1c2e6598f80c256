"""Thread-per-pixel integration of samples near the ends of the float32 range.

The weighted sum is taken about the median, which may not be finite (the mean of
the two middle samples overflows, also for a pixel with one sample alone), and
neither may the samples' differences from it.  The sums themselves stay below
the range's end here, as the answer does.

Bar (that of the other integration kernels): coverage and rejection maps
exact, master and weight within one float32 ulp.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import integration as oint
from tests.test_gpu_integrate import MODES, _stack_from, assert_within_ulp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 64, 100, 200])
@pytest.mark.parametrize("rej", ["sigma_clip", "none"])
def test_samples_of_any_size(native, rej, n):
    rng = np.random.default_rng(n)
    frames = (1.0 + 0.03 * rng.standard_normal((n, 6, 35))) * 1.0e30
    frames[1:, 1] = np.nan   # one sample a pixel, beyond half the range
    frames[0, 1] = 2.5e38 * (1.0 + 0.01 * rng.standard_normal(35))
    frames[2:, 2] = np.nan   # two, of both signs
    frames[0, 2], frames[1, 2] = 3.0e38, -2.0e38
    frames = frames.astype(np.float32)
    weights = rng.uniform(0.25, 0.5, n).astype(np.float32)
    s = _stack_from(native, frames)
    s.integrate_async(weights, MODES[rej], 3.0, 3.0, 3, 0.5, count_map_dtype="float32")
    master, weight, cov, low, high, _ = s.download_maps("full")
    s.close()
    with np.errstate(over="ignore", invalid="ignore"):
        em, ew, ec, el, eh = oint.weighted_integrate_stack(frames, weights, rej, 3.0, 3.0, 3, 0.5)
    assert np.isfinite(em).all() and np.isfinite(master).all()
    np.testing.assert_array_equal(cov, ec)
    np.testing.assert_array_equal(low, el)
    np.testing.assert_array_equal(high, eh)
    assert_within_ulp(weight, ew, 1, "weight")
    assert_within_ulp(master, em, 1, "master")
