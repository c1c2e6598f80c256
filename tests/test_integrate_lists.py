"""Thread-per-pixel integration on both sides of every list length.

Lists grow in steps of eight rows: 16 to 64 frames in one, 65 to 256 in two of
up to half the frames, so a count one below, at and one above each step, with
every frame weighted and with more frames without weight than a step holds.

Bar (that of the other integration kernels): coverage and rejection maps
exact, master and weight within one float32 ulp.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import integration as oint
from tests.test_gpu_integrate import MODES, _stack_from, assert_within_ulp
from tests.test_integrate_px import _columns

pytestmark = pytest.mark.gpu

STEPS = [40, 48, 56, 64, *range(80, 256, 16)]


@pytest.mark.parametrize("n", sorted({*STEPS, *(n + 1 for n in STEPS), 79, 255, 256}))
@pytest.mark.parametrize("kind", ["sky", "holes"])
def test_counts_match_oracle(native, kind, n):
    rng = np.random.default_rng(3 * n + len(kind))
    stack = _columns(kind, rng, n, (5, 39))
    weights = rng.uniform(0.5, 2.0, n).astype(np.float32)
    few = weights.copy()
    few[rng.permutation(n)[:n // 3]] = 0.0
    s = _stack_from(native, stack)
    for w in (weights, few):
        for rej in ("winsorized_sigma", "sigma_clip", "none"):
            s.integrate_async(w, MODES[rej], 2.5, 3.0, 3, 0.4, count_map_dtype="float32")
            master, weight, cov, low, high, _ = s.download_maps("full")
            em, ew, ec, el, eh = oint.weighted_integrate_stack(stack, w, rej, 2.5, 3.0, 3, 0.4)
            what = f"{kind} n={n} {rej}"
            np.testing.assert_array_equal(cov, ec, err_msg=what)
            np.testing.assert_array_equal(low, el, err_msg=what)
            np.testing.assert_array_equal(high, eh, err_msg=what)
            assert_within_ulp(weight, ew, 1, what + " weight")
            assert_within_ulp(master, em, 1, what + " master")
    s.close()
