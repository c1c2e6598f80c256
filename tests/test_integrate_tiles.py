"""Stacks of up to 32 frames on the side of the integrator that works in tiles:
frame counts on both sides of every line of the dispatch, a little more than
the 2^22 samples up to which the column kernel keeps them.  The frames repeat a
small patch, so the oracle's maps of the patch, repeated, are the answer.

Bar: rejection and coverage maps exact, master and weight within one float32
ulp, as for the other integration kernels."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import integration as oint
from tests.test_gpu_integrate import MODES, _stack_from, assert_within_ulp
from tests.test_integrate_px import _columns

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 9, 15, 16, 17, 24, 25, 31, 32])
@pytest.mark.parametrize("kind", ["sky", "zero", "ties", "holes"])
def test_small_stacks_match_oracle(native, kind, n):
    rng = np.random.default_rng(11 * n + len(kind))
    patch = _columns(kind, rng, n, (9, 39))
    down, across = 41, (1 << 22) // (n * 9 * 41 * 39) + 1
    weights = rng.uniform(0.5, 2.0, n).astype(np.float32)
    weights[n // 2] = 0.0
    s = _stack_from(native, np.tile(patch, (1, down, across)))
    try:
        for rej in ("winsorized_sigma", "sigma_clip", "none"):
            s.integrate_async(weights, MODES[rej], 2.5, 3.0, 3, 0.4, count_map_dtype="float32")
            master, weight, cov, low, high, dq = s.download_maps("full")
            em, ew, ec, el, eh = (np.tile(m, (down, across)) for m in
                                  oint.weighted_integrate_stack(patch, weights, rej, 2.5, 3.0, 3, 0.4))
            what = f"{kind} n={n} {rej}"
            np.testing.assert_array_equal(cov, ec, err_msg=what)
            np.testing.assert_array_equal(low, el, err_msg=what)
            np.testing.assert_array_equal(high, eh, err_msg=what)
            assert_within_ulp(weight, ew, 1, what + " weight")
            assert_within_ulp(master, em, 1, what + " master")
            np.testing.assert_array_equal(dq, oint.dq_map(master, weight, cov, low, high), err_msg=what)
    finally:
        s.close()
