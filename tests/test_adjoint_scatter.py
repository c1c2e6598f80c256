"""Image gradient of the Lanczos3 warp: cells kept per lane, summed over shuffles.

Maps whose windows move by one source row per output row for whole warps, for
some of their lanes only (rotations), and not at all (scales, shears, a map of
nine source rows per row), images of one column strip and of several, borders,
windows with non-finite taps.  Against float64 autograd of the PyTorch warp, to
1e-5 of the gradient's scale: the float32 weights are within 2e-7 of exact and
the largest of these sums adds under 100 of them.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.torch_warp_reference import warp_affine_reference

pytestmark = pytest.mark.gpu


def _maps(h, w):
    def similarity(scale, deg, dx, dy):
        c, s = scale * np.cos(np.deg2rad(deg)), scale * np.sin(np.deg2rad(deg))
        cx, cy = w / 2, h / 2
        return [c, -s, cx - c * cx + s * cy + dx, s, c, cy - s * cx - c * cy + dy]

    return {"identity": [1, 0, 0, 0, 1, 0], "shift": [1, 0, 2.25, 0, 1, -3.5], "small": similarity(1.0, 0.3, 0.4, -0.7),
            "turned": similarity(1.0, 7.0, 1.0, 2.0), "large": similarity(1.02, -0.8, 3.0, 1.0),
            "shrunk": similarity(0.7, 1.0, 0.0, 0.0), "half turn": similarity(1.0, 180.0, 0.3, 0.2),
            "steep": [1.0, 0.01, 0.3, 0.0, 9.0, 2.2], "outside": [1, 0, 1.0e6, 0, 1, 0]}


@pytest.mark.parametrize("h,w", [(12, 20), (40, 33), (67, 97), (9, 260)])
@pytest.mark.parametrize("name", list(_maps(10, 10)))
def test_image_and_parameter_gradients(native, name, h, w):
    from glass_gb300.adjoint import warp_affine

    rng = np.random.default_rng(h * w + len(name))
    image = (100.0 + 20.0 * rng.standard_normal((h, w))).astype(np.float32)
    if w > 50:
        image[h // 2, w // 2] = np.nan
    grad = rng.standard_normal((h, w)).astype(np.float32)
    grad[rng.random((h, w)) < 0.2] = 0.0
    theta = np.array(_maps(h, w)[name], dtype=np.float64)
    src = torch.from_numpy(image).cuda().requires_grad_()
    t = torch.from_numpy(theta).requires_grad_()
    out = warp_affine(src, t, "lanczos3", 0.0)
    got_src, got_t = torch.autograd.grad(out, (src, t), torch.from_numpy(grad).cuda())

    src64 = torch.from_numpy(image.astype(np.float64)).requires_grad_()
    t64 = torch.from_numpy(theta).requires_grad_()
    out64 = warp_affine_reference(src64, t64, "lanczos3", 0.0)
    want_src, want_t = torch.autograd.grad(out64, (src64, t64), torch.from_numpy(grad.astype(np.float64)))
    want_src = torch.nan_to_num(want_src)
    scale = want_src.abs().max().item()
    assert (got_src.cpu().double() - want_src).abs().max().item() <= 1e-5 * scale
    # each term's rounding: taps of 200 times weight sums of 6, some 2^-24 each,
    # times the incoming gradient and the coordinate
    limit = 1e-4 * np.abs(grad).sum() * np.array([w, h, 1, w, h, 1])
    assert np.all(np.abs((got_t - want_t).numpy()) <= limit)


def test_parameter_gradient_over_a_background(native):
    """A background of 3000 times its noise adds nothing to the derivatives; the
    terms of the sum keep their own rounding (a few 2^-24 each of up to twice the
    noise) and the sum of 6000 of them cancels to some tenth of its root."""
    from glass_gb300.adjoint import warp_affine

    h, w = 64, 96
    rng = np.random.default_rng(17)
    image = (30000.0 + 10.0 * rng.standard_normal((h, w))).astype(np.float32)
    grad = rng.standard_normal((h, w)).astype(np.float32)
    theta = np.array(_maps(h, w)["small"], dtype=np.float64)
    src = torch.from_numpy(image).cuda().requires_grad_()  # both gradients: the scatter kernel's sums
    t = torch.from_numpy(theta).requires_grad_()
    out = warp_affine(src, t, "lanczos3", 0.0)
    _, got = torch.autograd.grad(out, (src, t), torch.from_numpy(grad).cuda())
    t64 = torch.from_numpy(theta).requires_grad_()
    out64 = warp_affine_reference(torch.from_numpy(image.astype(np.float64)), t64, "lanczos3", 0.0)
    (want,) = torch.autograd.grad(out64, (t64,), torch.from_numpy(grad.astype(np.float64)))
    assert ((got - want).norm() / want.norm()).item() <= 1e-5
