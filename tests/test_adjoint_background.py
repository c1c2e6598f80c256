"""The warp's parameter gradient over a background, without the image gradient.

An image that asks for no gradient of its own takes another kernel; the bound is
that of the form with both gradients (tests/test_adjoint_scatter.py): a background
of 3000 times its noise adds nothing to the derivatives, whose terms keep a few
2^-24 of up to twice the noise.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.torch_warp_reference import warp_affine_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("background", [0.0, 1000.0, 30000.0])
@pytest.mark.parametrize("h,w", [(64, 96), (200, 300)])
def test_parameter_gradient_alone(native, background, h, w):
    from glass_gb300.adjoint import warp_affine

    rng = np.random.default_rng(17)
    image = (background + 10.0 * rng.standard_normal((h, w))).astype(np.float32)
    image[h // 2, w // 3] = np.nan
    grad = rng.standard_normal((h, w)).astype(np.float32)
    c, s = np.cos(np.deg2rad(0.3)), np.sin(np.deg2rad(0.3))
    theta = torch.tensor([c, -s, w / 2 - c * w / 2 + s * h / 2 + 0.4, s, c, h / 2 - s * w / 2 - c * h / 2 - 0.7],
                         dtype=torch.float64)
    t = theta.clone().requires_grad_()
    out = warp_affine(torch.from_numpy(image).cuda(), t, "lanczos3", 0.0)
    (got,) = torch.autograd.grad(out, (t,), torch.from_numpy(grad).cuda())
    t64 = theta.clone().requires_grad_()
    out64 = warp_affine_reference(torch.from_numpy(image.astype(np.float64)), t64, "lanczos3", 0.0)
    (want,) = torch.autograd.grad(out64, (t64,), torch.from_numpy(grad.astype(np.float64)))
    assert ((got - want).norm() / want.norm()).item() <= 1e-5
