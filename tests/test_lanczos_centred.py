"""Lanczos3 weights about the nearer tap, which the image gradient is made of.

CPU: the header's table is the fit; evaluated in float32 as the kernel does, each
weight is within 4e-7 of its own size (float32 Horner rounds each of some eight
steps by 2^-24, the pairs' difference loses a factor of three), each derivative
within 1e-6, and the weights' sum, of a number near 1 and a small one, within
1.2e-7.

GPU: at offsets next to a whole one the image gradient keeps that accuracy: a
pixel of it is a sum of 36 products of weights that vanish with the offset and
one that does not.  Two weights of 4e-7, the normalisation and the sum's
rounding make 1.5e-6 of each product; the bound takes the products' magnitudes.
"""

from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

from glass_gb300.lanczos_poly import CENTRED_DEGREE, fit_centred, lanczos3

HEADER = Path(__file__).resolve().parent.parent / "glass_gb300" / "csrc" / "adjoint.cuh"


def _table():
    out = {}
    for name, body in re.findall(r"kCentred_(\w+)\[\d+\] = \{(.*?)\};", HEADER.read_text(), re.S):
        out[name] = np.array([float(v) for v in re.findall(r"-?\d\.\d+e[+-]\d+", body)], dtype=np.float32)
    return out


def test_table_is_the_fit():
    table, fit = _table(), fit_centred()
    assert set(table) == set(CENTRED_DEGREE)
    for name, (c, err) in fit.items():
        assert err < 1e-9
        np.testing.assert_array_equal(table[name], c.astype(np.float32))


def _fma(a, b, c):
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(np.float32)


def _horner(c, x):
    p = np.full_like(x, c[-1])
    dp = np.full_like(x, np.float32(len(c) - 1) * c[-1])
    for j in range(len(c) - 2, -1, -1):
        p = _fma(p, x, c[j])
        if j > 0:
            dp = _fma(dp, x, np.float32(j) * c[j])
    return p, dp


def _weights(t):
    f32, table = np.float32, _table()
    lower = t <= f32(0.5)
    s = np.where(lower, t, f32(1.0) - t).astype(np.float32)
    x, s2 = s * s, s + s
    x2 = x + x
    v, d, even = [None] * 6, [None] * 6, np.float32(0.0)
    p0, dp0 = _horner(table["p"], x)
    p, dp = _horner(table["p"], x)
    v[2], d[2] = _fma(x, p, 1.0), s2 * _fma(x, dp, p)
    for k, near, far in ((1, 3, 1), (2, 4, 0)):
        q, dq = _horner(table[f"q{k}"], x)
        r, dr = _horner(table[f"r{k}"], x)
        even = even + q
        e, de, do = x * q, s2 * _fma(x, dq, q), _fma(x2, dr, r)
        v[near], v[far], d[near], d[far] = _fma(s, r, e), _fma(-s, r, e), de + do, de - do
    p, dp = _horner(table["s"], s)
    v[5], d[5] = x * p, _fma(x, dp, s2 * p)
    w = [np.where(lower, v[i], v[5 - i]) for i in range(6)]
    dw = [np.where(lower, d[i], -d[5 - i]) for i in range(6)]
    return np.array(w), np.array(dw), _fma(x, _fma(2.0, even, p0 + p), 1.0)


def test_float32_weights_have_relative_accuracy():
    t = np.concatenate([np.linspace(0.0, 1.0, 20001)[:-1], 10.0 ** np.linspace(-9, -1, 200)]).astype(np.float32)
    w, dw, total = _weights(t)
    d = t.astype(np.float64)[None] - np.arange(-2, 4)[:, None]
    want = lanczos3(d)
    # an offset of zero leaves np.sinc's own rounding of the vanishing taps
    assert (np.abs(w - want) <= 4e-7 * np.abs(want) + 1e-16).all()
    assert np.abs(total - want.sum(0)).max() <= 1.2e-7
    h = 1e-5
    slope = (lanczos3(d + h) - lanczos3(d - h)) / (2 * h)  # accurate to some 1e-9
    inside = (np.abs(d) + h) < 3.0
    assert np.abs(dw - slope)[inside].max() <= 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0.0, 1e-6, 1e-4, 1e-3, 0.02, 0.25, 0.5, 0.75, 0.999, 1.0 - 1e-6])
def test_image_gradient_next_to_a_whole_offset(native, shift):
    import torch

    from glass_gb300.adjoint import warp_affine
    from tests.torch_warp_reference import warp_affine_reference

    h, w = 40, 70
    rng = np.random.default_rng(3)
    image = torch.from_numpy(rng.normal(100.0, 20.0, (h, w)).astype(np.float32))
    grad = torch.from_numpy(rng.standard_normal((h, w)).astype(np.float32))
    theta = torch.tensor([1.0, 0.0, 2.0 + shift, 0.0, 1.0, -1.0 + 0.7 * shift], dtype=torch.float64)
    src = image.cuda().requires_grad_()
    t = theta.clone().requires_grad_()
    (got, _) = torch.autograd.grad(warp_affine(src, t, "lanczos3", 0.0), (src, t), grad.cuda())

    def exact(g):
        src64 = image.double().requires_grad_()
        out = warp_affine_reference(src64, theta, "lanczos3", 0.0)
        return torch.autograd.grad(out, src64, g)[0]

    # magnitudes of the products: the weights' signs undone axis by axis
    tx, ty = (theta[2] % 1.0).item(), (theta[5] % 1.0).item()
    ax, ay = (np.abs(lanczos3(v - np.arange(-2, 4))) for v in (tx, ty))
    norm = abs(lanczos3(tx - np.arange(-2, 4)).sum() * lanczos3(ty - np.arange(-2, 4)).sum())
    limit = np.zeros((h + 16, w + 16))
    x0, y0 = int(np.floor(theta[2].item())), int(np.floor(theta[5].item()))
    for y in range(h):
        for x in range(w):
            if 2 <= x + x0 < w - 3 and 2 <= y + y0 < h - 3:
                limit[y + y0 + 6:y + y0 + 12, x + x0 + 6:x + x0 + 12] += abs(grad[y, x].item()) * np.outer(ay, ax) / norm
    limit = 1.5e-6 * limit[8:-8, 8:-8] + 1e-15
    error = np.abs(got.cpu().double().numpy() - exact(grad.double()).numpy())
    assert (error <= limit).all(), (error / limit).max()
