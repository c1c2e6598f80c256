"""Coefficients of the Lanczos3 tap weights used by the CUDA warps.

For a sample at fractional offset t in [0, 1) the six taps k = -2..3 weigh
L(t - k) with L(d) = sinc(d) sinc(d / 3) (zero for |d| >= 3).  With
u = t - 1/2 the taps pair up as L(c + u) and L(c - u) for c = 1/2, 3/2, 5/2
(L is even), so each pair is E_c(u) +- O_c(u) with E_c even and O_c odd in
u.  This script fits E_c(u) = sum_j e_j u^(2j) and O_c(u) = u sum_j o_j u^(2j)
(j = 0..5) by float64 least squares on u in [0, 1/2] and prints the six
Horner evaluations, with the coefficients as float literals (immediate
operands of the fused multiply-adds), pasted into csrc/sampling.cuh; the fit
error is below 3e-10, far under float32 rounding.  It also prints the
derivatives d/dx of those float32 polynomials (coefficients j * c_j, degree
4), pasted into csrc/adjoint.cuh: the Gauss-Newton refinement differentiates
exactly the weights the warp samples with.

Those weights are accurate in absolute terms: near a whole offset, where all
but one tap vanish, the vanishing ones are what rounding leaves of E +- O.  The
image gradient of the warp adjoint spreads each pixel by its weights, so it takes
them from polynomials about the nearer tap instead (fit_centred): with s in
[0, 1/2] the distance to it and x = s^2, L(s) = 1 + x P(x), the pairs L(k - s)
and L(k + s), k = 1 and 2, are x Q(x) +- s R(x), and L(3 - s) = x S(s), so each
vanishes with s to full relative accuracy.  Fitted in float64 at Chebyshev points
(above s = 0.003, below which the quotients lose digits); the fit error is below
3e-11, for S 1e-9.
Run: python -m glass_gb300.lanczos_poly [--derivatives | --centred]
"""

from __future__ import annotations

import numpy as np

DEGREE = 5


def lanczos3(d: np.ndarray) -> np.ndarray:
    d = np.asarray(d, dtype=np.float64)
    out = np.sinc(d) * np.sinc(d / 3.0)
    out[np.abs(d) >= 3.0] = 0.0
    return out


def fit(center: float, samples: int = 20001):
    u = np.linspace(0.0, 0.5, samples)
    even = 0.5 * (lanczos3(center + u) + lanczos3(center - u))
    odd = 0.5 * (lanczos3(center + u) - lanczos3(center - u))
    basis = np.vander(u * u, DEGREE + 1, increasing=True)
    e, *_ = np.linalg.lstsq(basis, even, rcond=None)
    o, *_ = np.linalg.lstsq(u[:, None] * basis, odd, rcond=None)
    err = max(np.abs(basis @ e - even).max(), np.abs((u[:, None] * basis) @ o - odd).max())
    return e, o, err


CENTRED_DEGREE = {"p": 5, "q1": 5, "r1": 5, "q2": 5, "r2": 5, "s": 7}


def fit_centred(samples: int = 4000) -> dict[str, tuple[np.ndarray, float]]:
    """Coefficients (lowest power first) and fit error of each polynomial."""
    s = 0.25 * (1.0 - np.cos(np.pi * (np.arange(samples) + 0.5) / samples))
    s = s[s > 0.003]
    x = s * s
    values = {"p": ((lanczos3(s) - 1.0) / x, x), "s": (lanczos3(3.0 - s) / x, s)}
    for k in (1, 2):
        values[f"q{k}"] = (0.5 * (lanczos3(k - s) + lanczos3(k + s)) / x, x)
        values[f"r{k}"] = (0.5 * (lanczos3(k - s) - lanczos3(k + s)) / s, x)
    out = {}
    for name, (y, v) in values.items():
        basis = np.vander(v, CENTRED_DEGREE[name] + 1, increasing=True)
        c, *_ = np.linalg.lstsq(basis, y, rcond=None)
        out[name] = (c, float(np.abs(basis @ c - y).max()))
    return out


def horner_source(name: str, coefs) -> str:
    c = [f"{float(v):.9e}f" for v in coefs]
    body = f"  float p = {c[5]};\n"
    for j in (4, 3, 2, 1):
        body += f"  p = __fmaf_rn(p, x, {c[j]});\n"
    body += f"  return __fmaf_rn(p, x, {c[0]});\n"
    return f"__device__ __forceinline__ float l3_{name}(float x) {{\n{body}}}"


def derivative_source(name: str, coefs32) -> str:
    """d/dx of the float32 polynomial sum_j c_j x^j (degree 4, Horner)."""
    d = [float(j) * float(coefs32[j]) for j in range(1, DEGREE + 1)]
    c = [f"{float(np.float32(v)):.9e}f" for v in d]
    body = f"  float p = {c[4]};\n"
    for j in (3, 2, 1):
        body += f"  p = __fmaf_rn(p, x, {c[j]});\n"
    body += f"  return __fmaf_rn(p, x, {c[0]});\n"
    return f"__device__ __forceinline__ float l3_{name}_dx(float x) {{\n{body}}}"


def centred_source() -> str:
    lines = []
    for name, (c, _) in fit_centred().items():
        body = ", ".join(f"{float(np.float32(v)):.9e}f" for v in c)
        lines.append(f"constexpr float kCentred_{name}[{len(c)}] = {{{body}}};")
    return "\n".join(lines)


def main(derivatives: bool = False) -> None:
    for name, center in (("a", 0.5), ("b", 1.5), ("c", 2.5)):
        e, o, err = fit(center)
        if derivatives:
            print(derivative_source("even_" + name, e.astype(np.float32)))
            print(derivative_source("odd_" + name, o.astype(np.float32)))
            continue
        print(f"// pair {name.upper()} (c = {center}): max fit error {err:.1e}")
        print(horner_source("even_" + name, e.astype(np.float32)))
        print(horner_source("odd_" + name, o.astype(np.float32)))


if __name__ == "__main__":
    import sys

    if "--centred" in sys.argv[1:]:
        print(centred_source())
    else:
        main(derivatives="--derivatives" in sys.argv[1:])
