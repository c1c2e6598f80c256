"""Performance cases of the resident light-stack path, each through the entry
points that a program calls (ResidentPipeline, ResidentCalibratedStack,
warp_affine), with synthetic uint16 light frames made on the GPU.

Kinds:
  step       raw frames on the device -> calibrate, warp, weights, integrate: six maps
  calibrate  raw frames on the device -> calibrated float32 frames
  detect     star catalogs of resident frames
  align      triangle registration, Gauss-Newton refinement and quality of resident frames with catalogs
  warp       calibrate, then warp the frames in place by their registration matrices
  integrate  rejection and weighted integration of a resident, aligned stack: six maps
  graph      the fixed-matrix step (calibrate, weights, fused warp + integration) as one captured graph
  adjoint    differentiable warp of one image, forward and backward (image and parameter gradients)
  host       the whole step from pinned host frames to host maps, registration and local normalisation included
"""

import math

import numpy as np
import torch

from glass_gb300 import _lib
from glass_gb300.adjoint import warp_affine
from glass_gb300.pipeline import Masters, ResidentPipeline, StepConfig

REJECTION = {"none": _lib.GG_REJECT_NONE, "sigma": _lib.GG_REJECT_SIGMA_CLIP,
             "winsorized": _lib.GG_REJECT_WINSORIZED, "linear_fit": _lib.GG_REJECT_LINEAR_FIT}
LFC_ITERATIONS = 5  # integrate_async's default
FLAT_FLOOR = 1.0e-6


def listed():
    return [
        # a thumbnail or region-of-interest stack: nothing but launches
        {"name": "step_8x128", "kind": "step", "frames": 8, "height": 128, "width": 128, "interp": "lanczos3"},
        # ingest of a night's frames from a 16 Mpx camera
        {"name": "calibrate_16x4096", "kind": "calibrate", "frames": 16, "height": 4096, "width": 4096},
        # star catalogs of the same camera's frames
        {"name": "detect_8x4096", "kind": "detect", "frames": 8, "height": 4096, "width": 4096},
        # registration of a 32-frame stack once its catalogs are there
        {"name": "align_32x2048", "kind": "align", "frames": 32, "height": 2048, "width": 2048},
        # resampling onto the reference frame, the default interpolation
        {"name": "warp_16x4096", "kind": "warp", "frames": 16, "height": 4096, "width": 4096, "interp": "lanczos3"},
        # a cropped stack of odd size, bilinear
        {"name": "warp_20x1537x2047", "kind": "warp", "frames": 20, "height": 1537, "width": 2047,
         "interp": "bilinear"},
        # a night of 200 frames, the default rejection (a sixteenth of a 60 Mpx frame)
        {"name": "integrate_200", "kind": "integrate", "frames": 200, "height": 1605, "width": 2400,
         "reject": "winsorized"},
        # 40 frames with plain sigma clipping
        {"name": "integrate_40_sigma", "kind": "integrate", "frames": 40, "height": 2000, "width": 3000,
         "reject": "sigma"},
        # a short stack with linear-fit clipping
        {"name": "integrate_25_linear", "kind": "integrate", "frames": 25, "height": 1024, "width": 1024,
         "reject": "linear_fit"},
        # re-stacking with known matrices, captured once and replayed
        {"name": "graph_32x2048", "kind": "graph", "frames": 32, "height": 2048, "width": 2048,
         "interp": "lanczos3"},
        # gradient-based registration or image fitting in PyTorch
        {"name": "adjoint_4096", "kind": "adjoint", "height": 4096, "width": 4096, "interp": "lanczos3"},
        # what a whole run does for each stack, host to host
        {"name": "host_32x2048", "kind": "host", "frames": 32, "height": 2048, "width": 2048},
    ]


# kind: frames, side of the frame, most samples (frames x pixels) of a drawn case
_RANGES = {
    "step": ((4, 24), (96, 1024), 24 << 20),
    "calibrate": ((2, 32), (128, 4096), 16 << 24),
    "detect": ((1, 16), (256, 4096), 8 << 24),
    "align": ((4, 40), (512, 2048), 32 << 22),
    "warp": ((2, 24), (128, 4096), 16 << 24),
    "integrate": ((3, 256), (96, 3000), 200 * 1605 * 2400),
    "graph": ((4, 40), (128, 2048), 32 << 22),
    "adjoint": ((1, 1), (128, 4096), 1 << 24),
    "host": ((4, 32), (512, 2048), 32 << 22),
}


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(sorted(_RANGES))
    (f0, f1), (s0, s1), most = _RANGES[kind]
    case = {"kind": kind}
    if kind != "adjoint":
        case["frames"] = _log_uniform(rng, f0, f1)
    if kind == "integrate":
        case["reject"] = rng.choice(["winsorized", "winsorized", "sigma", "linear_fit", "none"])
        if case["reject"] == "linear_fit":
            case["frames"] = min(case["frames"], 64)
    if kind in ("step", "warp", "graph", "adjoint"):
        case["interp"] = rng.choice(["lanczos3", "lanczos3", "bilinear"])
    side = min(s1, math.sqrt(most / case.get("frames", 1)) / 1.2)
    h, w = (_log_uniform(rng, s0, side) for _ in range(2))
    # cameras have even sides, crops any
    if rng.random() < 0.6:
        h, w = h & ~1, w & ~3
    case.update(height=h, width=w)
    return case


# ---- inputs -----------------------------------------------------------------------


def _similarity(rng, i, max_shift, max_rotation_deg, integer):
    """Reference -> frame map of frame i (frame 0 is the reference)."""
    if i == 0:
        return np.eye(3)
    t = 0.0 if integer else math.radians(rng.uniform(-max_rotation_deg, max_rotation_deg))
    dx, dy = (rng.uniform(-max_shift, max_shift) for _ in range(2))
    if integer:
        dx, dy = float(round(dx)), float(round(dy))
    return np.array([[math.cos(t), -math.sin(t), dx], [math.sin(t), math.cos(t), dy], [0.0, 0.0, 1.0]])


def _sky(case, seed, integer=False):
    """Raw frames (int16 CUDA tensor with the uint16 bits), masters and the
    frames' moving -> reference matrices: a sky of 850-1150 ADU with a
    gradient, one Gaussian star of FWHM 2-5 px per 2100 px (peak 500-20000
    ADU), shot and read noise, cosmic rays on 1e-4 of the pixels, hot dark
    pixels and a vignetted flat."""
    n, h, w = case.get("frames", 1), case["height"], case["width"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def randn():
        return torch.randn((h, w), device="cuda", generator=gen)

    stars = max(40, h * w // 2100)
    xy = rng.uniform((-40.0, -40.0), (w + 40.0, h + 40.0), (stars, 2))
    peak = torch.as_tensor(np.exp(rng.uniform(math.log(500.0), math.log(20000.0), stars)), device="cuda")
    two_s2 = torch.as_tensor(2.0 * (rng.uniform(2.0, 5.0, stars) / 2.355) ** 2, device="cuda")[:, None, None]
    offs = torch.arange(-7, 8, device="cuda")
    yy = torch.linspace(-1.0, 1.0, h, device="cuda")[:, None]
    xx = torch.linspace(-1.0, 1.0, w, device="cuda")[None, :]
    vignette = 1.0 - 0.05 * (xx * xx + yy * yy)
    bias = 500.0 + 0.5 * randn()
    dark = 6.0 + 0.5 * randn()
    hot = torch.as_tensor(rng.integers(0, h * w, max(1, h * w // 10000)), device="cuda")
    dark.view(-1)[hot] = 1500.0
    flat = vignette * (1.0 + 0.005 * randn())
    raw = torch.empty((n, h, w), device="cuda", dtype=torch.int16)
    matrices = np.empty((n, 3, 3))
    for i in range(n):
        fwd = _similarity(rng, i, min(20.0, 0.1 * min(h, w)), 0.3, integer)
        matrices[i] = np.linalg.inv(fwd)
        pos = torch.as_tensor(xy @ fwd[:2, :2].T + fwd[:2, 2], device="cuda")
        centre = torch.floor(pos).to(torch.int64)
        gx, gy = (centre[:, k : k + 1] + offs[None, :] for k in (0, 1))
        ex, ey = ((g.to(torch.float64) - pos[:, k : k + 1]) ** 2 for k, g in ((0, gx), (1, gy)))
        psf = peak[:, None, None] * torch.exp(-(ey[:, :, None] + ex[:, None, :]) / two_s2)
        ok = ((gy >= 0) & (gy < h))[:, :, None] & ((gx >= 0) & (gx < w))[:, None, :]
        at = gy[:, :, None] * w + gx[:, None, :]
        signal = float(rng.uniform(850.0, 1150.0)) * (1.0 + 0.025 * float(rng.uniform(-1, 1)) * xx +
                                                      0.025 * float(rng.uniform(-1, 1)) * yy)
        signal.view(-1).index_put_((at[ok],), psf[ok].to(torch.float32), accumulate=True)
        signal = signal * vignette + dark
        frame = signal + torch.sqrt(signal) * randn() + 500.0 + 5.0 * randn()
        hits = rng.integers(0, h * w - w - 1, max(1, h * w // 25000))
        energy = torch.as_tensor(rng.uniform(5000.0, 60000.0, hits.size), device="cuda", dtype=torch.float32)
        for step in (0, 1, w, w + 1):
            frame.view(-1).index_put_((torch.as_tensor(hits + step, device="cuda"),), energy, accumulate=True)
        v = torch.clamp(torch.round(frame), 0.0, 65535.0).to(torch.int32)
        raw[i] = torch.where(v > 32767, v - 65536, v).to(torch.int16)
    return raw, [m.cpu().numpy() for m in (bias, dark, flat)], matrices


_stream_of_program = []


def _stream():
    """The one stream that the program enqueues its stacks' work on."""
    if not _stream_of_program:
        _stream_of_program.append(torch.cuda.Stream())
    return _stream_of_program[0].cuda_stream


def _config(case):
    return StepConfig(rejection=REJECTION[case.get("reject", "winsorized")],
                      interpolation=case.get("interp", "lanczos3"), star_max_stars=2048, refine_method="gradient",
                      local_normalization_tile=256 if case["kind"] == "host" else 0)


def _star_image(case, seed):
    raw, _, matrices = _sky(dict(case, frames=2), seed)
    image = raw[1].to(torch.int32).bitwise_and(0xFFFF).to(torch.float32) - 500.0
    inv = np.linalg.inv(matrices[1])
    grad = torch.randn((case["height"], case["width"]), device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(seed + 1))
    return image, torch.as_tensor(inv[:2].reshape(-1), dtype=torch.float32), grad


def _weights(case, seed):
    w = np.random.default_rng(seed + 2).uniform(0.5, 1.5, case["frames"]).astype(np.float32)
    w[case["frames"] // 3] = 0.0  # a frame that failed its quality check
    return w


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "adjoint":
        image, theta, grad = _star_image(case, seed)
        state.update(image=image.requires_grad_(), theta=theta.requires_grad_(), grad=grad)
        return state
    n, h, w = case["frames"], case["height"], case["width"]
    raw, masters, matrices = _sky(case, seed, integer=case["kind"] == "integrate")
    torch.cuda.synchronize()
    pipe = ResidentPipeline(n, h, w, Masters(*masters), _config(case))
    pipe.set_stream(_stream())
    state.update(pipe=pipe, raw=raw, matrices=matrices)
    if case["kind"] == "host":
        state["host_raw"] = raw.cpu().pin_memory().numpy().view(np.uint16)
        del state["raw"]
        kinds = (torch.float32, torch.float32, torch.int16, torch.int16, torch.int16, torch.int16)
        maps = [torch.empty((h, w), dtype=t).pin_memory().numpy() for t in kinds]
        state["maps"] = tuple(m.view(np.uint16) if 2 <= k <= 4 else m for k, m in enumerate(maps))
        return state
    if case["kind"] in ("detect", "align", "integrate"):
        pipe.calibrate_device(raw.data_ptr())
        if case["kind"] == "align":
            pipe.detect()
        if case["kind"] == "integrate":
            pipe.warp(matrices)  # integer shifts: borders without samples
            state["weights"] = _weights(case, seed)
        pipe.stack.synchronize()
        del state["raw"]
    if case["kind"] == "graph":
        pipe.capture_graph(raw.data_ptr(), matrices)
    return state


# ---- one pass ----------------------------------------------------------------------


class _Map:
    """Device memory of a stack, which lives as long as the tensor made of it."""

    def __init__(self, stack, address, shape, typestr):
        self.stack = stack
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (address, False), "version": 2,
                                         "strides": None}


def _device_maps(stack, shape):
    """The stack's six device maps as tensors (counts as 16-bit integers)."""
    p = stack.device_pointers()
    kinds = {"master": "<f4", "weight": "<f4", "coverage": "<i2", "low": "<i2", "high": "<i2", "dq": "<i2"}
    return {k: torch.as_tensor(_Map(stack, p[k], shape, t), device="cuda") for k, t in kinds.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "adjoint":
        out = warp_affine(state["image"], state["theta"], case["interp"], 0.0, True)
        grads = torch.autograd.grad(out, (state["image"], state["theta"]), state["grad"])
        return {"out": out, "grad_image": grads[0], "grad_theta": grads[1]}
    pipe = state["pipe"]
    shape = (case["height"], case["width"])
    if kind == "step":
        pipe.step_device(state["raw"].data_ptr(), state["matrices"])
        return _device_maps(pipe.stack, shape)
    if kind == "graph":
        pipe.launch_graph()
        return _device_maps(pipe.stack, shape)
    if kind == "integrate":
        pipe.stack.integrate_async(state["weights"], REJECTION[case["reject"]])
        return _device_maps(pipe.stack, shape)
    if kind == "calibrate":
        pipe.calibrate_device(state["raw"].data_ptr())
        return [pipe.stack.frame_tensor(k) for k in range(case["frames"])]
    if kind == "warp":
        pipe.calibrate_device(state["raw"].data_ptr())
        pipe.warp(state["matrices"])
        return [pipe.stack.frame_tensor(k) for k in range(case["frames"])]
    if kind == "detect":
        stars, info = pipe.stack.detect_stars(range(case["frames"]), 5.0, 2048, with_info=True,
                                              catalog_max_eccentricity=0.8)
        table = {f: np.zeros((len(stars), 2048), stars[0].dtype[f]) for f in stars[0].dtype.names if f != "pad"}
        for k, s in enumerate(stars):
            for f in table:
                table[f][k, : len(s)] = s[f]
        return {"stars": table, "count": np.array([len(s) for s in stars]),
                "median": np.array([i["median"] for i in info], np.float32),
                "mad": np.array([i["mad"] for i in info], np.float32)}
    if kind == "align":
        matrices, ok = pipe.register(0)
        matrices = pipe.refine(matrices, 0)
        quality = pipe.assess(matrices, 0)
        score = np.full(case["frames"], -1.0)
        for q in quality:
            score[q["frame"]] = q.get("score", -1.0)
        return {"matrices": matrices, "ok": ok, "score": score}
    maps = pipe.step_host(state["host_raw"], register=True, out=state["maps"])
    return {k: m.view(np.int16) if m.dtype == np.uint16 else m
            for k, m in zip(("master", "weight", "coverage", "low", "high", "dq"), maps)}


def work(case):
    """Bytes: raw 2 B, frames 4 B, masters 12 B and maps 16 B per pixel, each
    once.  Operations: two per tap of a window and per weight polynomial's
    coefficient, a sort's comparisons and a few sums per integrated sample."""
    px = case["height"] * case["width"]
    n = case.get("frames", 1)
    lanczos = case.get("interp", "lanczos3") == "lanczos3"
    warp = n * px * (156.0 if lanczos else 9.0)
    integrate = n * px * (math.log2(max(n, 2)) + 12.0)
    kind = case["kind"]
    if kind == "adjoint":
        return {"bytes": 16.0 * px, "flops": px * (450.0 if lanczos else 30.0)}
    if kind == "calibrate":
        return {"bytes": px * (6.0 * n + 12.0), "flops": 3.0 * n * px}
    if kind == "warp":  # calibrated frames in, warped frames out
        return {"bytes": px * (14.0 * n + 12.0), "flops": 3.0 * n * px + warp}
    if kind == "integrate":
        return {"bytes": px * (4.0 * n + 16.0), "flops": integrate}
    if kind == "detect":
        return {"bytes": 4.0 * n * px, "flops": 20.0 * n * px}
    if kind == "align":  # about a million samples of each frame and its reference
        samples = min(px / 9.0, 1.0e6) * n
        return {"bytes": 8.0 * samples, "flops": 2000.0 * samples}
    return {"bytes": px * (2.0 * n + 28.0), "flops": 3.0 * n * px + warp + integrate}


# ---- the same in 64 bits -----------------------------------------------------------


def _raw64(raw):
    return raw.to(torch.int32).bitwise_and(0xFFFF).to(torch.float64)


def _calibrated64(raw, masters):
    bias, dark, flat = (torch.as_tensor(m, device="cuda").to(torch.float64) for m in masters)
    return (_raw64(raw) - dark - bias) / torch.clamp(flat, min=FLAT_FLOOR)


def _l3(d):
    """sinc(d) sinc(d / 3) and its derivative."""
    a = math.pi * d
    small = a.abs() < 1e-8
    a = torch.where(small, torch.full_like(a, 1e-8), a)
    f, g = torch.sin(a) / a, torch.sin(a / 3) / (a / 3)
    df = math.pi * (torch.cos(a) - f) / a
    dg = math.pi * (torch.cos(a / 3) - g) / a
    return torch.where(small, torch.ones_like(a), f * g), torch.where(small, torch.zeros_like(a), df * g + f * dg)


def _window64(inv, h, w, lanczos):
    """(validity, first tap column and row, weights and derivatives per axis) of every output pixel."""
    y, x = (t.to(torch.float64) for t in torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"),
                                                       indexing="ij"))
    sx = float(inv[0, 0]) * x + float(inv[0, 1]) * y + float(inv[0, 2])
    sy = float(inv[1, 0]) * x + float(inv[1, 1]) * y + float(inv[1, 2])
    if lanczos:
        ok = (sx >= 2) & (sx < w - 3) & (sy >= 2) & (sy < h - 3)
    else:
        ok = (sx >= 0) & (sx <= w - 1) & (sy >= 0) & (sy <= h - 1)
    out = [ok]
    for s, size in ((sx, w), (sy, h)):
        s = torch.where(ok, s, torch.full_like(s, 3.0 if lanczos else 0.0))
        first = torch.floor(s)
        t = s - first
        if lanczos:
            taps = [_l3(t - k) for k in range(-2, 4)]
            cols = [(first + k).to(torch.int64) for k in range(-2, 4)]
        else:
            taps = [(1 - t, -torch.ones_like(t)), (t, torch.ones_like(t))]
            cols = [(first + k).to(torch.int64).clamp(max=size - 1) for k in (0, 1)]
        out.append((cols, taps))
    return out


def _sums64(image, inv, interp, derivatives=False):
    """Numerator and denominator of the window sums (and their derivatives along both axes)."""
    h, w = image.shape
    ok, (cx, wx), (cy, wy) = _window64(inv, h, w, interp == "lanczos3")
    sums = [torch.zeros((h, w), dtype=torch.float64, device="cuda") for _ in range(6 if derivatives else 2)]
    flat = image.reshape(-1)
    for j in range(len(cy)):
        for i in range(len(cx)):
            v = flat[cy[j] * w + cx[i]]
            parts = [wx[i][0] * wy[j][0]]
            if derivatives:
                parts += [wx[i][1] * wy[j][0], wx[i][0] * wy[j][1]]
            for k, p in enumerate(parts):
                sums[2 * k] += p * v
                sums[2 * k + 1] += p
    return ok, sums, (cx, wx), (cy, wy)


def _warped64(image, matrix, interp):
    ok, (num, den), _, _ = _sums64(image, np.linalg.inv(matrix), interp)
    return torch.where(ok, num / den, torch.full_like(num, math.nan))


def _adjoint64(case, seed):
    image, theta, grad = _star_image(case, seed)
    inv = np.eye(3)
    inv[:2] = theta.to(torch.float64).numpy().reshape(2, 3)
    image, grad = image.to(torch.float64), grad.to(torch.float64)
    ok, (num, den, nx, dx, ny, dy), (cx, wx), (cy, wy) = _sums64(image, inv, case["interp"], True)
    g = torch.where(ok, grad, torch.zeros_like(grad))
    out = num / den
    grad_image = torch.zeros_like(image).reshape(-1)
    for j in range(len(cy)):
        for i in range(len(cx)):
            grad_image.index_add_(0, (cy[j] * image.shape[1] + cx[i]).reshape(-1),
                                  (g / den * wx[i][0] * wy[j][0]).reshape(-1))
    gx, gy = g * (nx - out * dx) / den, g * (ny - out * dy) / den
    y, x = (t.to(torch.float64) for t in torch.meshgrid(*(torch.arange(s, device="cuda") for s in image.shape),
                                                       indexing="ij"))
    grad_theta = torch.stack([(s * c).sum() for s in (gx, gy) for c in (x, y, torch.ones_like(x))])
    return {"out": torch.where(ok, out, torch.zeros_like(out)), "grad_image": grad_image.reshape(image.shape),
            "grad_theta": grad_theta.cpu()}


def _kept_linear64(s, cnt, iterations):
    """Kept value interval of linear-fit clipping at 3 / 3: fit of the sorted
    samples to a line over their rank, mean absolute residual as the scale,
    samples clipped from both ends, repeated on the kept ranks."""
    n, px = s.shape
    rank = torch.arange(n, device="cuda")[:, None].expand(n, px)
    lo, hi = torch.zeros_like(cnt), cnt.clone()
    live = cnt >= 3
    for _ in range(iterations):
        live = live & (hi - lo >= 3)
        inside = (rank >= lo) & (rank < hi)
        y = torch.where(inside, s, torch.zeros_like(s))
        m = (hi - lo).clamp(min=1).to(torch.float64)
        r = torch.where(inside, rank - lo - 0.5 * (m - 1), torch.zeros_like(s))
        a, b = y.sum(0) / m, (r * y).sum(0) / (m * (m * m - 1) / 12).clamp(min=1e-30)
        fit = a + b * r
        sigma = torch.where(inside, (y - fit).abs(), torch.zeros_like(s)).sum(0) / m
        stay_lo = inside & ~(y < fit - 3.0 * sigma)
        stay_hi = inside & ~(y > fit + 3.0 * sigma)
        new_lo = torch.where(stay_lo, rank, n).amin(0)
        new_hi = torch.maximum(torch.where(stay_hi, rank, -1).amax(0) + 1, new_lo)
        live = live & (new_hi > new_lo)
        changed = live & ((new_lo != lo) | (new_hi != hi))
        # samples equal to a kept end are kept
        first = s.gather(0, new_lo.clamp(0, n - 1)[None])[0]
        last = s.gather(0, (new_hi - 1).clamp(0, n - 1)[None])[0]
        new_lo = torch.where(inside & (s == first), rank, n).amin(0)
        new_hi = torch.where(inside & (s == last), rank, -1).amax(0) + 1
        changed = changed & ((new_lo != lo) | (new_hi != hi))
        lo, hi = torch.where(changed, new_lo, lo), torch.where(changed, new_hi, hi)
        live = changed
    return s.gather(0, lo.clamp(0, n - 1)[None])[0], s.gather(0, (hi - 1).clamp(0, n - 1)[None])[0]


def _integrated64(v, w, reject):
    """Master and weight of the samples v (frames x pixels) with weights w at 3 / 3, 3 samples, half rejected."""
    w = torch.as_tensor(w, device="cuda", dtype=torch.float64)[:, None]
    valid = torch.isfinite(v) & (w > 0)
    cnt = valid.sum(0)
    kept = valid
    if reject != "none":
        s = torch.where(valid, v, torch.full_like(v, math.inf)).sort(0).values
        some = cnt.clamp(min=1)
        n = some.to(torch.float64)

        def pick(i):
            return s.gather(0, i.to(torch.int64).clamp(min=0)[None])[0]

        def percentile(q):
            pos = (n - 1) * q
            lo = torch.floor(pos)
            t = pos - lo
            return pick(lo) * (1 - t) + pick(torch.minimum(lo + 1, n - 1)) * t

        def std(x):
            mean = torch.where(valid, x, torch.zeros_like(x)).sum(0) / n
            return mean, torch.sqrt(torch.where(valid, (x - mean) ** 2, torch.zeros_like(x)).sum(0) / n)

        if reject == "linear_fit":
            low, high = _kept_linear64(s, cnt, LFC_ITERATIONS)
        else:
            centre = percentile(0.5)
            if reject == "sigma":
                scale = std(v)[1]
            else:
                scale = (percentile(0.75) - percentile(0.25)) / 1.349
                scale = torch.where(scale > 0, scale, std(v)[1])
                centre, wins = std(torch.minimum(torch.maximum(v, centre - 3.0 * scale), centre + 3.0 * scale))
                scale = torch.where(wins > 0, wins, scale)
            low, high = centre - 3.0 * scale, centre + 3.0 * scale
        out = valid & ((v < low) | (v > high))
        gone = out.sum(0)
        allowed = (cnt - gone >= 3) & (gone <= 0.5 * cnt)
        kept = valid & ~(out & allowed)
    total = torch.where(kept, w.expand_as(v), torch.zeros_like(v)).sum(0)
    some = torch.where(kept, w * v, torch.zeros_like(v)).sum(0)
    return torch.where(total > 0, some / total.clamp(min=1e-300), torch.zeros_like(total)), total


def _maps64(frames, w, reject):
    n, h, wd = frames.shape
    out = torch.empty((2, h, wd), dtype=torch.float64, device="cuda")
    rows = max(1, (1 << 26) // (n * wd))
    for y in range(0, h, rows):
        part = frames[:, y : y + rows].reshape(n, -1).to(torch.float64)
        m, t = _integrated64(part, w, reject)
        out[0, y : y + rows], out[1, y : y + rows] = m.reshape(-1, wd), t.reshape(-1, wd)
    return {"master": out[0], "weight": out[1], "coverage": None, "low": None, "high": None, "dq": None}


def _snr64(frames):
    out = []
    for f in frames:
        v = f[torch.isfinite(f)].to(torch.float64)
        mean = v.mean()
        out.append(float(mean.abs() / torch.sqrt(((v - mean) ** 2).mean())))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("detect", "align", "host"):
        # star lists, matrices and scores are searches and 64-bit results of their own; the whole run follows them
        return None
    if kind == "adjoint":
        return _adjoint64(case, seed)
    raw, masters, matrices = _sky(case, seed, integer=kind == "integrate")
    if kind == "calibrate":
        return [_calibrated64(r, masters) for r in raw]
    if kind == "integrate":
        # the aligned float32 frames themselves are the input here
        bias, dark, flat = (torch.as_tensor(m, device="cuda") for m in masters)
        n, h, w = raw.shape
        frames = torch.full((n, h, w), math.nan, device="cuda")
        for k in range(n):
            dx, dy = int(matrices[k, 0, 2]), int(matrices[k, 1, 2])
            one = (_raw64(raw[k]).to(torch.float32) - dark - bias) / torch.clamp(flat, min=FLAT_FLOOR)
            if k == 0:
                frames[k] = one
                continue
            # default interpolation's validity: 2 <= source < size - 3
            y0, y1, x0, x1 = 2 + dy, h - 3 + dy, 2 + dx, w - 3 + dx
            a, b, c, d = max(0, y0), min(h, y1), max(0, x0), min(w, x1)
            frames[k, a:b, c:d] = one[a - dy : b - dy, c - dx : d - dx]
        return _maps64(frames, _weights(case, seed), case["reject"])
    calibrated = [_calibrated64(r, masters) for r in raw]
    # the step and the warp leave the reference frame as it is, the fused form samples it too
    warped = [c if k == 0 and kind != "graph" else _warped64(c, matrices[k], case["interp"])
              for k, c in enumerate(calibrated)]
    if kind == "warp":
        return warped
    weights = _snr64(calibrated if kind == "graph" else warped)
    return _maps64(torch.stack(warped), weights, "winsorized")
