"""Launches that carry their parameters and finish their own work.

Calibration of any pixel count from any 2-byte aligned address (whole vectors,
shifted pairs of vectors, single samples at the ends of the buffer), with the
non-finite counts of a launch published by its last CTA; frame views whose slot
table is kept on the host until a warp moves a frame, captured warps included.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import calibration as ocal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(1, 1), (3, 5), (8, 8), (7, 9), (33, 41), (64, 130), (101, 203)])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_calibration_of_any_size_and_address(native, h, w, offset):
    import torch

    from glass_gb300 import _lib

    rng = np.random.default_rng(h * w + offset)
    n = 37  # two launches
    raw = rng.integers(0, 65536, (n, h, w), dtype=np.uint16)
    bias, dark = (rng.normal(m, 3.0, (h, w)).astype(np.float32) for m in (500.0, 20.0))
    flat = rng.uniform(0.5, 1.5, (h, w)).astype(np.float32)
    flat[h // 2, w // 3] = np.nan
    buffer = torch.zeros(offset + raw.size, dtype=torch.int16, device="cuda")
    buffer[offset:] = torch.from_numpy(raw.view(np.int16).reshape(-1)).cuda()
    torch.cuda.synchronize()
    s = native.ResidentCalibratedStack(n, h, w)
    s.set_calibration_masters(bias, dark, flat)
    params = _lib.CalibParams(0, 1.5, 1.0e-6, 0.25)
    # the last frame first, and frame 3 a second time with the raw of frame 4
    order = np.array([n - 1, *range(n - 1), 3], dtype=np.int64)[: n + 1]
    take = np.concatenate([order[:-1], [4]])
    shuffled = torch.empty(offset + (n + 1) * h * w, dtype=torch.int16, device="cuda")
    shuffled[offset:] = torch.from_numpy(raw[take].view(np.int16).reshape(-1)).cuda()
    torch.cuda.synchronize()
    _lib.call("gg_stack_calibrate_u16_device", s.handle, _lib.ptr(order), ctypes.c_int64(order.size),
              ctypes.c_void_p(shuffled.data_ptr() + 2 * offset), 0, ctypes.byref(params))
    for k in range(n):
        src = raw[4 if k == 3 else k]
        light = src.astype(np.float32)
        v = (light - dark * np.float32(1.5)) - bias
        v = v / np.maximum(flat, np.float32(1.0e-6)) + np.float32(0.25)
        np.testing.assert_array_equal(s.download_frame(k), v.astype(np.float32))
        assert s.frame_global_stats(k)["nonfinite_pixels"] == 1
    # one NaN per frame: the integrator must take the partly-valid formulas
    s.integrate_async(None, 2, 3.0, 3.0, 3, 0.5, count_map_dtype="float32")
    cov = s.download_maps("full")[2]
    assert cov[h // 2, w // 3] == 0.0
    s.close()


def test_frame_views_follow_warps_and_captured_warps(native):
    import torch

    rng = np.random.default_rng(2)
    n, h, w = 4, 48, 64
    frames = rng.normal(1000.0, 30.0, (n, h, w)).astype(np.float32)
    s = native.ResidentCalibratedStack(n, h, w)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    for k in range(n):
        s.upload_calibrated_frame(k, frames[k])

    def views_match():
        for k in range(n):
            np.testing.assert_array_equal(s.frame_tensor(k).cpu().numpy(), s.download_frame(k))

    views_match()
    views_match()  # from the kept table
    shift = np.tile(np.eye(3), (n, 1, 1))
    shift[:, 0, 2] = 1.0
    s.warp_frames_async(np.arange(n), shift, 1, 0.0)
    views_match()
    s.warp_frames_async([1, 3], shift[:2], 1, 0.0)
    views_match()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        s.warp_frames_async([2], shift[:1], 1, 0.0)
    for _ in range(3):  # replays move the frame behind the library's back
        graph.replay()
        torch.cuda.synchronize()
        views_match()
    expected = np.zeros_like(frames[2])
    expected[:, 4:] = frames[2][:, :-4]
    np.testing.assert_array_equal(s.download_frame(2)[:, 4:], expected[:, 4:])
    s.close()


@pytest.mark.parametrize("n", [3, 64, 65, 1025])
def test_frame_weights_with_priors(native, n):
    rng = np.random.default_rng(n)
    h, w = 9, 13
    frames = rng.normal(1000.0, 30.0, (n, h, w)).astype(np.float32)
    frames[n // 2, 2, 3] = np.nan
    frames[1] = 7.0
    prior = rng.uniform(0.5, 2.0, n).astype(np.float32)
    prior[2] = np.nan
    prior[0] = 0.0
    s = native.ResidentCalibratedStack(n, h, w)
    for k in range(n):
        s.upload_calibrated_frame(k, frames[k])
    for p in (None, prior):
        for _ in range(2):
            got = s.compute_frame_weights("simple_snr", p)
        v = frames.astype(np.float64).reshape(n, -1)
        mean, sd = np.nanmean(v, 1), np.nanstd(v, 1)
        want = np.where(sd <= np.float32(1e-6), 1e6, np.abs(mean) / np.maximum(sd, 1e-12))
        if p is not None:
            want = np.where(np.isfinite(p) & (p > 0), want * p, 0.0)
        np.testing.assert_allclose(got, want, rtol=1e-6)
        np.testing.assert_array_equal(s.compute_frame_weights("prior", p),
                                      np.where(np.isfinite(p) & (p > 0), p, 0) if p is not None else np.ones(n))
    s.close()
