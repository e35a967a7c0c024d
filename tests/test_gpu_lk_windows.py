"""The fused Lucas-Kanade iteration at every kind of window, against the
separate steps (isa_warp, isa_derivatives, isa_lucas_kanade), whose solve is
the plain division.

Images in multiples of 24 and whole-numbered flow make warps, derivatives,
their products and all window sums whole numbers, exact on both sides. So the
two sides solve the same 2 x 2 systems and may differ by the reciprocal
alone: rounded to FP32 by one last place, 2^-23 relative."""
import ctypes

import numpy as np
import pytest

from imagestackalignator_b200 import isa

pytestmark = pytest.mark.gpu
SZ = ctypes.c_size_t


def fused(flow, src, ref, min_det, window):
    import torch
    H, W = ref.shape
    out = torch.empty_like(flow)
    isa.check(isa.lib().isa_lk_iteration(isa.vp(flow), isa.vp(out), SZ(W * 8), isa.vp(src), isa.vp(ref), SZ(W * 4), W, H, ctypes.c_float(min_det),
                                         window, isa.stream_ptr()))
    return out


def steps(flow, src, ref, min_det, window):
    import torch
    H, W = ref.shape
    warped, ix, iy, it = (torch.empty((H, W), device="cuda") for _ in range(4))
    out = flow.clone()
    lib = isa.lib()
    isa.check(lib.isa_warp(isa.vp(src), SZ(W * 4), W, H, isa.vp(flow), SZ(W * 8), isa.vp(warped), SZ(W * 4), isa.stream_ptr()))
    isa.check(lib.isa_derivatives(isa.vp(warped), isa.vp(ref), SZ(W * 4), W, H, isa.vp(ix), isa.vp(iy), isa.vp(it), SZ(W * 4), isa.stream_ptr()))
    isa.check(lib.isa_lucas_kanade(isa.vp(out), SZ(W * 8), isa.vp(ix), isa.vp(iy), isa.vp(it), SZ(W * 4), W, H, ctypes.c_float(min_det), window,
                                   isa.stream_ptr()))
    return out, ix, iy


@pytest.mark.parametrize("window", [1, 2, 3, 5, 8, 11, 15, 17, 19, 20, 21, 27, 31])
@pytest.mark.parametrize("W,H,motion", [(131, 74, 0), (262, 150, 2), (70, 260, 1)])
def test_solve_equals_division(cuda, W, H, motion, window):
    import torch
    rng = np.random.default_rng(W + window)
    ref, src = 24.0 * rng.integers(0, 16, (H, W)), 24.0 * rng.integers(0, 16, (H, W))
    for a in (ref, src):
        a[10:60, 8:50] = 24.0 * 3                                    # flat: all sums zero
        a[:, 60:110] = a[:1, 60:110] if motion == 0 else a[:, 60:110]  # columns alike: rank one
    flow = torch.from_numpy(rng.integers(-motion, motion + 1, (H, W, 2)).astype(np.float32)).cuda()
    src, ref = torch.from_numpy(src.astype(np.float32)).cuda(), torch.from_numpy(ref.astype(np.float32)).cuda()
    _, ix, iy = steps(flow, src, ref, 0.01, window)
    ix, iy = ix.cpu().numpy().astype(np.float64), iy.cpu().numpy().astype(np.float64)
    assert np.array_equal(ix, np.round(ix)) and np.array_equal(iy, np.round(iy))
    # thresholds: the usual one, and the largest eigenvalue of one pixel's window, which half of the pixels stay below
    h = window // 2
    y, x = H // 2, W - h - 3
    gx, gy = ix[y - h:y + h + 1, x - h:x + h + 1], iy[y - h:y + h + 1, x - h:x + h + 1]
    a, b, d = (gx * gx).sum(), (gx * gy).sum(), (gy * gy).sum()
    level = 0.5 * (a + d) + np.sqrt(0.25 * (a - d) ** 2 + b * b)
    for min_det in (0.01, float(np.float32(level))):
        got, want = fused(flow, src, ref, min_det, window).cpu().numpy(), steps(flow, src, ref, min_det, window)[0].cpu().numpy()
        assert np.isfinite(want).all()
        near = np.abs(got - want) <= 2.0 ** -23 * np.abs(want) + 1e-12
        assert near.all(), (min_det, np.argwhere(~near)[:5], got[~near][:5], want[~near][:5])


def test_window_cost(cuda):
    """Window 21 on a large frame takes no more than 1.8 times the default window (measured: 1.6); strips too narrow for it
    took 1.9 times."""
    import torch
    W, H = 4000, 3000
    rng = np.random.default_rng(3)
    base = torch.from_numpy(rng.uniform(0, 1, (1, 1, H // 8, W // 8)).astype(np.float32)).cuda()
    img = torch.nn.functional.interpolate(base, size=(H, W), mode="bicubic")[0, 0].contiguous()
    src = torch.roll(img, (1, 2), (0, 1)).contiguous()
    flow = torch.full((H, W, 2), 0.5, device="cuda")

    def time(window):
        fused(flow, src, img, 0.01, window)
        best = float("inf")
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(4):
                fused(flow, src, img, 0.01, window)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert time(21) <= 1.8 * time(11)
