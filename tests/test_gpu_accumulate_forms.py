"""The accumulation's specialised kernels against its general one over the forms
both accept: the same call with 4-channel kernel parameters (specialised at
scales 1 and 2) and with 3-channel ones (always the general, tap-by-tap kernel).

Tolerance: a frame adds at most 25 products per channel in a chain of FP32
multiply-adds, folds and a final scaling, under 32 roundings of 2^-24 relative
to the sum of the products' magnitudes; the two sides together stay below
64 * 2^-24 = 4e-6 of the weight sum (samples are at most 1.05 of white)."""
import ctypes

import numpy as np
import pytest

from imagestackalignator_b200 import isa

pytestmark = pytest.mark.gpu

SZ = ctypes.c_size_t


def accumulate(raw, cfa, kp, flow, mask, scale, ox, oy, crop, Wo, Ho, start):
    import torch
    H, W = raw.shape
    acc, wsum = start.clone(), start.clone()
    isa.check(isa.lib().isa_accumulate(isa.vp(raw), SZ(W * 2), W, H, (ctypes.c_int * 4)(*cfa), isa.vp(acc), isa.vp(wsum), SZ(Wo * 12), Wo, Ho,
                                       isa.vp(mask), SZ(W // 2 * 16), isa.vp(kp), SZ(W * 4 * kp.shape[2]), kp.shape[2], isa.vp(flow), SZ(W * 8),
                                       (ctypes.c_float * 3)(15871.0, 15871.0, 15800.0), (ctypes.c_float * 3)(512.0, 500.0, 512.0),
                                       ctypes.c_float(scale), ox, oy, (ctypes.c_int * 4)(*crop), isa.stream_ptr()))
    torch.cuda.synchronize()
    return acc, wsum


# W, H, scale, ox, oy, crop (None: the frame), Wo, Ho (0: the whole scaled frame), CFA, flow amplitude (None: no flow), mask
CASES = [
    (130, 66, 2.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 3.0, "rand"),
    (130, 66, 2.0, 0, 0, None, 257, 129, (2, 1, 1, 0), 40.0, "rand"),        # every pixel near or over a border
    (64, 34, 2.0, 32, 17, (16, 8, 47, 24), 64, 34, (1, 0, 2, 1), 2.0, "rand"),  # central crop, odd origin
    (64, 34, 2.0, 33, 18, (17, 9, 46, 25), 61, 31, (1, 2, 0, 1), 2.0, "rand"),  # odd crop and origin
    (64, 34, 2.0, -3, 5, None, 127, 64, (0, 1, 1, 2), 1.0, "rand"),          # negative origin
    (520, 20, 2.0, 1, 2, None, 1037, 35, (0, 1, 1, 2), 2.0, "nonfinite"),
    (64, 64, 2.0, 0, 0, None, 0, 0, (0, 1, 1, 2), None, None),
    (64, 64, 2.0, 0, 0, None, 0, 0, (1, 0, 2, 1), 2.0, None),
    (64, 64, 2.0, 0, 0, (30, 30, 31, 31), 0, 0, (0, 1, 1, 2), 2.0, "rand"),  # a crop smaller than a 3 x 3 block
    (16, 16, 2.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 1.0, "zero"),
    (4, 4, 2.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 0.5, "rand"),
    (2, 2, 2.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 0.5, "rand"),
    (130, 66, 1.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 3.0, "rand"),
    (258, 34, 1.0, 0, 0, None, 257, 33, (2, 1, 1, 0), 40.0, "rand"),
    (64, 34, 1.0, 7, 5, (9, 6, 50, 30), 50, 27, (1, 0, 2, 1), 2.0, "rand"),    # odd origin and crop
    (64, 34, 1.0, -3, -2, None, 70, 40, (1, 2, 0, 1), 1.0, "nonfinite"),       # output beyond the frame
    (64, 64, 1.0, 0, 0, None, 0, 0, (0, 1, 1, 2), None, None),
    (64, 64, 1.0, 0, 0, None, 0, 0, (1, 2, 0, 1), 2.0, None),
    (64, 64, 1.0, 0, 0, (30, 30, 33, 33), 0, 0, (0, 1, 1, 2), 2.0, "rand"),    # a crop smaller than a 5 x 5 block
    (16, 16, 1.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 1.0, "zero"),
    (4, 4, 1.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 0.5, "rand"),
    (2, 2, 1.0, 0, 0, None, 0, 0, (0, 1, 1, 2), 0.5, "rand"),
]


@pytest.mark.parametrize("kernels", ["ordinary", "extreme"])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_specialised_equals_general(cuda, case, kernels):
    import torch
    W, H, scale, ox, oy, crop, Wo, Ho, cfa, amp, mk = CASES[case]
    rng = np.random.default_rng(100 + case)
    Wo, Ho, crop = Wo or int(W * scale), Ho or int(H * scale), crop or (0, 0, W - 1, H - 1)
    raw = torch.from_numpy(rng.integers(0, 16384, (H, W)).astype(np.int16)).cuda()
    th = rng.uniform(0, np.pi, (H, W))
    k1, k2 = rng.uniform(0.05, 0.8, (H, W)) ** 2, rng.uniform(0.05, 0.8, (H, W)) ** 2
    c, s = np.cos(th), np.sin(th)
    b11, b12, b22 = k1 * c * c + k2 * s * s, (k1 - k2) * c * s, k1 * s * s + k2 * c * c
    det = b11 * b22 - b12 * b12
    kp = np.stack([b22 / det, b11 / det, -b12 / det, 0 * det], -1).astype(np.float32)
    if kernels == "extreme":
        kp[::5, ::3, :3] = np.inf      # weights fall back to the cross
        kp[::7, ::4, 0] = np.nan
        kp[1::6, 1::5, :3] = (-30.0, -30.0, 0.0)  # weights up to e^120: sums beyond FP32 in either kernel
    flow = None
    if amp is not None:  # steps of 1 / 64 px: the flow sample and its rounding are exact on both sides at whole scales
        flow = torch.from_numpy((np.round(rng.uniform(-amp, amp, (H, W, 2)) * 64) / 64).astype(np.float32)).cuda()
    mask = None
    if mk is not None:
        m = rng.uniform(0, 1, (H // 2, W // 2, 4)).astype(np.float32)
        m[rng.uniform(size=m.shape) < 0.2] = 0.0
        if mk == "zero":
            m[:] = 0
        if mk == "nonfinite":
            m[rng.uniform(size=m.shape) < 0.1] = np.nan
            m[rng.uniform(size=m.shape) < 0.1] = np.inf
        mask = torch.from_numpy(m).cuda()
    start = torch.from_numpy(rng.uniform(0, 1, (Ho, Wo, 3)).astype(np.float32)).cuda()
    args = (flow, mask, scale, ox, oy, crop, Wo, Ho, start)
    a4, w4 = accumulate(raw, cfa, torch.from_numpy(kp).cuda(), *args)
    a3, w3 = accumulate(raw, cfa, torch.from_numpy(np.ascontiguousarray(kp[..., :3])).cuda(), *args)
    a4, w4, a3, w3 = (t.cpu().numpy().astype(np.float64) for t in (a4, w4, a3, w3))
    finite = np.isfinite(a3) & np.isfinite(w3) & (np.abs(w3) < 1e30) & (np.abs(a3) < 1e30)
    if kernels == "ordinary":
        assert finite.all()
    # beyond 1e30 both sides are on the tap-by-tap form, but may overflow at different taps
    tol = 4e-6 * (np.abs(w3) + 1.0)
    assert (np.abs(w4 - w3)[finite] <= tol[finite]).all(), np.max(np.abs(w4 - w3)[finite] / tol[finite])
    assert (np.abs(a4 - a3)[finite] <= tol[finite]).all(), np.max(np.abs(a4 - a3)[finite] / tol[finite])
