"""Black and white levels in the accumulation and its gradient.

Black comes off every sample before any rounding, so a constant added to the
samples and to black changes nothing, bit for bit, however dark the frame;
and sums overflow only where those of normalised samples would. Against the
oracle in 64 bits over the forms of test_gpu_accumulate_forms.py."""
import ctypes

import numpy as np
import pytest

from imagestackalignator_b200 import isa, params as P
from test_gpu_accumulate_forms import CASES

pytestmark = pytest.mark.gpu

SZ = ctypes.c_size_t


def accumulate(raw, cfa, kp, flow, mask, scale, ox, oy, crop, Wo, Ho, white, black):
    import torch
    H, W = raw.shape
    acc, wsum = torch.zeros((Ho, Wo, 3), device="cuda"), torch.zeros((Ho, Wo, 3), device="cuda")
    raw = torch.from_numpy(np.ascontiguousarray(raw).view(np.int16)).cuda()
    kp, flow, mask = (None if a is None else torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda() for a in (kp, flow, mask))
    isa.check(isa.lib().isa_accumulate(isa.vp(raw), SZ(W * 2), W, H, (ctypes.c_int * 4)(*cfa), isa.vp(acc), isa.vp(wsum), SZ(Wo * 12), Wo, Ho,
                                       isa.vp(mask), SZ(W // 2 * 16), isa.vp(kp), SZ(W * 4 * kp.shape[2]), kp.shape[2], isa.vp(flow), SZ(W * 8),
                                       (ctypes.c_float * 3)(*white), (ctypes.c_float * 3)(*black), ctypes.c_float(scale), ox, oy,
                                       (ctypes.c_int * 4)(*crop), isa.stream_ptr()))
    return acc.cpu().numpy(), wsum.cpu().numpy()


def kernels(rng, H, W, lo, hi):
    th = rng.uniform(0, np.pi, (H, W))
    k1, k2 = rng.uniform(lo, hi, (H, W)) ** 2, rng.uniform(lo, hi, (H, W)) ** 2
    c, s = np.cos(th), np.sin(th)
    b11, b12, b22 = k1 * c * c + k2 * s * s, (k1 - k2) * c * s, k1 * s * s + k2 * c * c
    det = b11 * b22 - b12 * b12
    return np.stack([b22 / det, b11 / det, -b12 / det, 0 * det], -1).astype(np.float32)


def inputs(case, scale=None):
    W, H, s, ox, oy, crop, Wo, Ho, cfa, amp, mk = CASES[case]
    rng = np.random.default_rng(300 + case)
    if scale is not None:
        s, Wo, Ho = scale, 0, 0
    Wo, Ho, crop = Wo or int(W * s), Ho or int(H * s), crop or (0, 0, W - 1, H - 1)
    flow = None if amp is None else (np.round(rng.uniform(-amp, amp, (H, W, 2)) * 64) / 64).astype(np.float32)
    mask = None
    if mk is not None:
        mask = rng.uniform(0, 1, (H // 2, W // 2, 4)).astype(np.float32)
        mask[rng.uniform(size=mask.shape) < 0.2] = 0.0
        if mk == "zero":
            mask[:] = 0
        if mk == "nonfinite":
            mask[rng.uniform(size=mask.shape) < 0.1] = np.nan
    return rng, W, H, cfa, (flow, mask, s, ox, oy, crop, Wo, Ho)


SCALE1 = [k for k, c in enumerate(CASES) if c[2] == 1.0]


@pytest.mark.parametrize("black", [(0.0, 0.0, 0.0), (3.0, 0.0, 7.0)])
@pytest.mark.parametrize("case,scale,kc", [(k, None, 4) for k in SCALE1] + [(12, None, 3), (14, None, 3), (14, 0.5, 4), (15, 1.5, 4), (13, 3.0, 3), (0, 2.0, 3)])
def test_levels_shift_exactly(cuda, case, scale, kc, black):
    """Samples of 1 .. 20 over black, both raised by 49152."""
    rng, W, H, cfa, args = inputs(case, scale)
    raw = rng.integers(1, 21, (H, W)).astype(np.uint16)
    kp = np.ascontiguousarray(kernels(rng, H, W, 0.05, 0.8)[..., :kc])
    white = (15871.0, 15871.0, 15800.0)
    a0, w0 = accumulate(raw, cfa, kp, *args, white, black)
    a1, w1 = accumulate(raw + np.uint16(49152), cfa, kp, *args, white, tuple(b + 49152.0 for b in black))
    assert np.array_equal(w0, w1) and np.array_equal(a0, a1)
    assert np.isfinite(a0).all()


@pytest.mark.parametrize("kc", [3, 4])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_forms_against_64_bits(cuda, oracle, case, kc):
    """Kernels of condition below 2.3: a tap's exponent x = q / 2 is off by at most 4.5 x times six roundings, its weight by
    4.5 x e^-x 3.6e-7 <= 6e-7, so 25 taps add 1.5e-5; the sums' own roundings are below 4e-6 of the weight sum
    (test_gpu_accumulate_forms.py)."""
    rng, W, H, cfa, args = inputs(case)
    flow, mask, s, ox, oy, crop, Wo, Ho = args
    raw = rng.integers(0, 16384, (H, W)).astype(np.uint16)
    kp = np.ascontiguousarray(kernels(rng, H, W, 0.6, 0.9)[..., :kc])
    white, black = (15871.0, 15871.0, 15800.0), (512.0, 500.0, 512.0)
    ga, gw = accumulate(raw, cfa, kp, *args, white, black)
    want_a, want_w = np.zeros((Ho, Wo, 3)), np.zeros((Ho, Wo, 3))
    oracle.accumulate(raw, cfa, want_a, want_w, (np.ones((H // 2, W // 2, 4)) if mask is None else mask).astype(np.float64),
                      kp[..., :3].astype(np.float64), (np.zeros((H, W, 2)) if flow is None else flow).astype(np.float64), white, black, s, (ox, oy), crop)
    tol = 1.5e-5 + 4e-6 * (want_w + 1.0)
    assert (np.abs(gw - want_w) <= tol).all(), np.max(np.abs(gw - want_w) / tol)
    assert (np.abs(ga - want_a) <= tol).all(), np.max(np.abs(ga - want_a) / tol)


@pytest.mark.parametrize("scale,kc", [(1.0, 4), (1.0, 3), (1.5, 4), (3.0, 3)])
def test_large_weights_stay_finite(cuda, scale, kc):
    """Weights up to e^(20.7 / 2 * 8) = 9e35: a frame's sums reach 4e36 normalised, and 16383 times that in raw units
    would be beyond FP32."""
    rng = np.random.default_rng(9)
    W, H = 64, 48
    raw = rng.integers(0, 16384, (H, W)).astype(np.uint16)
    kp = np.zeros((H, W, 4), np.float32)
    kp[..., :2] = -20.7
    Wo, Ho = int(W * scale), int(H * scale)
    a, w = accumulate(raw, (0, 1, 1, 2), np.ascontiguousarray(kp[..., :kc]), None, None, scale, 0, 0, (0, 0, W - 1, H - 1), Wo, Ho, (15871.0,) * 3,
                      (512.0,) * 3)
    assert np.isfinite(a).all() and np.isfinite(w).all() and w.max() > 1e35
    a, w = a[1:-1, 1:-1].astype(np.float64), w[1:-1, 1:-1].astype(np.float64)
    assert (w > 0).all() and (a / w).max() <= 1.0 + 1e-5 and (a / w).min() >= -512.0 / 15871.0 - 1e-5


@pytest.mark.parametrize("scale,over", [(1.5, (0, 0, 0)), (3.0, (0, 0, 0)), (1.5, (1, 0, 2))])
def test_gradient_keeps_the_last_digits_of_dark_frames(cuda, scale, over):
    """Equal frames of 1 .. 20 over black: no motion, full certainty, so raising the samples and black by 49152 changes
    nothing the gradient depends on. The two gradients differ by the order of the FP32 atomic sums alone: a term per
    weighted pixel and tap, 200 in all, so 200 * 2^-24 = 1.2e-5 of the terms' magnitudes; a few pixels are weighted, so that
    rounding errors do not average out."""
    import torch
    W, H, n = 336, 336, 3
    rng = np.random.default_rng(4)
    img = (10.0 + 6.0 * np.sin(np.arange(W)[None, :] / 9.0) * np.cos(np.arange(H)[:, None] / 7.0) + rng.uniform(-3, 3, (H, W))).round()
    frame = np.clip(img, 1, 20).astype(np.uint16)
    p = P.MergeParams(merge_scale=scale)
    outs, grads, losses = [], [], []
    for lift in (0, 49152):
        info = isa.IsaRawInfo()
        info.width, info.height = W, H
        info.cfa[:] = (0, 1, 1, 2)
        info.black[:] = tuple(float(lift + o) for o in over)
        info.white[:] = (15871.0,) * 3
        info.camera_white[:] = (1.0,) * 3
        info.noise_alpha, info.noise_beta = 1e-3, 8e-6
        raw = torch.from_numpy(np.repeat((frame + np.uint16(lift))[None], n, 0).view(np.int16)).cuda()
        m = isa.Merger(W, H, n, p)
        out = m.merge(raw, info).clone()
        if not outs:
            target = (out * 0.5).contiguous()
            om = torch.zeros(out.shape[:2], device="cuda")
            om[150:152, 200:204] = 1.0
        _, loss, grad = m.backward(raw, info, target, weight=om)
        outs.append(out.cpu().numpy())
        grads.append(grad[:6])
        losses.append(loss)
        m.close()
    assert np.array_equal(outs[0], outs[1]) and losses[0] == losses[1]
    assert np.abs(grads[0]).max() > 0
    assert np.allclose(grads[0], grads[1], rtol=1e-4, atol=1.2e-5 * np.abs(grads[0]).max()), (grads[0], grads[1])
