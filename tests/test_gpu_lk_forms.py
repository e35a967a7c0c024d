"""The Lucas-Kanade iteration at the edges of its strips: widths around a
strip's, heights around a step's, odd row pitches, the smallest and largest
windows, against the oracle's separate steps in 64 bits."""
import ctypes

import numpy as np
import pytest

from imagestackalignator_b200 import isa

pytestmark = pytest.mark.gpu
SZ = ctypes.c_size_t


@pytest.mark.parametrize("W,H,window,pad", [(50, 40, 11, 0), (51, 41, 11, 1), (49, 27, 11, 2), (101, 64, 11, 1), (157, 33, 11, 0), (61, 70, 31, 1),
                                            (90, 65, 31, 0), (113, 50, 3, 0), (58, 37, 5, 3)])
def test_iteration_strip_edges(cuda, oracle, W, H, window, pad):
    """White-noise frames: window matrices of condition below 30 from 11 x 11 on, so FP32 derivatives (relative error
    5e-7) keep the update to 1e-4; in smaller windows only the bulk of the pixels is that well conditioned."""
    import torch
    rng = np.random.default_rng(W * 100 + H)
    ref = rng.uniform(0, 1, (H, W)).astype(np.float32)
    src = rng.uniform(0, 1, (H, W)).astype(np.float32)
    flow0 = rng.uniform(-4, 4, (H, W, 2)).astype(np.float32)
    flow0[:3, :3] = [-30.5, -20.25]   # samples far outside the frame

    def pitched(a):
        t = torch.zeros((H, W + pad) + a.shape[2:], device="cuda")
        t[:, :W] = torch.from_numpy(a).cuda()
        return t

    f, s, r, o = pitched(flow0), pitched(src), pitched(ref), torch.zeros((H, W + pad, 2), device="cuda")
    isa.check(isa.lib().isa_lk_iteration(isa.vp(f), isa.vp(o), SZ((W + pad) * 8), isa.vp(s), isa.vp(r), SZ((W + pad) * 4), W, H,
                                         ctypes.c_float(0.01), window, isa.stream_ptr()))
    got = o.cpu().numpy()
    assert not got[:, W:].any()
    got = got[:, :W]
    warped = oracle.warp(src.astype(np.float64), flow0.astype(np.float64))
    ix, iy, it = oracle.derivatives(warped, ref.astype(np.float64))
    want = oracle.lucas_kanade(flow0.astype(np.float64), ix, iy, it, window // 2, float(np.float32(0.01)))
    err = np.abs(got - want).max(axis=2)
    assert np.percentile(err, 98) < 1e-4
    if window >= 11:
        assert err.max() < 2e-4
