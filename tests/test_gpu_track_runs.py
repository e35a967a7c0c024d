"""The tile search by warps over runs of several pairs (the next pair's block
in the other buffer, the template kept or changed inside a run, a last run
that is shorter), bit for bit against the same pairs searched one call each,
which a CTA each takes."""
import ctypes

import numpy as np
import pytest

from imagestackalignator_b200 import isa

pytestmark = pytest.mark.gpu
SZ = ctypes.c_size_t


@pytest.mark.parametrize("T,S", [(32, 1), (32, 2), (32, 4), (32, 5), (32, 6), (16, 2)])
def test_runs_equal_single_pairs(cuda, T, S):
    """28 pairs of 63 x 47 tiles: 82908 items, five to ten pairs a warp."""
    import torch
    n, tcx, tcy = 8, 63, 47
    W, H = tcx * T + 2 * S + 3, tcy * T + 2 * S + 1
    rng = np.random.default_rng(T * 10 + S)
    frames = [torch.from_numpy(rng.uniform(0, 1, (H, W)).astype(np.float32)).cuda() for _ in range(n)]
    ptrs = torch.tensor([f.data_ptr() for f in frames], device="cuda")
    pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    tab = (isa.IsaTrackPair * len(pairs))()
    for k, (a, b) in enumerate(pairs):
        tab[k].reference, tab[k].to_track, tab[k].grid = a, b, k
        if k % 5 in (2, 3):  # another template origin, some over the frame's edge, within a reference's pairs
            tab[k].base_shift_ref[:] = (float(k % 7) - 3.0, -2.0)
            tab[k].base_shift_trk[:] = (9.0, float(-b))
            tab[k].rotation_ref = 0.004 * a
            tab[k].rotation_trk = 0.01 * b
    raw = np.frombuffer(bytes(tab), np.uint8).reshape(len(pairs), -1)
    pre = rng.uniform(-6, 6, (len(pairs), tcy, tcx, 2)).astype(np.float32)
    pre[:, 0] -= 40.0
    pre[:, -1] += 40.0

    def search(ks):
        d = torch.from_numpy(raw[ks].copy()).cuda()
        g = torch.from_numpy(pre).cuda()
        sc = torch.zeros((len(ks), tcy, tcx, (2 * S + 1) ** 2), device="cuda")
        am = torch.zeros((len(ks), tcy, tcx), dtype=torch.int32, device="cuda")
        isa.check(isa.lib().isa_track_level(isa.vp(ptrs), SZ(W * 4), W, H, T, S, tcx, tcy, isa.vp(d), len(ks), isa.vp(g), SZ(tcx * 8),
                                            SZ(tcx * tcy * 8), ctypes.c_float(0.5), isa.vp(sc), isa.vp(am), isa.stream_ptr()))
        torch.cuda.synchronize()
        return g[ks], sc, am

    grids, scores, argmin = search(list(range(len(pairs))))
    for k in range(len(pairs)):
        g, s, a = search([k])
        assert torch.equal(s[0], scores[k]) and torch.equal(a[0], argmin[k]) and torch.equal(g[0], grids[k]), k


def test_shifts_beyond_the_integers(cuda):
    """Pre-shifts that no integer holds, by CTAs and by warps: replicated borders, as for any block far outside."""
    import torch
    T, S, n, tcx, tcy = 32, 2, 6, 40, 30
    W, H = tcx * T + 2 * S, tcy * T + 2 * S
    rng = np.random.default_rng(8)
    frames = [torch.from_numpy(rng.uniform(0, 1, (H, W)).astype(np.float32)).cuda() for _ in range(n)]
    ptrs = torch.tensor([f.data_ptr() for f in frames], device="cuda")
    pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    tab = (isa.IsaTrackPair * len(pairs))()
    for k, (a, b) in enumerate(pairs):
        tab[k].reference, tab[k].to_track, tab[k].grid = a, b, k
    raw = np.frombuffer(bytes(tab), np.uint8).reshape(len(pairs), -1)
    far = np.zeros((len(pairs), tcy, tcx, 2), np.float32)
    odd = (3e9, -3e9, 2147483520.0, -2147483648.0, 1e30, -1e30, np.inf, -np.inf, np.nan)
    near = far.copy()
    for k in range(len(pairs)):
        for i, v in enumerate(odd):
            far[k, i, (k + i) % 3, i % 2] = v
            near[k, i, (k + i) % 3, i % 2] = 0.0 if np.isnan(v) else np.clip(v, -1e6, 1e6)

    def search(ks, pre):
        d = torch.from_numpy(raw[ks].copy()).cuda()
        g = torch.from_numpy(pre).cuda()
        am = torch.zeros((len(ks), tcy, tcx), dtype=torch.int32, device="cuda")
        isa.check(isa.lib().isa_track_level(isa.vp(ptrs), SZ(W * 4), W, H, T, S, tcx, tcy, isa.vp(d), len(ks), isa.vp(g), SZ(tcx * 8),
                                            SZ(tcx * tcy * 8), ctypes.c_float(0.5), None, isa.vp(am), isa.stream_ptr()))
        torch.cuda.synchronize()
        return am

    every = list(range(len(pairs)))
    assert len(pairs) * tcx * tcy >= 8000  # by warps
    want = search(every, near)
    assert torch.equal(search(every, far), want)
    for k in every:
        assert torch.equal(search([k], far)[0], want[k]), k
