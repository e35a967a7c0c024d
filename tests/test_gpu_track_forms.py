"""The tile search's two kernels (a CTA, or in large searches a warp, per pair
and tile) against each other: one large call must give, bit for bit, the maps,
minima and pre-shifts of the same pairs searched one call each."""
import ctypes

import numpy as np
import pytest

from imagestackalignator_b200 import isa

pytestmark = pytest.mark.gpu
SZ = ctypes.c_size_t


@pytest.mark.parametrize("T,S,W,H,n", [(32, 2, 1034, 774, 5), (32, 4, 650, 710, 5), (32, 1, 1000, 800, 5), (32, 3, 1030, 774, 5), (32, 5, 717, 651, 5),
                                       (32, 6, 655, 655, 5), (16, 2, 1015, 790, 5), (16, 1, 1010, 790, 5)])
def test_large_search_equals_single_pairs(cuda, T, S, W, H, n):
    import torch
    rng = np.random.default_rng(T * 10 + S)
    frames = [torch.from_numpy(rng.uniform(0, 1, (H, W)).astype(np.float32)).cuda() for _ in range(n)]
    ptrs = torch.tensor([f.data_ptr() for f in frames], device="cuda")
    tcx, tcy = (W - 2 * S) // T, (H - 2 * S) // T
    pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    tab = (isa.IsaTrackPair * len(pairs))()
    for k, (a, b) in enumerate(pairs):
        tab[k].reference, tab[k].to_track, tab[k].grid = a, b, k
        if k % 3 == 1:   # pre-alignment: template and block move, some over the frame's edge
            tab[k].base_shift_ref[:] = (float(a), -1.0)
            tab[k].base_shift_trk[:] = (9.0, float(-b))
            tab[k].rotation_trk = 0.01 * b
    raw = np.frombuffer(bytes(tab), np.uint8).reshape(len(pairs), -1)
    pre = rng.uniform(-6, 6, (len(pairs), tcy, tcx, 2)).astype(np.float32)
    pre[:, 0] -= 40.0    # blocks beyond the top edge

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
