"""The chunk maps of the PEF and DNG decoders over the chunks that a warp takes
(one to eight, by the number of chunks), remainders included, bit-exact."""
import numpy as np
import pytest

from imagestackalignator_b200 import isa, synthetic

import raw as R

pytestmark = pytest.mark.gpu

BOOK = R.canonical_book()
TABLE = R.huff_table(R.maker_note_bytes(*BOOK))


def frame(W, H, seed):
    """Smooth shading, a step every 300 columns and noise of 13 to 14 difference bits now and then."""
    rng = np.random.default_rng(seed)
    img = 5000.0 + 2000.0 * np.sin(np.arange(W) / 37.0)[None, :] + 1500.0 * ((np.arange(W) // 300) % 2)[None, :] + rng.normal(0, 120, (H, W))
    img[rng.uniform(size=(H, W)) < 0.01] = 16000
    return np.clip(img, 0, 16383).astype(np.uint16)


@pytest.mark.parametrize("W,H", [(336, 336), (800, 640), (1000, 700), (1262, 958), (1402, 1000), (1800, 1200), (2000, 1500), (2504, 1806)])
def test_groups(cuda, W, H):
    import torch
    img = frame(W, H, W)
    s = torch.from_numpy(np.ascontiguousarray(R.encode(img, *BOOK))).cuda()
    assert np.array_equal(isa.pef_decode(s, TABLE, W, H).cpu().numpy().view(np.uint16), img)
    f, offs, cnts = synthetic.dng_tiled_file(img, 256, 256)
    got = isa.dng_decode(f, W, H, offs, cnts, tiled=True, tile_w=256, tile_h=256).cpu().numpy().view(np.uint16)
    assert np.array_equal(got, img)


@pytest.mark.parametrize("cat", [4, 13])
def test_groups_without_common_places(cuda, cat):
    """Every symbol equally long: no two candidate starts meet, so a full warp lists 8 x 32 places."""
    import torch
    H, W = 1500, 2500
    img = np.broadcast_to(1000 + (1 << (cat - 1)) * ((np.arange(W) // 2) % 2), (H, W)).astype(np.uint16)
    s = torch.from_numpy(np.ascontiguousarray(R.encode(img, *BOOK))).cuda()
    assert np.array_equal(isa.pef_decode(s, TABLE, W, H).cpu().numpy().view(np.uint16), img)
