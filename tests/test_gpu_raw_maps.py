"""The chunk maps of the PEF and DNG decoders where candidate starts never
meet (every symbol equally long: the lists of places run over a warp's 32
lanes) and chunk counts that are no multiple of a warp's eight, bit-exact."""
import numpy as np
import pytest

from imagestackalignator_b200 import isa, synthetic

import raw as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cat", [1, 4, 8, 13])
@pytest.mark.parametrize("shape", [(40, 66), (101, 130), (77, 514)])
def test_equal_symbols(cuda, shape, cat):
    """Differences of one category along the rows: +a, -a, +a, ..."""
    import torch
    H, W = shape
    img = np.broadcast_to(1000 + (1 << (cat - 1)) * ((np.arange(W) // 2) % 2), shape).astype(np.uint16)
    book = R.canonical_book()
    table = R.huff_table(R.maker_note_bytes(*book))
    s = torch.from_numpy(np.ascontiguousarray(R.encode(img, *book))).cuda()
    got = isa.pef_decode(s, table, W, H).cpu().numpy().view(np.uint16)
    assert np.array_equal(got, img)
    f, offs, cnts = synthetic.dng_tiled_file(img, 64, 64)
    got = isa.dng_decode(f, W, H, offs, cnts, tiled=True, tile_w=64, tile_h=64).cpu().numpy().view(np.uint16)
    assert np.array_equal(got, img)
