"""Workloads that the framework's speed is measured on.

Each case is one thing that a user of the library has it do, at a size and
with the options it is used with: whole merges of a burst (a preview, a full
sensor at 2x), a batch of small bursts, one step of a parameter fit (merge and
gradient), the single operators that a host calls one by one (tracking image,
tile search, Lucas-Kanade refinement, accumulation), and the ends of the raw
flow (PEF and DNG decoding, 16-bit output). Inputs are synthetic bursts made
on the GPU from the seed: a scene with edges and texture, moved by a shift
and a small rotation per frame, mosaicked, with Poisson-Gaussian noise,
14-bit over a black level of 512.

listed() gives the fixed cases, draw() more of the same ranges, prepare() the
inputs and handles a program holds before the call, run() one pass through
the public entry points, work() the bytes and operations a pass cannot do
without, exact() the outputs in 64 bits where they are computed numbers of a
single operator.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from imagestackalignator_b200 import isa, params as P

BLACK, WHITE = 512.0, 16383.0
NOISE_A, NOISE_B = 1e-3, 8e-6
CFA = {"RGGB": (0, 1, 1, 2), "BGGR": (2, 1, 1, 0), "GRBG": (1, 0, 2, 1), "GBRG": (1, 2, 0, 1)}


def listed():
    return [
        # the quickest whole call: a preview of a short burst, the reference's plain mode (1x); launches and latency count
        {"name": "merge_preview", "kind": "merge", "n": 5, "w": 640, "h": 480, "scale": 0.0, "cfa": "RGGB"},
        # the headline workload: 20 frames of a 24 MP sensor merged at 2x
        {"name": "merge_24mp_2x", "kind": "merge", "n": 20, "w": 6016, "h": 4000, "scale": 2.0, "cfa": "RGGB"},
        # a server's queue: small bursts merged side by side, one context and stream each
        {"name": "batch_small", "kind": "batch", "bursts": 6, "contexts": 3, "n": 6, "w": 1024, "h": 768, "scale": 2.0, "cfa": "GRBG"},
        # one step of a parameter fit: merge at 1.5x and the gradient of the eight parameters
        {"name": "fit_step_1p5x", "kind": "fit", "n": 6, "w": 2000, "h": 1500, "scale": 1.5, "cfa": "RGGB"},
        # the tracking image of one full-sensor frame: demosaic, gamma, high-pass, Gauss
        {"name": "tracking_24mp", "kind": "tracking", "w": 6016, "h": 4000, "cfa": "RGGB"},
        # the finest level of the tile search, all pairs of an 8-frame burst
        {"name": "tiles_8x3mp", "kind": "tiles", "n": 8, "w": 2048, "h": 1536, "tile": 32, "shift": 2},
        # Lucas-Kanade refinement of one 12 MP frame, three iterations
        {"name": "lk_12mp", "kind": "lk", "w": 4000, "h": 3000, "iterations": 3},
        # the accumulation frame by frame, as a host's own loop calls it: 1x of a ragged size, and 2x
        {"name": "accumulate_1x", "kind": "accumulate", "n": 4, "w": 3010, "h": 2006, "scale": 1.0, "cfa": "BGGR"},
        {"name": "accumulate_2x", "kind": "accumulate", "n": 4, "w": 2048, "h": 1536, "scale": 2.0, "cfa": "RGGB"},
        # raw frames in: a compressed PEF strip, a DNG of 256 x 256 lossless-JPEG tiles
        {"name": "pef_12mp", "kind": "pef", "w": 4000, "h": 3000},
        {"name": "dng_6mp", "kind": "dng", "w": 3000, "h": 2000},
        # the 2x image out: colour, tone curve and gamma to 16-bit RGB
        {"name": "post_24mp_2x", "kind": "post", "w": 12032, "h": 8000},
    ]


def _even(v):
    return int(v) // 2 * 2


def _size(rng, lo_mp, hi_mp):
    """An even frame size of lo_mp..hi_mp megapixels (log-uniform), aspect 1:1 to 16:9, either way up, often ragged."""
    mp = math.exp(rng.uniform(math.log(lo_mp), math.log(hi_mp))) * 1e6
    a = rng.uniform(1.0, 1.78)
    w, h = math.sqrt(mp * a), math.sqrt(mp / a)
    if rng.random() < 0.2:
        w, h = h, w
    step = rng.choice((2, 8, 16))
    return max(336, int(w) // step * step), max(336, _even(h))


def draw(rng):
    kind = rng.choice(("merge", "merge", "merge", "batch", "fit", "tracking", "tiles", "lk", "accumulate", "accumulate", "pef", "dng", "post"))
    cfa = rng.choice(sorted(CFA))
    if kind == "merge":
        w, h = _size(rng, 0.3, 12.0)
        n = rng.randint(3, 16)
        n = max(3, min(n, int(100e6 / (w * h))))
        return {"kind": kind, "n": n, "w": w, "h": h, "scale": rng.choice((0.0, 2.0, 2.0, 1.5)), "cfa": cfa}
    if kind == "batch":
        w, h = _size(rng, 0.3, 1.5)
        return {"kind": kind, "bursts": rng.randint(3, 8), "contexts": rng.randint(2, 4), "n": rng.randint(3, 8), "w": w, "h": h,
                "scale": rng.choice((0.0, 2.0)), "cfa": cfa}
    if kind == "fit":
        w, h = _size(rng, 0.5, 4.0)
        return {"kind": kind, "n": rng.randint(3, 8), "w": w, "h": h, "scale": rng.choice((1.0, 1.5, 2.0)), "cfa": cfa}
    if kind == "tracking":
        w, h = _size(rng, 0.3, 24.0)
        return {"kind": kind, "w": w, "h": h, "cfa": cfa}
    if kind == "tiles":
        w, h = _size(rng, 0.3, 6.0)
        tile, shift = rng.choice(((32, 2), (32, 2), (32, 4), (16, 2), (16, 4)))
        return {"kind": kind, "n": rng.randint(3, 10), "w": w, "h": h, "tile": tile, "shift": shift}
    if kind == "lk":
        w, h = _size(rng, 0.3, 24.0)
        return {"kind": kind, "w": w - rng.randint(0, 1), "h": h - rng.randint(0, 1), "iterations": rng.choice((1, 3, 3, 4))}
    if kind == "accumulate":
        w, h = _size(rng, 0.3, 6.0)
        return {"kind": kind, "n": rng.randint(1, 6), "w": w, "h": h, "scale": rng.choice((1.0, 1.0, 2.0, 2.0, 1.5, 3.0)), "cfa": cfa}
    if kind == "pef":
        w, h = _size(rng, 0.5, 16.0)
        return {"kind": kind, "w": w, "h": h}
    if kind == "dng":
        w, h = _size(rng, 0.5, 8.0)
        return {"kind": kind, "w": w, "h": h}
    w, h = _size(rng, 1.0, 90.0)
    return {"kind": "post", "w": w + rng.randint(0, 3), "h": h}


# ---- inputs ------------------------------------------------------------------

def _rand_map(gen, channels, h, w, cells):
    """Smooth random map: unit normal values on a grid of about `cells` cells across, bicubic in between."""
    gh, gw = max(4, round(cells * h / max(h, w))), max(4, round(cells * w / max(h, w)))
    g = torch.randn((1, channels, gh, gw), generator=gen, device="cuda")
    return F.interpolate(g, size=(h, w), mode="bicubic", align_corners=False)[0]


def _scene(gen, h, w):
    """Linear RGB scene (3 x h x w): shading, coloured regions with hard edges, texture from coarse to about 3 px."""
    s = 0.3 + 0.06 * _rand_map(gen, 3, h, w, 5)
    for cells, amp in ((max(h, w) / 130.0, 0.10), (max(h, w) / 40.0, 0.07)):
        region = torch.sign(_rand_map(gen, 1, h, w, cells))
        s += amp * region * (0.7 + 0.3 * torch.randn((3, 1, 1), generator=gen, device="cuda"))
    s += 0.05 * _rand_map(gen, 3, h, w, max(h, w) / 12.0)
    s += 0.03 * _rand_map(gen, 1, h, w, max(h, w) / 3.0)
    return s.clamp_(0.02, 0.95)


def _motion(case, seed):
    r = np.random.default_rng(seed * 7919 + 3)
    n = case.get("n", 2)
    shifts = r.uniform(-8.0, 8.0, (n, 2))
    rots = np.deg2rad(r.uniform(-0.15, 0.15, n))
    shifts[0], rots[0] = 0.0, 0.0
    return shifts, rots


def _moved(scene, h, w, margin, shift, rot):
    """The scene under a rotation about the frame centre and a shift (3 x h x w)."""
    hp, wp = scene.shape[1:]
    y = torch.arange(h, device="cuda", dtype=torch.float32).view(h, 1) - (h - 1) / 2.0
    x = torch.arange(w, device="cuda", dtype=torch.float32).view(1, w) - (w - 1) / 2.0
    c, s = math.cos(rot), math.sin(rot)
    sx = c * x - s * y + (w - 1) / 2.0 + shift[0] + margin
    sy = s * x + c * y + (h - 1) / 2.0 + shift[1] + margin
    grid = torch.stack([(sx + 0.5) / wp * 2 - 1, (sy + 0.5) / hp * 2 - 1], dim=-1)[None]
    return F.grid_sample(scene[None], grid, mode="bicubic", padding_mode="border", align_corners=False)[0].clamp_(0, 1)


def _frames(case, seed):
    """n moved RGB frames of the case's size, one at a time."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["h"], case["w"]
    shifts, rots = _motion(case, seed)
    margin = 12 + int(0.003 * math.hypot(h, w))
    scene = _scene(gen, h + 2 * margin, w + 2 * margin)
    for shift, rot in zip(shifts, rots):
        yield _moved(scene, h, w, margin, shift, rot), gen


def _mosaic(rgb, cfa, gen):
    """14-bit Bayer frame (int16 storage of uint16) of a linear RGB frame, with shot and read noise."""
    h, w = rgb.shape[1:]
    m = torch.empty((h, w), device="cuda")
    for k, c in enumerate(CFA[cfa]):
        m[k >> 1::2, k & 1::2] = rgb[c, k >> 1::2, k & 1::2]
    m += torch.sqrt(NOISE_A * m + NOISE_B) * torch.randn((h, w), generator=gen, device="cuda")
    return torch.round(BLACK + m * (WHITE - BLACK)).clamp_(0, WHITE).to(torch.int16)


def _burst(case, seed):
    raw = torch.empty((case.get("n", 1), case["h"], case["w"]), dtype=torch.int16, device="cuda")
    for i, (rgb, gen) in enumerate(_frames(case, seed)):
        if i < len(raw):
            raw[i] = _mosaic(rgb, case["cfa"], gen)
    return raw


def _info(case):
    info = isa.IsaRawInfo()
    info.width, info.height = case["w"], case["h"]
    for k in range(4):
        info.cfa[k] = CFA[case["cfa"]][k]
    for c in range(3):
        info.black[c], info.white[c], info.camera_white[c] = BLACK, WHITE - BLACK, 1.0
    info.noise_alpha, info.noise_beta = NOISE_A, NOISE_B
    return info


def _gray_frames(case, seed, high_pass):
    """Gray frames as the tile search (high-passed, [0, 1]) or the refinement (gamma curve) meets them."""
    out = []
    for rgb, gen in _frames(case, seed):
        g = (0.2989 * rgb[0] + 0.587 * rgb[1] + 0.1141 * rgb[2]).pow_(1 / 2.4)
        g += 0.01 * torch.randn(g.shape, generator=gen, device="cuda")
        if high_pass:
            low = F.avg_pool2d(F.pad(g[None, None], (32, 32, 32, 32), mode="replicate"), 65, 1)[0, 0]
            g = g - low
        out.append(g.clamp_(0, 1))
    return out


def _tile_counts(case, tile, shift):
    return (case["w"] - 2 * shift) // tile, (case["h"] - 2 * shift) // tile


def _kernels(gen, h, w):
    """Kernel parameters (h x w x 4) of the range the library computes: a rotated Gaussian per pixel, k_detail .. k_denoise."""
    k1 = (0.25 * torch.exp(1.4 * torch.rand((h, w), generator=gen, device="cuda"))).square_()
    k2 = (0.12 * torch.exp(1.8 * torch.rand((h, w), generator=gen, device="cuda"))).square_()
    th = math.pi * torch.rand((h, w), generator=gen, device="cuda")
    c, s = torch.cos(th), torch.sin(th)
    b11, b12, b22 = k1 * c * c + k2 * s * s, (k1 - k2) * c * s, k1 * s * s + k2 * c * c
    det = b11 * b22 - b12 * b12
    return torch.stack([b22 / det, b11 / det, -b12 / det, torch.zeros_like(det)], dim=-1).contiguous()


def _accumulate_inputs(case, seed):
    raw = _burst(case, seed)
    n, h, w = raw.shape
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    kp = _kernels(gen, h, w)
    flows, masks = [], []
    for i in range(n):
        # a frame's flow: its shift, a slow drift and LK's pixel noise, in steps of 1 / 64 px (the rounding of
        # the scaled flow is then the same in 32 and in 64 bits at whole scales)
        f = torch.randn((2, 1, 1), generator=gen, device="cuda") * 6 + 0.5 * _rand_map(gen, 2, h, w, 6)
        f = f + 0.1 * torch.randn((2, h, w), generator=gen, device="cuda")
        flows.append((torch.round(f * 64) / 64).permute(1, 2, 0).contiguous() if i else None)
        m = (1.1 + 0.5 * _rand_map(gen, 4, h // 2, w // 2, 40) + 0.1 * torch.randn((4, h // 2, w // 2), generator=gen, device="cuda")).clamp_(0, 1)
        masks.append(m.permute(1, 2, 0).contiguous() if i else None)
    return raw, kp, flows, masks


def _params(case):
    return P.MergeParams(merge_scale=case["scale"])


def _bayer_frame(case, seed):
    c = dict(case, cfa="RGGB", n=1)
    return _burst(c, seed)[0]


CODE_LENGTHS = (2, 3, 3, 3, 3, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13)


def _codes(lengths):
    """Canonical prefix code words of the category lengths (right-aligned)."""
    code, c = [0] * len(lengths), 0
    for ln in range(1, 17):
        for k, v in enumerate(lengths):
            if v == ln:
                code[k] = c
                c += 1
        c <<= 1
    return code


def _fields(d, lengths):
    """Code and difference bits of the differences d (any shape, int64): (bit field, bit count)."""
    mag = d.abs()
    cat = torch.ceil(torch.log2(mag.double() + 1)).long()  # bit length of |d|
    clen = torch.tensor(lengths, device="cuda")[cat]
    code = torch.tensor(_codes(lengths), device="cuda")[cat]
    bits = torch.where(d >= 0, d, d - 1) & ((1 << cat) - 1)
    return (code << cat) | bits, clen + cat


def _pack(field, flen, start, nbytes):
    """The fields as a byte string, MSB first, field i at bit start[i]."""
    w = start >> 5
    at = 64 - (start & 31) - flen  # low bit in the 64-bit pair of words (w, w + 1)
    hi = torch.where(at >= 32, field << (at - 32).clamp(min=0), field >> (32 - at).clamp(min=0))
    lo = torch.where(at >= 32, torch.zeros_like(field), (field << at.clamp(max=31)) & 0xFFFFFFFF)
    words = torch.zeros(nbytes // 4 + 3, dtype=torch.int64, device="cuda")
    words.index_add_(0, w, hi)
    words.index_add_(0, w + 1, lo)
    return words.view(torch.uint8).reshape(-1, 8)[:, [3, 2, 1, 0]].reshape(-1)[:nbytes].contiguous()


def _pef_stream(img):
    """A compressed PEF strip of the frame: differences to two columns left, or two rows up in the first two columns."""
    v = img.long()
    d = v.clone()
    d[:, 2:] -= v[:, :-2]
    d[2:, :2] -= v[:-2, :2]
    field, flen = _fields(d.reshape(-1), CODE_LENGTHS[:15])
    end = torch.cumsum(flen, 0)
    return _pack(field, flen, end - flen, (int(end[-1]) + 7) // 8)


def _pef_table():
    import struct
    lens = CODE_LENGTHS[:15]
    left = [c << (12 - n) for c, n in zip(_codes(lens), lens)]
    note = struct.pack("<H", 3) + bytes(12) + struct.pack("<15H", *left) + bytes(lens)
    return isa.pef_huff_table(note)


def _dng_file(img, tile=256):
    """A file image holding the frame as lossless-JPEG tiles (two interleaved components, predictor 1): (file, offsets, counts)."""
    h, w = img.shape
    th, tw = -(-h // tile), -(-w // tile)
    v = torch.zeros((th * tile, tw * tile), dtype=torch.int64, device="cuda")
    v[:h, :w] = img
    t = v.reshape(th, tile, tw, tile).permute(0, 2, 1, 3).reshape(th * tw, tile, tile)
    d = t.clone()
    d[:, :, 2:] -= t[:, :, :-2]
    d[:, 0, :2] -= 1 << 13
    d[:, 1:, :2] -= t[:, :-1, :2]
    field, flen = _fields(d.reshape(th * tw, -1), CODE_LENGTHS)
    bits = flen.sum(1)
    nbytes = (bits + 7) // 8
    first = torch.cumsum(nbytes, 0) - nbytes
    pad = nbytes * 8 - bits  # the last byte is padded with ones
    field = torch.cat([field, ((1 << pad) - 1)[:, None]], 1)
    flen = torch.cat([flen, pad[:, None]], 1)
    start = torch.cumsum(flen, 1) - flen + 8 * first[:, None]
    data = _pack(field.reshape(-1), flen.reshape(-1), start.reshape(-1), int(nbytes.sum())).cpu().numpy()
    counts = [CODE_LENGTHS.count(n) for n in range(1, 17)]
    values = sorted(range(16), key=lambda k: (CODE_LENGTHS[k], k))
    head = bytes([0xFF, 0xD8, 0xFF, 0xC3, 0, 14, 14, tile >> 8, tile & 255, tile // 2 >> 8, tile // 2 & 255, 2, 1, 0x11, 0, 2, 0x11, 0,
                  0xFF, 0xC4, 0, 35, 0] + counts + values + [0xFF, 0xDA, 0, 10, 2, 1, 0, 2, 0, 1, 0, 0])
    head = np.frombuffer(head, np.uint8)
    parts, offs, cnts, pos = [np.zeros(64, np.uint8)], [], [], 64
    for a, n in zip(first.tolist(), nbytes.tolist()):
        body = data[a:a + n]
        body = np.insert(body, np.flatnonzero(body == 0xFF) + 1, 0)
        parts += [head, body, np.array([0xFF, 0xD9], np.uint8)]
        offs.append(pos)
        cnts.append(len(head) + len(body) + 2)
        pos += cnts[-1]
    return np.concatenate(parts), np.array(offs, np.uint32), np.array(cnts, np.uint32)


# ---- a pass ------------------------------------------------------------------

def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "merge":
        s.update(raw=_burst(case, seed), info=_info(case), merger=isa.Merger(case["w"], case["h"], case["n"], _params(case)))
    elif kind == "batch":
        p = _params(case)
        s["mergers"] = [isa.Merger(case["w"], case["h"], case["n"], p) for _ in range(case["contexts"])]
        s["streams"] = [torch.cuda.Stream() for _ in range(case["contexts"])]
        wo, ho = s["mergers"][0].output_size(case["w"], case["h"])
        info = _info(case)
        s["bursts"] = [{"raw": _burst(case, seed * 64 + b), "info": info, "out": torch.empty((ho, wo, 3), device="cuda")}
                       for b in range(case["bursts"])]
    elif kind == "fit":
        raw, info = _burst(case, seed), _info(case)
        m = isa.Merger(case["w"], case["h"], case["n"], _params(case))
        wo, ho = m.output_size(case["w"], case["h"])
        clean = next(_frames(case, seed))[0]
        target = F.interpolate(clean[None], size=(ho, wo), mode="bilinear", align_corners=False)[0].permute(1, 2, 0).contiguous()
        s.update(raw=raw, info=info, merger=m, target=target)
    elif kind == "tracking":
        s.update(raw=_burst(dict(case, n=1), seed)[0].contiguous(), info=_info(case), merger=isa.Merger(case["w"], case["h"], 2, P.MergeParams()),
                 out=torch.empty((case["h"], case["w"]), device="cuda"))
    elif kind == "tiles":
        frames = _gray_frames(case, seed, True)
        shifts, rots = _motion(case, seed)
        tcx, tcy = _tile_counts(case, case["tile"], case["shift"])
        pairs = [(r, t) for r in range(case["n"]) for t in range(r + 1, case["n"])]
        tab = (isa.IsaTrackPair * len(pairs))()
        for k, (r, t) in enumerate(pairs):
            tab[k].reference, tab[k].to_track, tab[k].grid = r, t, k
        # what the coarser level leaves: the pair's motion at each tile within about half a pixel
        cy = (torch.arange(tcy, device="cuda") + 0.5) * case["tile"] - case["h"] / 2
        cx = (torch.arange(tcx, device="cuda") + 0.5) * case["tile"] - case["w"] / 2
        gen = torch.Generator(device="cuda").manual_seed(seed + 5)
        pre = torch.empty((len(pairs), tcy, tcx, 2), device="cuda")
        for k, (r, t) in enumerate(pairs):
            a = rots[t] - rots[r]
            pre[k, ..., 0] = shifts[r][0] - shifts[t][0] + a * cy[:, None]
            pre[k, ..., 1] = shifts[r][1] - shifts[t][1] - a * cx[None, :]
        pre += 0.4 * torch.randn(pre.shape, generator=gen, device="cuda")
        s.update(frames=frames, ptrs=torch.tensor([f.data_ptr() for f in frames], device="cuda"), pre=pre, grids=torch.empty_like(pre),
                 argmin=torch.empty((len(pairs), tcy, tcx), dtype=torch.int32, device="cuda"), npairs=len(pairs), tcx=tcx, tcy=tcy, pairs=pairs,
                 tab=torch.frombuffer(bytearray(bytes(tab)), dtype=torch.uint8).cuda())
    elif kind == "lk":
        ref, src = _gray_frames(dict(case, n=2), seed, False)
        shifts, rots = _motion(dict(case, n=2), seed)
        tcx, tcy = _tile_counts(case, 32, 2)
        cy = (torch.arange(tcy, device="cuda") + 0.5) * 32 - case["h"] / 2
        cx = (torch.arange(tcx, device="cuda") + 0.5) * 32 - case["w"] / 2
        tiles = torch.empty((tcy, tcx, 2), device="cuda")
        tiles[..., 0] = -shifts[1][0] + rots[1] * cy[:, None]
        tiles[..., 1] = -shifts[1][1] - rots[1] * cx[None, :]
        gen = torch.Generator(device="cuda").manual_seed(seed + 6)
        tiles += 0.2 * torch.randn(tiles.shape, generator=gen, device="cuda")
        s.update(src=src, ref=ref, tiles=tiles, flow=torch.empty((case["h"], case["w"], 2), device="cuda"),
                 scratch=torch.empty((case["h"], case["w"], 2), device="cuda"))
    elif kind == "accumulate":
        raw, kp, flows, masks = _accumulate_inputs(case, seed)
        wo, ho = round(case["w"] * case["scale"]), round(case["h"] * case["scale"])
        s.update(raw=raw, kp=kp, flows=flows, masks=masks, acc=torch.empty((ho, wo, 3), device="cuda"), wsum=torch.empty((ho, wo, 3), device="cuda"))
    elif kind == "pef":
        data = _pef_stream(_bayer_frame(case, seed))
        need = isa.lib().isa_pef_decode_scratch(ctypes.c_size_t(data.numel()), case["w"], case["h"])
        s.update(data=data, table=_pef_table(), scratch=torch.empty(need, dtype=torch.uint8, device="cuda"),
                 out=torch.empty((case["h"], case["w"]), dtype=torch.int16, device="cuda"))
    elif kind == "dng":
        f, offs, cnts = _dng_file(_bayer_frame(case, seed))
        kw = dict(tiled=True, tile_w=256, tile_h=256)
        need = isa.dng_decode_scratch(f, case["w"], case["h"], offs, cnts, **kw)
        s.update(file=f, dev=torch.from_numpy(f).cuda(), offs=offs, cnts=cnts, kw=kw, scratch=torch.empty(need, dtype=torch.uint8, device="cuda"),
                 out=torch.empty((case["h"], case["w"]), dtype=torch.int16, device="cuda"))
    elif kind == "post":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        img = _scene(gen, case["h"], case["w"])
        img += 0.01 * torch.randn(img.shape, generator=gen, device="cuda")
        c2p, cw, _ = isa.pef_color_spec(np.array([2.1, 1.0, 1.6], np.float32))
        t1, t2 = isa.color_twists(c2p)
        lx = np.arange(256, dtype=np.float32) / 255.0
        ly = (lx ** 0.9 * (1.2 - 0.2 * lx)).astype(np.float32)
        pp, keep = isa.post_params((8, 6, case["w"] - 16, case["h"] - 12), cw, t1, t2, lx, ly, 0.3)
        s.update(img=img.permute(1, 2, 0).contiguous(), pp=pp, keep=keep,
                 out=torch.empty((case["h"] - 12, case["w"] - 16, 3), dtype=torch.int16, device="cuda"))
    return s


def _sz(v):
    return ctypes.c_size_t(int(v))


def run(s):
    case = s["case"]
    kind, w, h = case["kind"], case["w"], case["h"]
    lib = isa.lib()
    if kind == "merge":
        return s["merger"].merge(s["raw"], s["info"])
    if kind == "batch":
        here = torch.cuda.current_stream()
        for st in s["streams"]:
            st.wait_stream(here)
        status = isa.merge_batch(s["mergers"], s["bursts"], s["streams"])
        if any(status):
            raise RuntimeError(f"merge_batch: {status}")
        for st in s["streams"]:
            here.wait_stream(st)
        return [b["out"] for b in s["bursts"]]
    if kind == "fit":
        out, loss, grad = s["merger"].backward(s["raw"], s["info"], s["target"])
        # sums of 32-bit terms
        return {"out": out, "loss": np.float32(loss), "grad": grad.astype(np.float32)}
    if kind == "tracking":
        isa.check(lib.isa_bw_image(s["merger"].ctx, isa.vp(s["raw"]), _sz(w * 2), w, h, ctypes.byref(s["info"]), ctypes.c_float(0.5), 1,
                                   isa.vp(s["out"]), _sz(w * 4), isa.stream_ptr()))
        return s["out"]
    if kind == "tiles":
        s["grids"].copy_(s["pre"])  # the search updates the grids in place
        tcx, tcy = s["tcx"], s["tcy"]
        isa.check(lib.isa_track_level(isa.vp(s["ptrs"]), _sz(w * 4), w, h, case["tile"], case["shift"], tcx, tcy, isa.vp(s["tab"]), s["npairs"],
                                      isa.vp(s["grids"]), _sz(tcx * 8), _sz(tcx * tcy * 8), ctypes.c_float(1.0), None, isa.vp(s["argmin"]),
                                      isa.stream_ptr()))
        return {"grids": s["grids"], "argmin": s["argmin"]}
    if kind == "lk":
        tcx, tcy = s["tiles"].shape[1], s["tiles"].shape[0]
        isa.check(lib.isa_lk_refine(isa.vp(s["src"]), isa.vp(s["ref"]), _sz(w * 4), w, h, isa.vp(s["tiles"]), _sz(tcx * 8), tcx, tcy,
                                    (ctypes.c_float * 2)(0.0, 0.0), ctypes.c_float(0.0), case["iterations"], ctypes.c_float(0.01), 11,
                                    isa.vp(s["flow"]), isa.vp(s["scratch"]), _sz(w * 8), isa.stream_ptr()))
        return s["flow"]
    if kind == "accumulate":
        s["acc"].zero_()
        s["wsum"].zero_()
        wo, ho = s["acc"].shape[1], s["acc"].shape[0]
        cfa = (ctypes.c_int * 4)(*CFA[case["cfa"]])
        white, black = (ctypes.c_float * 3)(*[WHITE - BLACK] * 3), (ctypes.c_float * 3)(*[BLACK] * 3)
        crop = (ctypes.c_int * 4)(0, 0, w - 1, h - 1)
        for raw, flow, mask in zip(s["raw"], s["flows"], s["masks"]):
            isa.check(lib.isa_accumulate(isa.vp(raw), _sz(w * 2), w, h, cfa, isa.vp(s["acc"]), isa.vp(s["wsum"]), _sz(wo * 12), wo, ho, isa.vp(mask),
                                         _sz(w // 2 * 16), isa.vp(s["kp"]), _sz(w * 16), 4, isa.vp(flow), _sz(w * 8), white, black,
                                         ctypes.c_float(case["scale"]), 0, 0, crop, isa.stream_ptr()))
        return {"acc": s["acc"], "wsum": s["wsum"]}
    if kind == "pef":
        return isa.pef_decode(s["data"], s["table"], w, h, s["out"], s["scratch"])
    if kind == "dng":
        return isa.dng_decode(s["file"], w, h, s["offs"], s["cnts"], file_dev=s["dev"], scratch=s["scratch"], out=s["out"], **s["kw"])
    return isa.postprocess(s["img"], s["pp"], isa.POST_RGB16, s["out"])


# ---- what a pass cannot do without --------------------------------------------

def _merge_flops(n, w, h, wo, ho):
    px, pairs = w * h, n * (n - 1) / 2
    # per frame pixel: demosaic, gamma and high-pass about 120; three LK iterations of warp, derivatives, products,
    # sliding window sums and solve about 120 each; mask about 60. Tile search: a subtraction and a multiply-add per
    # template pixel and shift over the four levels (5 x 5, then 9 x 9 shifts). Accumulation: 25 weighted taps in two sums.
    track = 3.0 * pairs * px * (25 + 81 * (1 / 4 + 1 / 16 + 1 / 64))
    return n * px * (120 + 360 + 60) + track + n * wo * ho * 25 * 4.0


def work(case):
    kind, w, h = case["kind"], case["w"], case["h"]
    px = float(w * h)
    if kind in ("merge", "batch", "fit"):
        s = case["scale"] or 1.0
        wo, ho, n = round(w * s), round(h * s), case["n"]
        k = case.get("bursts", 1)
        b, f = n * px * 2 + wo * ho * 12.0, _merge_flops(n, w, h, wo, ho)
        if kind == "fit":  # the target is read too; the gradient repeats the accumulation and needs its derivatives
            b, f = b + wo * ho * 12.0, f + n * wo * ho * 25 * 8.0
        return {"bytes": k * b, "flops": k * f}
    if kind == "tracking":
        return {"bytes": px * 6, "flops": px * (100 + 2.5 * 2 * math.log2(w) + 10)}
    if kind == "tiles":
        tcx, tcy = _tile_counts(case, case["tile"], case["shift"])
        pairs, d = case["n"] * (case["n"] - 1) / 2, 2 * case["shift"] + 1
        return {"bytes": case["n"] * px * 4 + pairs * tcx * tcy * 20, "flops": 3.0 * pairs * tcx * tcy * case["tile"] ** 2 * d * d}
    if kind == "lk":
        return {"bytes": px * 16, "flops": case["iterations"] * px * 120}
    if kind == "accumulate":
        wo, ho, n = round(w * case["scale"]), round(h * case["scale"]), case["n"]
        return {"bytes": n * px * 14 + px * 16 + wo * ho * 24.0, "flops": n * wo * ho * 25 * 4.0}
    if kind in ("pef", "dng"):
        return {"bytes": px * 4, "flops": 0}
    return {"bytes": px * 18, "flops": px * 150}


# ---- the outputs in 64 bits ----------------------------------------------------

def _mirror(i, n):
    j = torch.remainder(i, 2 * n)
    return torch.where(j >= n, 2 * n - 1 - j, j)


def _sample(img, x, y, fold):
    """Bilinear samples of img (h x w) at texel coordinates x, y, with indices folded by `fold`."""
    h, w = img.shape
    fx, fy = torch.floor(x), torch.floor(y)
    a, b = x - fx, y - fy
    x0, x1, y0, y1 = fold(fx.long(), w), fold(fx.long() + 1, w), fold(fy.long(), h), fold(fy.long() + 1, h)
    return ((1 - a) * (1 - b) * img[y0, x0] + a * (1 - b) * img[y0, x1] + (1 - a) * b * img[y1, x0] + a * b * img[y1, x1])


def _clamp(i, n):
    return i.clamp(0, n - 1)


def _exact_tracking(case, seed):
    raw = _burst(dict(case, n=1), seed)[0].double()
    h, w = raw.shape
    lin = raw - BLACK
    yy, xx = torch.arange(h, device="cuda").view(h, 1), torch.arange(w, device="cuda").view(1, w)
    code = torch.tensor(CFA[case["cfa"]], device="cuda")[(yy % 2) * 2 + xx % 2]
    inner = (xx >= 2) & (xx < w - 2) & (yy >= 2) & (yy < h - 2)

    def at(a, dy, dx):
        return F.pad(a, (2, 2, 2, 2))[2 + dy:2 + dy + h, 2 + dx:2 + dx + w]

    def along(dy, dx):
        m2, m1, p1, p2 = at(lin, -2 * dy, -2 * dx), at(lin, -dy, -dx), at(lin, dy, dx), at(lin, 2 * dy, 2 * dx)
        return 0.5 * (p1 - m1).abs() + 0.25 * (2 * lin - m2 - p2).abs(), 0.125 * (-m2 + 4 * m1 + 2 * lin + 4 * p1 - p2)

    gx, ix = along(0, 1)
    gy, iy = along(1, 0)
    wt = gy / (gx + gy + 1e-9)
    g = torch.where(code == 1, lin, wt * ix + (1 - wt) * iy) * inner
    d = lin - g
    hor = g + 0.5 * (at(d, 0, -1) + at(d, 0, 1))
    ver = g + 0.5 * (at(d, -1, 0) + at(d, 1, 0))
    dia = g + 0.25 * (at(d, -1, -1) + at(d, -1, 1) + at(d, 1, -1) + at(d, 1, 1))
    red_row = torch.tensor([0 in CFA[case["cfa"]][:2], 0 in CFA[case["cfa"]][2:]], device="cuda")[yy % 2]
    r = torch.where(code == 0, lin, torch.where(code == 2, dia, torch.where(red_row, hor, ver)))
    b = torch.where(code == 2, lin, torch.where(code == 0, dia, torch.where(red_row, ver, hor)))
    gray = 0.0
    for wgt, v in ((0.2989, r), (0.5870, g), (0.1141, b)):
        v = ((v * inner) / (WHITE - BLACK)).clamp(0, 1)
        v = torch.where(v <= 0.0031308, 12.92 * v, 1.055 * v.clamp(min=1e-12) ** (1 / 2.4) - 0.055)
        gray = gray + float(np.float32(wgt)) * v
    ky = torch.arange(h, device="cuda", dtype=torch.float64).view(h, 1)
    ky = torch.where(ky > h * 0.5, ky - h, ky) / h
    kx = torch.arange(w // 2 + 1, device="cuda", dtype=torch.float64).view(1, -1) / w
    dist = torch.sqrt(kx * kx + ky * ky)
    hp, hps = float(np.float32(0.01)) + float(np.float32(0.0025)), float(np.float32(0.0025))
    low = torch.exp(-((dist - hp) ** 2) / (2 * hps * hps))
    fil = torch.where(dist >= hp, torch.ones_like(low), torch.where(low > 0.001, low, torch.zeros_like(low)))
    img = torch.fft.irfft2(torch.fft.rfft2(gray) * fil, s=(h, w)).clamp(0, 1)
    t = math.exp(-2.0)
    t = torch.tensor([t, 1.0, t], device="cuda", dtype=torch.float64) / (1 + 2 * t)
    for ax in (0, 1):
        p = F.pad(img[None, None], (1, 1, 0, 0) if ax == 0 else (0, 0, 1, 1), mode="replicate")[0, 0]
        img = t[0] * p[:, :-2] + t[1] * p[:, 1:-1] + t[2] * p[:, 2:] if ax == 0 else t[0] * p[:-2] + t[1] * p[1:-1] + t[2] * p[2:]
    return img


def _exact_tiles(case, seed):
    s = prepare(case, seed)
    T, S, D = case["tile"], case["shift"], 2 * case["shift"] + 1
    h, w, tcx, tcy = case["h"], case["w"], s["tcx"], s["tcy"]
    ty, tx = torch.arange(tcy, device="cuda").view(-1, 1) * T, torch.arange(tcx, device="cuda").view(1, -1) * T
    u, v = torch.arange(T, device="cuda"), torch.arange(T + 2 * S, device="cuda")
    out = s["pre"].double()
    best = torch.empty((len(s["pairs"]), tcy, tcx), dtype=torch.int32, device="cuda")

    def block(img, oy, ox, k):  # tiles x tiles x k x k blocks with replicated borders
        yy = (oy[..., None] + k).clamp(0, h - 1)
        xx = (ox[..., None] + k).clamp(0, w - 1)
        return img[yy[..., :, None], xx[..., None, :]]

    for k, (r, t) in enumerate(s["pairs"]):
        tpl = block(s["frames"][r].double(), (ty + S).expand(tcy, tcx), (tx + S).expand(tcy, tcx), u)
        pre = s["pre"][k].double()
        off = torch.sign(pre) * torch.floor(pre.abs() + 0.5)
        blk = block(s["frames"][t].double(), ty + off[..., 1].long(), tx + off[..., 0].long(), v)
        maps = torch.stack([((tpl - blk[:, :, j:j + T, i:i + T]) ** 2).sum((2, 3)) for j in range(D) for i in range(D)], -1)
        mn, mi = maps.min(-1)
        best[k] = mi.int()
        iy, ix = mi // D, mi % D
        edge = (ix < 1) | (iy < 1) | (ix >= 2 * S) | (iy >= 2 * S)
        m = maps.reshape(tcy, tcx, D, D)
        q = [[m.reshape(tcy, tcx, -1).gather(2, (((iy + a).clamp(0, D - 1)) * D + (ix + b).clamp(0, D - 1))[..., None])[..., 0]
              for b in (-1, 0, 1)] for a in (-1, 0, 1)]
        a11 = 0.25 * (q[0][0] - 2 * q[0][1] + q[0][2]) + 0.5 * (q[1][0] - 2 * q[1][1] + q[1][2]) + 0.25 * (q[2][0] - 2 * q[2][1] + q[2][2])
        a22 = 0.25 * (q[0][0] - 2 * q[1][0] + q[2][0]) + 0.5 * (q[0][1] - 2 * q[1][1] + q[2][1]) + 0.25 * (q[0][2] - 2 * q[1][2] + q[2][2])
        a12 = 0.25 * (q[0][0] - q[0][2] - q[2][0] + q[2][2])
        b1 = 0.125 * (q[0][2] - q[0][0] + q[2][2] - q[2][0]) + 0.25 * (q[1][2] - q[1][0])
        b2 = 0.125 * (q[2][0] - q[0][0] + q[2][2] - q[0][2]) + 0.25 * (q[2][1] - q[0][1])
        a11, a22 = a11.clamp(min=0), a22.clamp(min=0)
        det = a11 * a22 - a12 * a12
        a12 = torch.where(det < 0, torch.zeros_like(a12), a12)
        det = torch.where(det < 0, a11 * a22, det)
        ok = det != 0
        dd = torch.where(ok, det, torch.ones_like(det))
        mx, my = (a22 * b1 - a12 * b2) / dd, (a11 * b2 - a12 * b1) / dd
        mx = torch.where(ok & (mx.abs() <= 1), mx, torch.zeros_like(mx))
        my = torch.where(ok & (my.abs() <= 1), my, torch.zeros_like(my))
        none = edge | (1.0 + mn > maps.amax(-1))
        z = torch.zeros_like(mx)
        out[k, ..., 0] += torch.where(none, z, ix - mx - S)
        out[k, ..., 1] += torch.where(none, z, iy - my - S)
    return {"grids": out, "argmin": None}


def _exact_lk(case, seed):
    s = prepare(case, seed)
    h, w = case["h"], case["w"]
    src, ref, tiles = s["src"].double(), s["ref"].double(), s["tiles"].double()
    tcy, tcx = tiles.shape[:2]
    y = torch.arange(h, device="cuda", dtype=torch.float64).view(h, 1).expand(h, w)
    x = torch.arange(w, device="cuda", dtype=torch.float64).view(1, w).expand(h, w)
    u, v = (_sample(tiles[..., c], (x + 0.5) / w * tcx - 0.5, (y + 0.5) / h * tcy - 0.5, _clamp) for c in (0, 1))
    R, min_det = 5, float(np.float32(0.01))

    def five(a):  # five-tap difference along the last axis, mirrored with the edge repeated
        n = a.shape[-1]
        p = a[..., _mirror(torch.arange(-2, n + 2, device="cuda"), n)]
        return (p[..., 4:] - 8 * p[..., 3:-1] + 8 * p[..., 1:-3] - p[..., :-4]) / 12

    def window(a):  # sums over 11 x 11, valid part
        c = F.pad(a.cumsum(0), (0, 0, 1, 0))
        c = c[2 * R + 1:] - c[:-2 * R - 1]
        c = F.pad(c.cumsum(1), (1, 0))
        return c[:, 2 * R + 1:] - c[:, :-2 * R - 1]

    for _ in range(case["iterations"]):
        warped = _sample(src, x + u, y + v, _mirror)
        both = 0.5 * (warped + ref)
        gx, gy, gt = five(both), five(both.T).T, warped - ref
        a, b, d, p, q = (window(m) for m in (gx * gx, gx * gy, gy * gy, gx * gt, gy * gt))
        # the symmetric window matrix's pseudo-inverse: closed form where it is well conditioned, else its eigenvectors,
        # each direction kept unless its singular value is zero; no update where the larger one is below min_det
        root = torch.sqrt((0.5 * (a - d)) ** 2 + b * b)
        l1, l2 = 0.5 * (a + d) + root, 0.5 * (a + d) - root
        th = 0.5 * torch.atan2(2 * b, a - d)
        c, sn = torch.cos(th), torch.sin(th)
        e1 = (c * p + sn * q) / torch.where(l1 != 0, l1, torch.ones_like(l1))
        e2 = (c * q - sn * p) / torch.where(l2 != 0, l2, torch.ones_like(l2)) * (l2 != 0)
        det = a * d - b * b
        well = det > 1e-3 * l1 * l1
        dd = torch.where(well, det, torch.ones_like(det))
        du = torch.where(well, (d * p - b * q) / dd, c * e1 - sn * e2)
        dv = torch.where(well, (a * q - b * p) / dd, sn * e1 + c * e2)
        live = l1 >= min_det
        u, v = u.clone(), v.clone()
        u[R:h - R, R:w - R] += torch.where(live, du, torch.zeros_like(du))
        v[R:h - R, R:w - R] += torch.where(live, dv, torch.zeros_like(dv))
    return torch.stack([u, v], -1)


def _exact_accumulate(case, seed):
    raw, kp, flows, masks = _accumulate_inputs(case, seed)
    h, w, s = case["h"], case["w"], case["scale"]
    wo, ho = round(w * s), round(h * s)
    if case["n"] * wo * ho > 120e6:
        return None
    s = float(np.float32(s))
    y, x = torch.arange(1, ho - 1, device="cuda").view(-1, 1), torch.arange(1, wo - 1, device="cuda").view(1, -1)
    xb, yb = ((x + 0.5).double() / s - 0.5).expand(ho - 2, wo - 2), ((y + 0.5).double() / s - 0.5).expand(ho - 2, wo - 2)
    k = [_sample(kp[..., c].double(), xb, yb, _clamp) for c in range(3)]
    code = torch.tensor(CFA[case["cfa"]], device="cuda")
    acc = torch.zeros((3, ho - 2, wo - 2), dtype=torch.float64, device="cuda")
    wsum = torch.zeros_like(acc)

    def at(p, sh, n):
        return torch.floor((p + sh).double() / s).long().clamp(0, n - 1)

    for f in range(case["n"]):
        sx = sy = torch.zeros((), dtype=torch.int64, device="cuda")
        if flows[f] is not None:
            sx, sy = (_sample(flows[f][..., c].double(), xb, yb, _mirror) * s for c in (0, 1))
            sx, sy = (torch.sign(t) * torch.floor(t.abs() + 0.5) for t in (sx, sy))
        img = (raw[f].double() - BLACK) / (WHITE - BLACK)
        for py in range(-2, 3):
            for px in range(-2, 3):
                wt = torch.exp(-0.5 * (px * px * k[0] + 2 * px * py * k[2] + py * py * k[1]))
                qx, qy = at(x, px + sx, w), at(y, py + sy, h)
                c = code[(qy % 2) * 2 + qx % 2].expand(ho - 2, wo - 2)
                if masks[f] is not None:
                    wt = wt * masks[f][at(y, py, h) // 2, at(x, px, w) // 2].double().gather(2, c[..., None])[..., 0]
                acc.scatter_add_(0, c[None], (wt * img[qy, qx])[None])
                wsum.scatter_add_(0, c[None], wt[None])
    full = [F.pad(t, (1, 1, 1, 1)).permute(1, 2, 0).contiguous() for t in (acc, wsum)]
    return {"acc": full[0], "wsum": full[1]}


def exact(case, seed):
    """The operators' outputs in 64 bits; None for whole merges (their discrete decisions follow from 32-bit stages) and whole-number outputs."""
    f = {"tracking": _exact_tracking, "tiles": _exact_tiles, "lk": _exact_lk, "accumulate": _exact_accumulate}.get(case["kind"])
    return f(case, seed) if f else None
