"""The measured workloads of this framework: what its users have it do, over the range they use.

Paths (``case["path"]``):

* ``image``   one sRGB image in page-locked host memory to fitted tiles (``frontend.refine_image``):
              the encoder's fast fit as one call, from thumbnails to full frames;
* ``device``  the same fit over tiles that are already resident (``pools.DeviceRefinedFit``), pools
              generated in the run, replayed from its CUDA graph: what a service runs per frame;
* ``plain``   the reference greedy over full candidate pools (``BatchedFit.graph``): the encoder's
              search, with rounds and re-seeds;
* ``grad``    forward and backward of the stack loss (``StackLoss``): differentiable refinement;
* ``refine``  fused loss + gradient + Adam steps (``FusedRefiner``), residual-aware or not;
* ``walk``    the decoder's primitive walk into a device image (``weftk_render_tiles``), at the encoded
              size or scaled, with and without residual grids: a decoder rendering frame after frame;
* ``raster``  the decoder's raster branch on the device: walk, DCT residual layer, u8 resize;
* ``decode``  a WEFT file in host memory to its pixels (``encode.decode_file``), the whole call;
* ``score``   the drop-in scorer on host records (``gpu_batch_score_prepacked``), as the reference's
              encoder calls it each round.

Images are the canonical synthetic ones (``synth.make_image_u8``) with the density of the 1024x1024,
600-primitive workload; tiles come from the variance quadtree.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from weft_b200 import _lib, bitstream, encode, frontend, gpu_render, pools, raster, render, synth
from weft_b200._lib import PRIM_DTYPE, TILE_DECODE_DTYPE
from weft_b200.fit import BatchedFit, unpack_cands
from weft_b200.quadtree import QuadTile
from weft_b200.refine import FusedRefiner, StackLoss, StackSet

F64 = torch.float64
TILE_PX = 1024 * 1024 / 7435  # pixels per quadtree tile of the canonical images, about
# candidates per tile and kind of the reference's pools on these images (constant, linear, line, curve, triangle)
POOL = (26, 86, 86, 45, 39)
KIND_OPS = (10, 24, 28, 509, 26)  # FP32 operations per pixel to evaluate and blend a primitive


def listed():
    return [
        # a thumbnail: launches, copies and host work decide
        {"name": "image_256", "path": "image", "w": 256, "h": 256, "quality": 75, "steps": 10},
        # the headline workload, end to end
        {"name": "image_1024", "path": "image", "w": 1024, "h": 1024, "quality": 75, "steps": 10},
        # the largest frame of the repository's workloads, resident
        {"name": "device_2048", "path": "device", "w": 2048, "h": 2048, "quality": 75, "steps": 10},
        # the plain greedy on the headline image
        {"name": "plain_1024", "path": "plain", "w": 1024, "h": 1024, "quality": 75},
        # high quality: more rounds, deeper stacks, re-seeds
        {"name": "plain_512_q92", "path": "plain", "w": 512, "h": 512, "quality": 92},
        # autograd through stacks of every kind
        {"name": "grad_512", "path": "grad", "w": 512, "h": 512, "layers": 4, "residual": False},
        # refinement of a deep fit with the decoded-error loss
        {"name": "refine_1024", "path": "refine", "w": 1024, "h": 1024, "layers": 3, "steps": 20, "residual": True},
        # frame decode to a 4K target
        {"name": "walk_4k", "path": "walk", "w": 1024, "h": 1024, "tw": 3840, "th": 2160, "residuals": False},
        # an odd-sized frame at its own size, with the residual grids every file of this encoder carries
        {"name": "walk_1919_res", "path": "walk", "w": 1919, "h": 1079, "tw": 1919, "th": 1079, "residuals": True},
        # a file with a DCT layer to a 4K target
        {"name": "raster_4k", "path": "raster", "w": 1024, "h": 1024, "tw": 3840, "th": 2160, "residuals": True},
        # a file from host memory to host pixels
        {"name": "decode_1024", "path": "decode", "w": 1024, "h": 1024, "tw": 1024, "th": 1024, "residuals": True},
        # one round of the reference's encoder on a 256x256 image's tiles
        {"name": "score_379", "path": "score", "tiles": 379, "evals": 282, "depth": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case; frames from 64 px to the listed largest of their path, any side, any aspect up to 2:1."""
    path = rng.choice(("image", "device", "plain", "grad", "refine", "walk", "walk", "raster", "decode", "score"))
    if path == "score":
        return {"path": path, "tiles": _log(rng, 1, 379), "evals": _log(rng, 8, 282), "depth": rng.randint(1, 2)}
    most = {"image": 1024, "device": 2048, "plain": 700, "grad": 512, "refine": 1024, "walk": 1440, "raster": 1024,
            "decode": 1024}[path]
    side = _log(rng, 64, most)
    w = max(33, min(most, int(side * rng.uniform(0.71, 1.41))))
    h = max(33, min(most, int(side * side / w)))
    case = {"path": path, "w": w, "h": h}
    if path in ("image", "device"):
        case.update(quality=rng.choice((50, 75, 75, 75, 92)), steps=rng.choice((10, 10, 20)))
    elif path == "plain":
        case.update(quality=rng.choice((50, 75, 75)))
    elif path in ("grad", "refine"):
        case.update(layers=rng.randint(1, 4 if path == "grad" else 3), residual=rng.random() < 0.5)
        if path == "refine":
            case.update(steps=rng.randint(1, 20))
    else:
        up = rng.choice((1.0, 1.0, 0.5, 1.5, 2.0) if path == "decode" else (1.0, 0.5, 1.5, 2.0, 2.25))
        limit = 1920 if path == "decode" else 3840
        case.update(tw=max(16, min(limit, int(w * up))), th=max(16, min(limit, int(h * up))),
                    residuals=rng.random() < 0.6)
    return case


# --------------------------------------------------------------------------------------- inputs
def _image(case, seed):
    prims = max(4, round(case["w"] * case["h"] * 600 / 2 ** 20))
    return synth.make_image_u8(case["w"], case["h"], prims, seed)


def _tiles(u8):
    """The image on the device, its quadtree (host (n, 3) int32) and its tiles' float4 pixels."""
    img = torch.from_numpy(u8).cuda()
    tiles, _ = frontend.decompose_device(img)
    host = tiles.cpu().numpy()
    src4, px_off = frontend.extract_device(img, tiles, host[:, 2])
    return host, src4, px_off


def _tile_set(case, seed):
    """Tiles of the image in fixed numbers of each side (the canonical images' mix, n = w h / TILE_PX), so
    that every seed of a case has the same layout: as ``_tiles``."""
    img = torch.from_numpy(_image(case, seed)).cuda()
    found, _ = frontend.decompose_device(img)
    found = found.cpu().numpy()
    rng = np.random.default_rng(seed + 3)
    n = max(8, round(case["w"] * case["h"] / TILE_PX))
    counts = {16: round(0.141 * n), 32: round(0.0305 * n), 64: round(0.0051 * n)}
    counts[8] = n - sum(counts.values())
    parts = []
    for s, k in sorted(counts.items()):
        have = found[found[:, 2] == s]
        if len(have):
            parts.append(have[rng.permutation(np.arange(max(k, len(have))) % len(have))[:k]])
        else:  # an image without tiles of this side: squares of it anywhere
            xy = np.stack([rng.integers(0, case["w"], k), rng.integers(0, case["h"], k)], 1)
            parts.append(np.concatenate([xy, np.full((k, 1), s)], 1).astype(np.int32))
    host = np.concatenate(parts)[np.random.default_rng(n).permutation(n)].astype(np.int32)
    src4, px_off = frontend.extract_device(img, torch.from_numpy(host).cuda(), host[:, 2])
    return host, src4, px_off


def _primitives(rng, kinds, sides, colours):
    """Records of the given kinds over tiles of the given sides, around the given colours: coordinates
    inside the tile and the wire range, thickness 0.4 .. 3, alpha 0.2 .. 1."""
    n = len(kinds)
    top = np.minimum(sides - 1.0, 15.0)[:, None]
    rec = np.zeros(n, PRIM_DTYPE)
    rec["kind"] = kinds
    geom = (rng.uniform(0.0, 1.0, (n, 7)) * top).astype(np.float32)
    thick = rng.choice(np.array([0.4, 0.5, 0.8, 1.0, 1.2, 2.0, 3.0], np.float32), n)
    geom[:, 4] = np.where(kinds == 2, thick, geom[:, 4])
    geom[:, 6] = np.where(kinds == 3, thick, geom[:, 6])
    used = np.array([0, 4, 5, 7, 6])[kinds]
    rec["geom"] = np.where(np.arange(7) < used[:, None], geom, 0.0)
    rec["color0"] = np.clip(colours + rng.normal(0.0, 0.08, (n, 3)), 0.0, 1.0)
    rec["color1"] = np.where(kinds[:, None] == 1, np.clip(colours + rng.normal(0.0, 0.08, (n, 3)), 0.0, 1.0), 0.0)
    rec["alpha"] = np.where(kinds == 0, rng.choice([1.0, 1.0, 1.0, 0.7], n), rng.uniform(0.2, 1.0, n))
    return rec


def _tile_colours(rng, src4, px_off, sides):
    """One pixel's colour per tile."""
    at = px_off.cpu().numpy().astype(np.int64) + rng.integers(0, sides.astype(np.int64) ** 2)
    return src4[torch.from_numpy(at).to(src4.device), :3].cpu().numpy().astype(np.float64)


def _scene(case, seed):
    """Tiles and stacks of a decoded file: mostly lone constant layers, some linear, some deeper."""
    rng = np.random.default_rng(seed)
    tiles, src4, px_off = _tiles(_image(case, seed))
    sides = tiles[:, 2]
    n = len(tiles)
    u = rng.random(n)
    counts = np.where(u < 0.97, 1, rng.integers(2, 5, n))
    off = np.concatenate([[0], np.cumsum(counts)])
    tile = np.repeat(np.arange(n), counts)
    kinds = np.where(u[tile] < 0.94, 0, np.where(u[tile] < 0.97, 1, rng.integers(0, 5, len(tile))))
    kinds[off[:-1]] = np.where(u < 0.94, 0, np.where(u < 0.97, 1, 0))
    rec = _primitives(rng, kinds, sides[tile], _tile_colours(rng, src4, px_off, sides)[tile])
    rec["color0"] = np.round(rec["color0"] * 255.0) / 255.0
    rec["color1"] = np.round(rec["color1"] * 255.0) / 255.0
    res0 = res1 = None
    if case["residuals"]:
        res0 = rng.integers(-12, 13, (n, 3))
        res1 = np.clip(np.round(rng.normal(0.0, 6.0, (n, 48))), -127, 127).astype(np.int8)
    return tiles, rec, off, res0, res1


def _descs(case, tiles, off, res0, tw, th):
    """Decode descriptors: every tile's target rect (edges rounded, as the decoder does) and stack."""
    sx, sy = tw / case["w"], th / case["h"]
    x, y, s = tiles[:, 0].astype(np.float64), tiles[:, 1].astype(np.float64), tiles[:, 2]
    x0, y0 = np.rint(x * sx), np.rint(y * sy)
    d = np.zeros(len(tiles), TILE_DECODE_DTYPE)
    d["prim_offset"], d["prim_count"] = off[:-1], np.diff(off)
    d["target_x0"], d["target_y0"] = x0, y0
    d["target_w"] = np.maximum(1, np.rint((x + s) * sx) - x0)
    d["target_h"] = np.maximum(1, np.rint((y + s) * sy) - y0)
    d["source_size"] = s
    d["res1_index"] = -1 if res0 is None else np.arange(len(tiles))
    if res0 is not None:
        r = res0.astype(np.float32) / np.float32(255.0)
        d["res0_r"], d["res0_g"], d["res0_b"] = r[:, 0], r[:, 1], r[:, 2]
    return d


def _walk_state(case, seed, tw, th):
    tiles, rec, off, res0, res1 = _scene(case, seed)
    d = _descs(case, tiles, off, res0, tw, th)
    items = render.decode_items(d, th, tw, rec)
    dev = torch.device("cuda")
    s = {"lib": _lib.lib_for_device(0), "n": len(d), "n_items": len(items), "h": th, "w": tw,
         "descs": torch.from_numpy(d.view(np.uint8)).to(dev), "items": torch.from_numpy(items).to(dev),
         "prims": torch.from_numpy(rec.view(np.uint8)).to(dev), "res1": None, "n_res1": 0,
         "out": torch.zeros((th, tw, 3), dtype=torch.float32, device=dev)}
    if res1 is not None:
        s["res1"] = torch.from_numpy(res1.astype(np.float32) / np.float32(255.0)).to(dev)
        s["n_res1"] = len(res1)
    return s, tiles


def _walk(s):
    _lib.check(s["lib"].weftk_render_tiles(_lib.ptr(s["descs"]), s["n"], _lib.ptr(s["items"]), s["n_items"],
                                           _lib.ptr(s["prims"]), 0, 0, _lib.ptr(s["res1"]), s["n_res1"],
                                           _lib.ptr(s["out"]), s["h"], s["w"], 0,
                                           torch.cuda.current_stream().cuda_stream), "weftk_render_tiles")
    return s["out"]


def _dct_block(tiles, seed):
    """A DCT residual layer in the reference encoder's default form: every tile, YCbCr 4:2:0, frequency
    weight 4, the q75 step, band-major for odd seeds and tile-major for even ones, Laplacian
    coefficients whose scale falls with frequency."""
    rng = np.random.default_rng(seed + 1)
    step = float(max(0.003, min(0.20, 0.26 ** 2 * 0.20)))
    layout = seed & 1
    blocks = {}
    for s in np.unique(tiles[:, 2]):
        m = int((tiles[:, 2] == s).sum())
        for c in range(3):
            n = int(s) if c == 0 else int(s) // 2
            f = np.arange(n, dtype=np.float64)
            scale = 6.0 / (1.0 + f[:, None] + f[None, :])
            v = np.round(rng.exponential(1.0, (m, n, n)) * scale * rng.choice([-1.0, 1.0], (m, n, n)))
            blocks[int(s), c] = np.clip(v, -32768, 32767).astype(np.int16)
    if layout == 0:
        at = {s: 0 for s in np.unique(tiles[:, 2]).tolist()}
        parts = []
        for s in tiles[:, 2].tolist():
            parts += [blocks[s, c][at[s]].reshape(-1) for c in range(3)]
            at[s] += 1
    else:
        parts = []
        for s in sorted(at for at, c in blocks if c == 0):
            for c in range(3):
                b = blocks[s, c]
                parts.append(b.reshape(len(b), -1)[:, _zigzag(b.shape[1])].T.reshape(-1))
    return raster.DctBlock(np.concatenate(parts), step, 3, 4.0, 2,
                           np.packbits(np.ones(len(tiles), np.uint8), bitorder="little").tobytes(), len(tiles),
                           layout, b""), blocks


def _zigzag(n):
    """Row-major index of each zigzag position: anti-diagonals, rows descending on even ones."""
    out = []
    for s in range(2 * n - 1):
        rows = range(max(0, s - n + 1), min(s, n - 1) + 1)
        out += [u * n + s - u for u in (reversed(rows) if s % 2 == 0 else rows)]
    return np.array(out)


def _stacks(case, seed):
    """Random stacks of 1 .. layers primitives of every kind over an image's tiles."""
    rng = np.random.default_rng(seed)
    tiles, src4, px_off = _tile_set(case, seed)
    sides = tiles[:, 2]
    counts = np.random.default_rng(len(tiles)).integers(1, case["layers"] + 1, len(tiles))
    off = np.concatenate([[0], np.cumsum(counts)])
    tile = np.repeat(np.arange(len(tiles)), counts)
    kinds = rng.integers(0, 5, len(tile)).astype(np.int32)
    n = len(tile)
    rows = np.zeros((n, 16), np.float32)
    top = np.minimum(sides[tile] - 1.0, 14.5)[:, None]
    used = np.array([0, 4, 4, 6, 6])[kinds]
    rows[:, :7] = np.where(np.arange(7) < used[:, None], 1.0 + rng.random((n, 7)) * (top - 1.0), 0.0)
    thick = rng.uniform(0.7, 3.5, n)
    rows[:, 4] = np.where(kinds == 2, thick, rows[:, 4])
    rows[:, 6] = np.where(kinds == 3, thick, rows[:, 6])
    rows[:, 7:10] = rng.uniform(0.05, 0.95, (n, 3))
    rows[:, 10:13] = np.where(kinds[:, None] == 1, rng.uniform(0.05, 0.95, (n, 3)), 0.0)
    rows[:, 13] = rng.uniform(0.15, 0.9, n)
    ss = StackSet(src4, px_off, torch.from_numpy(sides.astype(np.int32)).cuda(), off, kinds, sizes_host=sides)
    return ss, torch.from_numpy(rows).cuda(), tiles, src4, off, kinds


def _full_pools(sides, src4, px_off, quality, seed):
    """Constant and linear candidates of the device generator, then lines, curves and triangles as the
    reference's templates place them (axis-parallel and diagonal lines in five thicknesses, arcs through
    the tile, corner and diagonal triangles), around each tile's own colours."""
    rng = np.random.default_rng(seed + 2)
    dev, n, stride = src4.device, len(sides), pools.MAX_CONST_LINEAR
    cand = torch.zeros(n * stride * PRIM_DTYPE.itemsize, dtype=torch.uint8, device=dev)
    cnt = torch.zeros(n, dtype=torch.int32, device=dev)
    p_off = torch.arange(n, dtype=torch.int32, device=dev) * stride
    pools.generate_pools(src4, px_off, sides, p_off, cand, cnt, quality)
    first = cand.cpu().numpy().view(PRIM_DTYPE).reshape(n, stride)
    c1 = cnt.cpu().numpy().astype(np.int64)
    more = np.array(POOL[2:])
    m = int(more.sum())
    kinds = np.tile(np.repeat([2, 3, 4], more), (n, 1)).reshape(-1)
    tile = np.repeat(np.arange(n), m)
    colours = np.repeat(_tile_colours(rng, src4, px_off, sides)[:, None], m, 1).reshape(-1, 3)
    rec = _primitives(rng, kinds, sides[tile], colours)
    top = (sides - 1.0)[tile]
    f = rng.choice([0.0, 0.25, 0.5, 0.75, 1.0], (len(tile), 6))
    rnd = rng.random((len(tile), 6))
    grid = np.where(rng.random((len(tile), 1)) < 0.6, f, rnd) * top[:, None]
    rec["geom"][:, :4] = grid[:, :4]
    rec["geom"][:, 4:6] = np.where(kinds[:, None] == 2, rec["geom"][:, 4:6], grid[:, 4:6])
    rec["alpha"] = np.where(kinds == 4, rng.choice([0.6, 0.5, 0.3], len(tile)), rec["alpha"])
    rec = rec.reshape(n, m)
    both = np.concatenate([first, rec], 1)
    keep = np.concatenate([np.arange(stride) < c1[:, None], np.ones((n, m), bool)], 1)
    return both[keep], c1 + m


# --------------------------------------------------------------------------------------- prepare / run
def prepare(case, seed):
    path = case["path"]
    s = {"path": path}
    if path == "image":
        s["pin"] = torch.from_numpy(_image(case, seed)).pin_memory()
        s["u8"], s["quality"], s["steps"] = s["pin"].numpy(), case["quality"], case["steps"]
        # the caller's own arrays, for as many tiles as the image can have
        most = -(-case["w"] // 64) * -(-case["h"] // 64) * 64
        s["own"] = (np.zeros((most, 3), np.int32), np.zeros((most, 16), np.float32), np.zeros(most, np.int32))
    elif path == "device":
        tiles, src4, _ = _tile_set(case, seed)
        s["fit"] = pools.DeviceRefinedFit(src4, tiles[:, 2], case["quality"], caps=[16] * len(tiles),
                                          steps=case["steps"], autotune=False)
    elif path == "plain":
        tiles, src4, px_off = _tile_set(case, seed)
        sides = tiles[:, 2]
        rec, cnt = _full_pools(sides, src4, px_off, case["quality"], seed)
        fit = BatchedFit.from_arrays(src4[:, :3].cpu().numpy(), sides, rec, cnt, case["quality"],
                                     caps=[16] * len(tiles))
        s["graph"] = fit.graph()
    elif path == "grad":
        s["ss"], rows, *_ = _stacks(case, seed)
        s["p"] = rows.requires_grad_(True)
        s["residual"] = case["residual"]
    elif path == "refine":
        ss, s["rows"], *_ = _stacks(case, seed)
        s["refiner"] = FusedRefiner(ss, s["rows"], lr=1e-2, residual=case["residual"])
        s["steps"] = case["steps"]
    elif path == "walk":
        s["walk"], _ = _walk_state(case, seed, case["tw"], case["th"])
    elif path == "raster":
        s["walk"], tiles = _walk_state(case, seed, case["w"], case["h"])
        s["dct"] = raster.DctLaunch(_dct_block(tiles, seed)[0], tiles.tolist(), case["w"], case["h"])
        s["tw"], s["th"] = case["tw"], case["th"]
    elif path == "decode":
        tiles, rec, off, res0, res1 = _scene(case, seed)
        prims = unpack_cands(rec)
        qt = [QuadTile(*t) for t in tiles.tolist()]
        s["blob"] = bitstream.encode_weft(
            case["w"], case["h"], 75, qt, [prims[a:b] for a, b in zip(off[:-1], off[1:])],
            residuals=None if res0 is None else res0.tolist(),
            res1_maps=None if res1 is None else list(res1.reshape(-1, 4, 4, 3)))
        s["tw"], s["th"] = case["tw"], case["th"]
    else:
        s["args"] = _score_inputs(case, seed)[:6]
    return s


def _score_inputs(case, seed):
    """What the reference's fit hands its scorer in one round: per tile the selected stack with each
    candidate on top, the pool's mix of kinds."""
    rng = np.random.default_rng(seed)
    u8 = synth.make_image_u8(256, 256, 40, seed)
    img = synth.srgb_u8_to_linear(u8)
    n, m, depth = case["tiles"], case["evals"], case["depth"]
    sides = rng.choice([8, 8, 8, 8, 16, 16, 32], n)
    x, y = (rng.integers(0, 256 - sides + 1) for _ in range(2))
    patches = [img[b:b + s, a:a + s] for a, b, s in zip(x.tolist(), y.tolist(), sides.tolist())]
    flat = np.concatenate([p.reshape(-1) for p in patches])
    p_off = np.concatenate([[0], np.cumsum(3 * sides.astype(np.int64) ** 2)])
    base = np.stack([p.mean((0, 1)) for p in patches]).astype(np.float64)
    pick = rng.choice(5, (n, m), p=np.array(POOL) / sum(POOL))
    kinds = np.concatenate([np.zeros((n, m, depth - 1), np.int64), pick[..., None]], 2).reshape(-1)
    tile = np.repeat(np.arange(n), m * depth)
    rec = _primitives(rng, kinds, sides[tile], base[tile]).reshape(n, m * depth)
    return (flat, {i: int(o) for i, o in enumerate(p_off[:-1])}, list(range(n)), sides.tolist(), list(rec),
            [[depth] * m] * n, sides, patches)


def run(s):
    path = s["path"]
    if path == "image":
        for own, got in zip(s["own"], frontend.refine_image(s["u8"], s["quality"], 16, s["steps"])):
            own[:len(got)] = got
        return s["own"]
    if path == "device":
        rows = s["fit"].run()
        return rows, s["fit"].rf.kinds
    if path == "plain":
        f = s["graph"].replay()
        return {"sel": f.t_sel, "n_sel": f.t_n_sel, "rows": f.t_qrows, "kinds": f.t_qkind, "composite": f.t_bg}
    if path == "grad":
        p = s["p"]
        p.grad = None
        loss = StackLoss.apply(p, s["ss"], False, s["residual"])
        (loss * s["ss"].weights).sum().backward()
        return loss.detach(), p.grad
    if path == "refine":
        r = s["refiner"]
        r.restart(s["rows"])
        return r.run(s["steps"]), r.loss
    if path == "walk":
        return _walk(s["walk"])
    if path == "raster":
        img = _walk(s["walk"])
        s["dct"].run(img, torch.cuda.current_stream().cuda_stream)
        return raster.resize(img, s["tw"], s["th"])
    if path == "decode":
        return encode.decode_file(s["blob"], s["tw"], s["th"])
    return np.concatenate(gpu_render.gpu_batch_score_prepacked(*s["args"]))


# --------------------------------------------------------------------------------------- work
def work(case):
    """Every input once in, every output once out; for the scored and rendered paths the operations of
    each candidate or layer over its pixels once."""
    path = case["path"]
    if path == "score":
        px = 190.0
        evals = case["tiles"] * case["evals"]
        ops = sum(p * k for p, k in zip(POOL, KIND_OPS)) / sum(POOL)
        return {"bytes": case["tiles"] * px * 12 + evals * (60 * case["depth"] + 4),
                "flops": evals * px * (ops + 9 + 10 * (case["depth"] - 1))}
    px = float(case["w"] * case["h"])
    n = px / TILE_PX
    if path == "image":
        return {"bytes": px * 3 + n * 80, "flops": n * 64 * 110}
    if path == "device":
        return {"bytes": px * 16 + n * 68, "flops": n * 64 * 110}
    if path == "plain":
        return {"bytes": px * 32 + n * (60 * sum(POOL) + 16 * 72),
                "flops": px * sum(p * (k + 9) for p, k in zip(POOL, KIND_OPS))}
    layers = n * (1 + case.get("layers", 1)) / 2
    if path in ("grad", "refine"):
        ops = sum(KIND_OPS) / 5 + 60
        return {"bytes": px * 16 + layers * 64 * 2, "flops": px * (1 + case["layers"]) / 2 * ops * case.get("steps", 1)}
    out = float(case["tw"] * case["th"])
    scene = n * (48 + 60) * 1.06 + (n * 192 if case["residuals"] else 0)
    if path == "walk":
        return {"bytes": out * 12 + scene, "flops": out * 10}
    if path == "raster":
        same = (case["tw"], case["th"]) == (case["w"], case["h"])
        return {"bytes": px * 3 + scene + out * 12, "flops": px * 1.5 * 4 * 10 + (0 if same else out * 3 * 4)}
    return {"bytes": n * 12 + (n * 51 if case["residuals"] else 0) + out * 12, "flops": out * 10}


# --------------------------------------------------------------------------------------- 64-bit values
def _coverage(kind, g, x, y, soft):
    """Coverage and colour-ramp position of primitives of one kind at points (float64)."""
    def seg(ax, ay, bx, by):
        vx, vy = bx - ax, by - ay
        t = (((x - ax) * vx + (y - ay) * vy) / (vx * vx + vy * vy + 1e-8)).clamp(0.0, 1.0)
        ex, ey = x - ax - t * vx, y - ay - t * vy
        return ex * ex + ey * ey

    if kind == 2:
        return torch.exp(-seg(g[0], g[1], g[2], g[3]) / (2 * g[4].clamp(min=0.5) ** 2))
    if kind == 3:
        ts = np.linspace(0, 1, 32, dtype=np.float32).astype(np.float64)
        pts = [((1 - t) ** 2 * g[0] + 2 * (1 - t) * t * g[2] + t * t * g[4],
                (1 - t) ** 2 * g[1] + 2 * (1 - t) * t * g[3] + t * t * g[5]) for t in ts]
        best = seg(*pts[0], *pts[1])
        for j in range(1, 31):
            best = torch.minimum(best, seg(*pts[j], *pts[j + 1]))
        return torch.exp(-best / (2 * g[6].clamp(min=0.5) ** 2))
    den = (g[3] - g[5]) * (g[0] - g[4]) + (g[4] - g[2]) * (g[1] - g[5])
    a = ((g[3] - g[5]) * (x - g[4]) + (g[4] - g[2]) * (y - g[5])) / den
    b = ((g[5] - g[1]) * (x - g[4]) + (g[0] - g[4]) * (y - g[5])) / den
    hard = ((a >= 0) & (b >= 0) & (1 - a - b >= 0) & (den.abs() >= 1e-6)).to(F64).detach()
    if not soft:
        return hard
    vx, vy = [g[0], g[2], g[4]], [g[1], g[3], g[5]]
    o = torch.where((vx[1] - vx[0]) * (vy[2] - vy[0]) - (vy[1] - vy[0]) * (vx[2] - vx[0]) >= 0, 1.0, -1.0)
    cov = 1.0
    for i in range(3):
        ia, ib = (i + 1) % 3, (i + 2) % 3
        ex, ey = vx[ib] - vx[ia], vy[ib] - vy[ia]
        sd = o * (ex * (y - vy[ia]) - ey * (x - vx[ia])) / (torch.sqrt(ex * ex + ey * ey) + 1e-12)
        cov = cov * torch.sigmoid(sd / 0.5)
    return hard + cov - cov.detach()  # the backward's surrogate


def _composite(rows, kinds, first, count, owner, x, y, soft=False):
    """Stacks over black at points: ``owner`` names each point's stack (float64, (n, 3))."""
    c = torch.zeros((len(x), 3), dtype=F64, device=x.device)
    for k in range(int(count.max()) if len(count) else 0):
        at = torch.nonzero(count[owner] > k).flatten()
        row = first[owner[at]] + k
        kk = kinds[row]
        for kind in range(5):
            sel = torch.nonzero(kk == kind).flatten()
            if len(sel) == 0:
                continue
            i, r = at[sel], rows[row[sel]]
            g = [r[:, j] for j in range(7)]
            a, col = r[:, 13].clamp(0.0, 1.0), r[:, 7:10]
            if kind == 1:
                vx, vy = g[2] - g[0], g[3] - g[1]
                t = (((x[i] - g[0]) * vx + (y[i] - g[1]) * vy) / (vx * vx + vy * vy + 1e-8)).clamp(0.0, 1.0)[:, None]
                col = col * (1 - t) + r[:, 10:13] * t
            elif kind > 1:
                a = a * _coverage(kind, g, x[i], y[i], soft)
            a = a[:, None]
            c = c.index_copy(0, i, col * a + c[i] * (1 - a))
    return c


def _rows64(rec):
    rows = np.zeros((len(rec), 16))
    rows[:, :7], rows[:, 7:10], rows[:, 10:13], rows[:, 13] = rec["geom"], rec["color0"], rec["color1"], rec["alpha"]
    return torch.from_numpy(rows).cuda()


def _grid_axis(p, n):
    g = ((p + 0.5) * 4.0 / n - 0.5).clamp(0.0, 3.0)
    lo = g.floor()
    return lo.long(), (lo + 1).clamp(max=3).long(), g - lo


def _exact_walk(case, seed, tw, th, scene=None):
    """The decoder's image in float64; pixels in rows of tiles, so memory stays bounded."""
    tiles, rec, off, res0, res1 = scene or _scene(case, seed)
    d = _descs(case, tiles, off, res0, tw, th)
    rows, kinds = _rows64(rec), torch.from_numpy(rec["kind"].astype(np.int64)).cuda()
    first, count = torch.from_numpy(off[:-1]).cuda(), torch.from_numpy(np.diff(off)).cuda()
    own = np.full((th, tw), -1, np.int64)
    for i, (a, b, w, h) in enumerate(zip(*(d[k].tolist() for k in ("target_x0", "target_y0", "target_w", "target_h")))):
        own[b:b + h, a:a + w] = i
    out = torch.zeros((th, tw, 3), dtype=F64, device="cuda")
    side = torch.from_numpy(np.maximum(d["target_w"], d["target_h"]).astype(np.float64)).cuda()
    step = torch.from_numpy(d["source_size"].astype(np.float64)).cuda() / side
    x0, y0 = (torch.from_numpy(d[k].astype(np.float64)).cuda() for k in ("target_x0", "target_y0"))
    hh = torch.from_numpy(d["target_h"].astype(np.float64)).cuda()
    for ya in range(0, th, 256):
        o = torch.from_numpy(own[ya:ya + 256]).cuda()
        at = torch.nonzero(o >= 0)
        t = o[at[:, 0], at[:, 1]]
        lx, ly = at[:, 1].to(F64) - x0[t], (at[:, 0] + ya).to(F64) - y0[t]
        c = _composite(rows, kinds, first, count, t, (lx + 0.5) * step[t], (ly + 0.5) * step[t])
        if res0 is not None:
            c = (c + torch.from_numpy(res0 / 255.0).cuda()[t]).clamp(0.0, 1.0)
            grid = torch.from_numpy(res1.astype(np.float64) / 255.0).cuda().view(-1, 4, 4, 3)
            xa, xb, wx = _grid_axis(lx, hh[t])
            yl, yh, wy = _grid_axis(ly, hh[t])
            wx, wy = wx[:, None], wy[:, None]
            top = grid[t, yl, xa] * (1 - wx) + grid[t, yl, xb] * wx
            c = c + top * (1 - wy) + (grid[t, yh, xa] * (1 - wx) + grid[t, yh, xb] * wx) * wy
        out[at[:, 0] + ya, at[:, 1]] = c.clamp(0.0, 1.0)
    return out


def _exact_raster(case, seed):
    tw, th = case["w"], case["h"]
    scene = _scene(case, seed)
    tiles = scene[0]
    img = _exact_walk(case, seed, tw, th, scene)
    block, blocks = _dct_block(tiles, seed)
    pad = torch.zeros((th + 64, tw + 64, 3), dtype=F64, device="cuda")
    pad[:th, :tw] = img
    yuv = torch.tensor([[1.0, 0.0, 1.402], [1.0, -0.344136, -0.714136], [1.0, 1.772, 0.0]], dtype=F64, device="cuda")
    step32 = float(np.float32(block.quant_step))
    for s in np.unique(tiles[:, 2]).tolist():
        idx = np.flatnonzero(tiles[:, 2] == s)
        planes = []
        for c in range(3):
            n = s if c == 0 else s // 2
            k = torch.arange(n, dtype=F64, device="cuda")
            basis = torch.cos(math.pi * (2 * k[None, :] + 1) * k[:, None] / (2 * n)) * math.sqrt(2.0 / n)
            basis[0] = math.sqrt(1.0 / n)
            q = torch.from_numpy(blocks[s, c].astype(np.float64)).cuda()
            q = q * (step32 * (1.5 if c else 1.0)) * (1.0 + 4.0 * (k[:, None] + k[None, :]) / (2.0 * (n - 1)))
            v = basis.T @ q @ basis
            planes.append(v if c == 0 else v.repeat_interleave(2, 1).repeat_interleave(2, 2))
        rgb = torch.stack(planes, -1) @ yuv.T
        ys = torch.from_numpy(tiles[idx, 1].astype(np.int64)).cuda()[:, None] + torch.arange(s, device="cuda")
        xs = torch.from_numpy(tiles[idx, 0].astype(np.int64)).cuda()[:, None] + torch.arange(s, device="cuda")
        pad[ys[:, :, None], xs[:, None, :]] += rgb
    img = pad[:th, :tw].clamp(0.0, 1.0)
    if (case["tw"], case["th"]) == (tw, th):
        return img
    u8 = (img.to(torch.float32) * 255.0).clamp(0.0, 255.0).to(torch.int64)

    def taps(n_in, n_out):
        """Pillow's triangle filter: a dense (n_out, n_in) matrix of 22-bit integer weights."""
        scale = n_in / n_out
        fs = max(scale, 1.0)
        m = np.zeros((n_out, n_in))
        for o in range(n_out):
            centre = (o + 0.5) * scale
            lo, hi = max(0, int(centre - fs + 0.5)), min(n_in, int(centre + fs + 0.5))
            w = [max(0.0, 1.0 - abs((p - centre + 0.5) * (1.0 / fs))) for p in range(lo, hi)]
            total = 0.0
            for v in w:
                total += v
            m[o, lo:hi] = [int(0.5 + v / total * (1 << 22)) for v in w]
        return torch.from_numpy(m).cuda()

    def apply(m, v):  # integers below 2^53: exact in float64
        return torch.floor((m @ v + (1 << 21)) / (1 << 22)).clamp(0.0, 255.0)

    v = apply(taps(tw, case["tw"]), u8.to(F64).permute(1, 0, 2).reshape(tw, -1)).view(case["tw"], th, 3)
    v = apply(taps(th, case["th"]), v.permute(1, 0, 2).reshape(th, -1)).view(case["th"], case["tw"], 3)
    return v / 255.0


def _exact_loss(rows, tiles, src4, off, kinds, residual):
    """Per-tile losses in float64, differentiable in ``rows``."""
    sides = tiles[:, 2].astype(np.int64)
    px = sides ** 2
    owner = torch.from_numpy(np.repeat(np.arange(len(px)), px)).cuda()
    local = torch.arange(int(px.sum()), device="cuda") - torch.from_numpy(np.cumsum(px) - px).cuda()[owner]
    side = torch.from_numpy(sides).cuda()[owner]
    x, y = (local % side).to(F64) + 0.5, (local // side).to(F64) + 0.5
    first, count = torch.from_numpy(off[:-1]).cuda(), torch.from_numpy(np.diff(off)).cuda()
    c = _composite(rows, torch.from_numpy(kinds.astype(np.int64)).cuda(), first, count, owner, x, y, True)
    e = c.clamp(0.0, 1.0) - src4[:, :3].to(F64)
    if residual:
        b = side // 4
        cell = (local // side) // b * 4 + (local % side) // b
        at = owner * 16 + cell
        m = torch.zeros((len(px) * 16, 3), dtype=F64, device="cuda").index_add(0, at, e / (b * b)[:, None].to(F64))
        xa, xb, wx = _grid_axis((local % side).to(F64), side.to(F64))
        ya, yb, wy = _grid_axis((local // side).to(F64), side.to(F64))
        wx, wy, o = wx[:, None], wy[:, None], owner * 16
        top = m[o + ya * 4 + xa] * (1 - wx) + m[o + ya * 4 + xb] * wx
        e = e - top * (1 - wy) - (m[o + yb * 4 + xa] * (1 - wx) + m[o + yb * 4 + xb] * wx) * wy
    n = torch.from_numpy(px.astype(np.float64)).cuda()
    return torch.zeros(len(px), dtype=F64, device="cuda").index_add(0, owner, (e * e).sum(1)) / (3.0 * n)


def exact(case, seed):
    path = case["path"]
    if path in ("image", "device", "plain"):
        return None  # a search: its outputs are the choices it makes
    if path == "walk":
        return _exact_walk(case, seed, case["tw"], case["th"])
    if path == "decode":
        scene = list(_scene(case, seed))
        rec = scene[1]
        rec["alpha"] = np.round(rec["alpha"].astype(np.float64) * 65535.0) / 65535.0
        thick = np.where(rec["kind"] == 2, 4, np.where(rec["kind"] == 3, 6, -1))[:, None] == np.arange(7)
        top = np.where(thick, 4.0, 15.0)
        rec["geom"] = np.round(np.clip(rec["geom"] / top, 0, 1) * 65535.0) / 65535.0 * top
        return _exact_walk(case, seed, case["tw"], case["th"], scene)
    if path == "raster":
        return _exact_raster(case, seed)
    if path == "score":
        *_, recs, counts, sides, patches = _score_inputs(case, seed)
        out = []
        for rec, cnt, s, patch in zip(recs, counts, sides.tolist(), patches):
            m, depth = len(cnt), cnt[0]
            owner = torch.arange(m, device="cuda").repeat_interleave(s * s)
            p = torch.arange(s * s, device="cuda").repeat(m)
            c = _composite(_rows64(rec), torch.from_numpy(rec["kind"].astype(np.int64)).cuda(),
                           torch.arange(m, device="cuda") * depth, torch.full((m,), depth, device="cuda"), owner,
                           (p % s).to(F64) + 0.5, (p // s).to(F64) + 0.5)
            e = c.clamp(0.0, 1.0).view(m, -1) - torch.from_numpy(patch.astype(np.float64)).cuda().reshape(1, -1)
            out.append((e * e).mean(1))
        return torch.cat(out)
    ss, rows, tiles, src4, off, kinds = _stacks(case, seed)
    weights = ss.weights.to(F64)
    p = rows.to(F64)
    if path == "grad":
        p.requires_grad_(True)
        loss = _exact_loss(p, tiles, src4, off, kinds, case["residual"])
        (loss * weights).sum().backward()
        return loss.detach(), p.grad
    # Adam with the projection onto the wire's ranges, as the refiner's steps
    k = torch.from_numpy(kinds).cuda()
    top = torch.ones((len(k), 16), dtype=F64, device="cuda")
    top[:, :7] = 15.0
    top[k == 2, 4] = 4.0
    top[k == 3, 6] = 4.0
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    p = torch.minimum(p.clamp(min=0.0), top)
    for t in range(1, case["steps"] + 1):
        q = p.clone().requires_grad_(True)
        loss = _exact_loss(q, tiles, src4, off, kinds, case["residual"])
        (g,) = torch.autograd.grad((loss * weights).sum(), q)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 1e-2 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
        p = torch.minimum(p.clamp(min=0.0), top)
    return p, loss.detach()
