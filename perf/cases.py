"""The calls a terrain program makes of this package on one GPU, as performance cases.

Each case is one public call (or one evaluation of a whole layer stack) on device memory: the
noise sources and layers, crater shaping, boulder relief, a whole stack, a batch of tiles, the
diamond-square refinement of a DEM and the seam chain of overlapping patches. `listed` gives the
cases, `draw` others of the same ranges, `prepare` a case's inputs, `run` one pass, `work` what a
pass cannot do without and `exact` its outputs in 64-bit arithmetic, restated here in torch.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from terraingen_b200 import Device
from terraingen_b200 import workloads as W
from terraingen_b200.batch import TILE, Batch, TileSet, layout
from terraingen_b200.chain import PatchChain, Seams, Window
from terraingen_b200.device import GridSpec, centered
from terraingen_b200.layouts import fractal, noise_layer_kernel

# Per square meter, the synthetic 4097^2 terrain's craters and boulders.
_AREA = (4097 * 0.5) ** 2
_CRATERS = 200000.0 / (_AREA * (1.0 ** -2.0 - 500.0 ** -2.0))
_BOULDERS = 1e6 / (_AREA * (0.2 ** -2.5 - 3.0 ** -2.5))


def listed():
    return [
        # A small preview or a collision patch around a rover: latency of one short call.
        dict(name="source_257", kind="source", width=257, height=257, pixel=0.5, octaves=8),
        # The synthetic terrain's source: an 8-octave fBm over a whole tile.
        dict(name="source_4097", kind="source", width=4097, height=4097, pixel=0.5, octaves=8),
        # A stack of differing fractals (bases, types, a warp, blends) added to a tile.
        dict(name="layer_1025", kind="layer", width=1025, height=1025, pixel=1.0, octaves=6),
        # A source on a sphere: a regional map in longitude and latitude.
        dict(name="body_1025", kind="body", width=1025, height=1025, pixel=5e-5, octaves=8),
        # A streamed tile's crater layer.
        dict(name="craters_513", kind="craters", width=513, height=513, pixel=0.5, profile=0,
             density=1.0),
        # The crater layer of a whole 4097^2 tile.
        dict(name="craters_4097", kind="craters", width=4097, height=4097, pixel=0.5, profile=0,
             density=1.0),
        # The benchmark's whole stack: source, craters with peaks and terraces, boulders.
        dict(name="terrain_4097", kind="terrain", width=4097, height=4097, pixel=0.5, octaves=8),
        # A batch of uneven tiles of the same stack, as a tile server's prefetch makes.
        dict(name="tiles_96", kind="tiles", tiles=96, low=65, high=1025, density=0.1),
        # A DEM refined tenfold (the refinement configuration's patch, halved).
        dict(name="refine_5121", kind="refine", width=5121, height=5121, pixel=0.5, posts=5.0,
             spline=False),
        # The Catmull-Rom refinement, a ragged window.
        dict(name="refine_spline_1411", kind="refine", width=1411, height=1187, pixel=0.625,
             posts=5.0, spline=True),
        # 2 x 2 patches of one DEM joined by Height seams.
        dict(name="seams_5121", kind="seams", side=5121, pixel=0.5, overlap=64, mode="height"),
        # The same where slopes must match too (the fourth-order seam).
        dict(name="seams_slope_2049", kind="seams", side=2049, pixel=0.5, overlap=64,
             mode="slope"),
    ]


def _side(rng, low, high):
    """A size spread over the logarithm of its range, odd more often than not."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return min(max(n + (1 - n % 2 if rng.random() < 0.7 else 0), low), high)


def draw(rng):
    kind = rng.choice(["source", "layer", "body", "craters", "boulders", "terrain", "tiles",
                       "refine", "seams"])
    if kind == "tiles":
        return dict(kind=kind, tiles=rng.randint(4, 96), low=rng.randint(33, 129),
                    high=rng.randint(257, 1025), density=rng.choice([0.05, 0.1]))
    if kind == "seams":
        mode = rng.choice(["height", "height", "slope", "feather"])
        return dict(kind=kind, side=_side(rng, 513, 2049 if mode == "slope" else 5121),
                    pixel=rng.choice([0.25, 0.5, 1.0]), overlap=rng.choice([32, 48, 64]),
                    mode=mode)
    high = {"layer": 2049, "body": 1537}.get(kind, 4097)
    width = _side(rng, 65, high)
    case = dict(kind=kind, width=width,
                height=min(max(65, int(width * rng.uniform(0.5, 2.0))), high))
    if kind == "body":
        return dict(case, pixel=rng.choice([1e-5, 5e-5, 1e-3]), octaves=rng.randint(4, 10))
    if kind == "refine":
        return dict(case, pixel=rng.choice([0.5, 0.625, 1.0, 2.5]), posts=5.0,
                    spline=rng.random() < 0.4)
    pixel = rng.choice([0.25, 0.5, 0.7, 1.0])
    if kind == "craters":
        return dict(case, pixel=pixel, profile=rng.choice([0, 0, 1]),
                    density=rng.choice([0.25, 1.0]) * (0.5 if pixel > 0.5 else 1.0))
    if kind == "boulders":
        return dict(case, pixel=min(pixel, 0.5), density=rng.choice([0.2, 1.0]))
    if kind == "terrain":
        return dict(case, pixel=min(pixel, 0.5), octaves=rng.randint(6, 8))
    return dict(case, pixel=pixel, octaves=rng.randint(4, 12 if kind == "source" else 8))


# --- inputs ------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _device():
    return Device(0)


def _grid(case, seed):
    """The case's grid somewhere within a kilometer or so of the origin."""
    r = np.random.default_rng([5, seed])
    cx, cy = (float(v) for v in np.round(r.uniform(-1000.0, 1000.0, 2)))
    return centered(case["width"], case["height"], case["pixel"], cx, cy)


def _bytes(array):
    return torch.from_numpy(np.ascontiguousarray(array).view(np.uint8).reshape(-1).copy()).cuda()


def _device_craters(batch):
    kernel, records, data, footprints = batch
    return (kernel, _bytes(records), torch.from_numpy(data).cuda(),
            torch.from_numpy(footprints).cuda())


def _base(grid, seed):
    """Rolling ground of a few meters, the heights beneath a layer."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    coarse = torch.randn((1, 1, grid.height // 48 + 4, grid.width // 48 + 4), generator=g,
                         device="cuda")
    return (3.0 * torch.nn.functional.interpolate(
        coarse, size=(grid.height, grid.width), mode="bicubic")[0, 0]).contiguous()


def _fractals(case, seed):
    if case["kind"] == "layer":
        o = case["octaves"]
        return [fractal(seed=seed + 1, wavelength=300.0, amplitude=20.0, octaves=o, type=1,
                        warp_amplitude=25.0, warp_wavelength=150.0),  # warped ridges
                fractal(seed=seed + 2, wavelength=120.0, amplitude=4.0, octaves=o, basis=1),
                fractal(seed=seed + 3, wavelength=60.0, amplitude=1.5, octaves=3, basis=2, type=2),
                fractal(seed=seed + 4, wavelength=80.0, amplitude=2.0, octaves=2, basis=3)]
    return [fractal(seed=seed + 7, wavelength=512.0, amplitude=5.0, octaves=case["octaves"])]


def _posts(case, seed):
    """A DEM of kilometers of relief covering the case's grid, and its grid."""
    ratio = case["pixel"] / case["posts"]
    w = int(math.ceil(case["width"] * ratio)) + 5
    h = int(math.ceil(case["height"] * ratio)) + 5
    grid = centered(w, h, case["posts"])
    r = torch.Generator(device="cuda").manual_seed(seed + 3)
    total = torch.zeros((h, w), device="cuda", dtype=torch.float64)
    for k in range(6):
        step = 2 ** (7 - k)
        coarse = torch.randn((1, 1, h // step + 4, w // step + 4), generator=r, device="cuda",
                             dtype=torch.float64)
        total += 400.0 * 0.5 ** k * torch.nn.functional.interpolate(coarse, size=(h, w),
                                                                   mode="bicubic")[0, 0]
    return total.float().contiguous(), grid


def _patches(case, seed):
    """Four overlapping surveys of one DEM that disagree by meters."""
    side, half = case["side"], case["side"] // 2
    lo, hi = half + case["overlap"] // 2, half - case["overlap"] // 2
    windows = [Window(0, 0, lo, lo), Window(hi, 0, side - hi, lo), Window(0, hi, lo, side - hi),
               Window(hi, hi, side - hi, side - hi)]
    g = torch.Generator(device="cuda").manual_seed(seed + 9)

    def ground(step, scale):
        n = side // step + 4
        coarse = torch.randn((1, 1, n, n), generator=g, device="cuda")
        return scale * torch.nn.functional.interpolate(coarse, size=(side, side),
                                                       mode="bicubic")[0, 0]

    common = ground(256, 100.0) + ground(32, 4.0)
    patches = [(common + ground(64, 2.0) + ground(4, 0.1))[w.slices()].contiguous()
               for w in windows]
    return windows, patches


def _tile_set(case, seed):
    """Uneven tiles (their sides and spacings the case's, their places and layers the seed's) of
    the synthetic terrain's stack, anywhere on a disk of 1700 km."""
    shapes = W.uneven_tile_grids(case["tiles"], (case["low"], case["high"]), (0.25, 2.0))
    r = np.random.default_rng([8, seed])
    far, turn = 1.7e6 * np.sqrt(r.random(len(shapes))), r.uniform(0.0, 2.0 * np.pi, len(shapes))
    grids = [centered(g.width, g.height, g.pixel, float(x), float(y))
             for g, x, y in zip(shapes, far * np.cos(turn), far * np.sin(turn))]
    craters = W.crater_population(seed + 1, case["density"] * _CRATERS, 1.0, 500.0)
    boulders = W.boulder_population(seed + 1, case["density"] * _BOULDERS)
    tiles = np.zeros(len(grids), TILE)
    tiles["height_offset"], tiles["pitch"] = layout(grids)
    batches = [W.crater_batch(craters, g) for g in grids]
    stones = [W.generate_boulders(boulders, g) for g in grids]
    for t, g in zip(tiles, grids):
        t["width"], t["height"], t["boulder_width"] = g.width, g.height, g.pixel
        t["origin_x"], t["pixel_width"] = g.x0, g.pixel
        t["origin_y"], t["pixel_height"] = g.y0, -g.pixel
    for name, counts in (("crater", [len(b[1]) for b in batches]),
                         ("boulder", [len(b) for b in stones])):
        tiles[name + "_count"] = counts
        tiles[name + "_begin"] = np.cumsum([0] + counts[:-1])
    tiles["data_begin"] = np.cumsum([0] + [len(b[2]) for b in batches[:-1]])
    return TileSet(tiles=tiles, fractals=np.array(_fractals(dict(case, octaves=8), seed)),
                   elevation=0.0, crater_kernel=batches[0][0],
                   crater_records=np.concatenate([b[1] for b in batches]),
                   crater_data=np.concatenate([b[2] for b in batches]),
                   crater_footprints=np.concatenate([b[3] for b in batches]),
                   boulders=np.concatenate(stones), grids=grids)


def prepare(case, seed):
    kind = case["kind"]
    device = _device()
    if kind == "tiles":
        tiles = _tile_set(case, seed)
        batch = Batch(device)
        batch.load(tiles)
        out = torch.zeros(tiles.output_floats, dtype=torch.float32, device="cuda")
        return dict(kind=kind, batch=batch, tiles=tiles, out=out)
    if kind == "seams":
        windows, patches = _patches(case, seed)
        grid = centered(case["side"], case["side"], case["pixel"])
        decay = case["overlap"] * case["pixel"] / 3.0
        seams = Seams(mode=case["mode"], width=3.0 * decay, decay_length=decay)
        return dict(kind=kind, chain=PatchChain(device, grid, windows, seams), windows=windows,
                    patches=patches, grid=grid)
    state = dict(kind=kind, device=device)
    if kind == "refine":
        posts, post_grid = _posts(case, seed)
        grid = centered(case["width"], case["height"], case["pixel"])
        state.update(posts=posts, post_grid=post_grid, seed=seed + 7, interp=int(case["spline"]))
    elif kind == "body":
        r = np.random.default_rng([6, seed])
        lon, lat = (float(v) for v in r.uniform([-170.0, -50.0], [170.0, 50.0]))
        grid = centered(case["width"], case["height"], case["pixel"], lon, lat)
    else:
        grid = _grid(case, seed)
    state.update(grid=grid, out=torch.zeros((grid.height, grid.width), dtype=torch.float32,
                                            device="cuda"))
    if kind in ("source", "body", "terrain"):
        state["fractals"] = np.array(_fractals(case, seed))
    if kind == "layer":
        state["kernel"] = noise_layer_kernel(_fractals(case, seed))
    if kind in ("layer", "craters", "boulders"):
        state["base"] = _base(grid, seed)
    if kind == "craters":
        state["host"] = W.crater_batch(W.crater_population(seed + 1, case["density"] * _CRATERS,
                                                           1.0, 500.0), grid,
                                       profile=case["profile"])
        state["craters"] = _device_craters(state["host"])
    if kind == "terrain":
        state["host"] = W.crater_batch(W.crater_population(seed + 1, _CRATERS, 1.0, 500.0), grid,
                                       shaping=W.config2_shaping())
        state["craters"] = _device_craters(state["host"])
    if kind in ("boulders", "terrain"):
        stones = W.generate_boulders(
            W.boulder_population(seed + 1, case.get("density", 1.0) * _BOULDERS), grid)
        state["boulders"] = torch.from_numpy(stones).cuda()
    return state


def run(state):
    kind = state["kind"]
    if kind == "tiles":
        state["batch"].evaluate(state["out"])
        return state["out"]
    if kind == "seams":
        return state["chain"].compose(state["patches"])
    device, grid, out = state["device"], state["grid"], state["out"]
    if kind == "source":
        return device.noise_source(state["fractals"], grid, out)
    if kind == "body":
        return device.noise_source_body(state["fractals"], grid, 1737400.0, out)
    if kind == "refine":
        return device.ds_refine(state["posts"], state["post_grid"], grid, out, 2.2, 1.5,
                                seed=state["seed"], interp=state["interp"])
    if kind == "terrain":
        return device.evaluate(grid, out, fractals=state["fractals"], craters=state["craters"],
                               boulders=state["boulders"], boulder_width=grid.pixel)
    out.copy_(state["base"])
    if kind == "layer":
        return device.noise_layer(state["kernel"], grid, out)
    if kind == "craters":
        kernel, records, data, footprints = state["craters"]
        return device.craters_apply(kernel, records, data, grid, out, footprints)
    return device.boulders_bake(state["boulders"], grid, out, grid.pixel)


# Operations a pass cannot do without: a Perlin octave at one cell (turn, lattice position,
# fades, four gradients, interpolation), a crater or a boulder at a cell it reaches, a
# diamond-square node (its draw and mean), an unknown's share of a seam solve.
_OCTAVE, _OCTAVE3, _CRATER, _BOULDER, _NODE, _UNKNOWN = 60.0, 140.0, 105.0, 80.0, 60.0, 400.0


def work(case):
    kind = case["kind"]
    if kind == "tiles":
        n, lo, hi = case["tiles"], case["low"], case["high"] + 1
        cells = n * (hi ** 2 - lo ** 2) / (2.0 * math.log(hi / lo))
        return dict(bytes=4.0 * cells, flops=cells * (8 * _OCTAVE + 5.0 * case["density"] * _CRATER))
    if kind == "seams":
        side, overlap = case["side"], case["overlap"]
        # Each patch read, the heights written; three seams' bands solved.
        return dict(bytes=8.0 * side * side, flops=3.0 * side * overlap * _UNKNOWN)
    cells = float(case["width"] * case["height"])
    area = cells * case["pixel"] ** 2
    if kind == "refine":
        posts = cells * (case["pixel"] / case["posts"]) ** 2
        levels = max(0, math.ceil(math.log2(case["posts"] / case["pixel"]) - 1e-9))
        return dict(bytes=4.0 * cells + 4.0 * posts, flops=posts * (4.0 ** levels) * _NODE)
    # Craters of N(>D) ~ c D^-2 within 1.5 radii: pairs per cell = 2 c pi 0.75^2 ln(dmax / dmin).
    craters = case.get("density", 1.0) * _CRATERS * area
    boulders = case.get("density", 1.0) * _BOULDERS * area * 2.0 ** -2.5
    reach = 2.0 * case.get("density", 1.0) * _CRATERS * math.pi * 0.75 ** 2 * math.log(500.0)
    if kind == "source":
        return dict(bytes=4.0 * cells, flops=cells * case["octaves"] * _OCTAVE)
    if kind == "body":
        return dict(bytes=4.0 * cells, flops=cells * case["octaves"] * _OCTAVE3)
    if kind == "layer":
        octaves = 8 + 2 * case["octaves"] + 3 + 2 * 4  # two warps; a Worley octave is four or so
        return dict(bytes=8.0 * cells, flops=cells * octaves * _OCTAVE)
    if kind == "craters":
        return dict(bytes=8.0 * cells + 300.0 * craters, flops=cells * reach * _CRATER)
    if kind == "boulders":
        return dict(bytes=8.0 * cells + 40.0 * boulders, flops=cells * 0.2 * _BOULDER)
    return dict(bytes=4.0 * cells + 300.0 * craters + 40.0 * boulders,
                flops=cells * (case["octaves"] * _OCTAVE + reach * _CRATER + 0.2 * _BOULDER))


# --- the same in 64 bits -----------------------------------------------------------------------

_M = 0xFFFFFFFF
# The planar turn between octaves is defined by its single-precision constants.
_TURN = (float(np.float32(-0.7373688780783197)), float(np.float32(0.6754902942615238)))
_TURN3 = torch.tensor([[-0.6132711010727254, -0.293401570821183, 0.7333580809050306],
                       [0.7897926788435601, -0.24097777005594262, 0.5640542870894418],
                       [0.011228581128535142, 0.9251190369776896, 0.37951111497202883]],
                      dtype=torch.float64)


def _pcg(v):
    state = (v * 747796405 + 2891336453) & _M
    word = (((state >> ((state >> 28) + 4)) ^ state) * 277803737) & _M
    return (word >> 22) ^ word


def _pcg3d(x, y, z):
    x, y, z = ((v * 1664525 + 1013904223) & _M for v in (x, y, z))
    x = (x + y * z) & _M
    y = (y + z * x) & _M
    z = (z + x * y) & _M
    x, y, z = x ^ (x >> 16), y ^ (y >> 16), z ^ (z >> 16)
    x = (x + y * z) & _M
    y = (y + z * x) & _M
    z = (z + x * y) & _M
    return x, y, z


def _unit(h):
    return (h >> 8) * 2.0 ** -24


def _fade(t):
    return t * t * t * (t * (t * 6.0 - 15.0) + 10.0)


def _lerp(t, a, b):
    return a + t * (b - a)


def _gradient2(h, x, y):
    h = h & 7
    axis = torch.where((h & 2) != 0, y, x)
    axis = torch.where((h & 1) != 0, -axis, axis)
    both = torch.where(h == 5, -x, x) + torch.where(h == 6, -y, y)
    return torch.where(h < 4, axis, torch.where(h == 7, -both, both) * math.sqrt(0.5))


def _perlin2(x, y, seed):
    cx, cy = torch.floor(x), torch.floor(y)
    fx, fy = x - cx, y - cy
    ix, iy = cx.long() & _M, cy.long() & _M

    def corner(dx, dy):
        return _gradient2(_pcg3d((ix + dx) & _M, (iy + dy) & _M, seed)[0], fx - dx, fy - dy)

    u, v = _fade(fx), _fade(fy)
    return math.sqrt(2.0) * _lerp(v, _lerp(u, corner(0, 0), corner(1, 0)),
                                  _lerp(u, corner(0, 1), corner(1, 1)))


def _simplex2(x, y, seed):
    skew, unskew = (math.sqrt(3.0) - 1.0) / 2.0, (3.0 - math.sqrt(3.0)) / 6.0
    s = (x + y) * skew
    cx, cy = torch.floor(x + s), torch.floor(y + s)
    u = (cx + cy) * unskew
    x0, y0 = x - (cx - u), y - (cy - u)
    stepx = (x0 > y0).double()
    stepy = 1.0 - stepx
    i, j = cx.long() & _M, cy.long() & _M

    def corner(di, dj, dx, dy):
        t = 0.5 - dx * dx - dy * dy
        h = _pcg3d((i + di) & _M, (j + dj) & _M, seed)[0]
        return torch.where(t <= 0.0, 0.0, t ** 4 * _gradient2(h, dx, dy))

    return 99.0 * (corner(0, 0, x0, y0) +
                   corner(stepx.long(), stepy.long(), x0 - stepx + unskew, y0 - stepy + unskew) +
                   corner(1, 1, x0 - 1.0 + 2.0 * unskew, y0 - 1.0 + 2.0 * unskew))


def _value2(x, y, seed):
    cx, cy = torch.floor(x), torch.floor(y)
    ix, iy = cx.long() & _M, cy.long() & _M

    def corner(dx, dy):
        return 2.0 * _unit(_pcg3d((ix + dx) & _M, (iy + dy) & _M, seed)[1]) - 1.0

    u, v = _fade(x - cx), _fade(y - cy)
    return _lerp(v, _lerp(u, corner(0, 0), corner(1, 0)), _lerp(u, corner(0, 1), corner(1, 1)))


def _worley_f1(x, y, seed):
    cx, cy = torch.floor(x), torch.floor(y)
    ix, iy, fx, fy = cx.long(), cy.long(), x - cx, y - cy
    best = torch.full_like(x, 1e30)
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            _, h1, h2 = _pcg3d((ix + dx) & _M, (iy + dy) & _M, seed)
            best = torch.minimum(best, (dx + _unit(h1) - fx) ** 2 + (dy + _unit(h2) - fy) ** 2)
    return 2.0 * torch.clamp(torch.sqrt(best) * math.sqrt(0.5), max=1.0) - 1.0


_BASES = {0: _perlin2, 1: _simplex2, 2: _value2, 3: _worley_f1}


def _fractal2(x, y, seed, wavelength, octaves, gain=0.5, lacunarity=2.0, basis=0, type=0,
              offset=1.0):
    """The octave sum at (x, y); `seed` a number or a tensor of x's shape."""
    frequency, c, s = 1.0 / wavelength, 1.0, 0.0
    weight, total, feedback = 1.0, 0.0, torch.ones_like(x)
    out = torch.zeros_like(x)
    for o in range(octaves):
        h, h1, h2 = _pcg3d(seed, o, 0)
        n = _BASES[basis]((x * c - y * s) * frequency + _unit(h1),
                          (x * s + y * c) * frequency + _unit(h2), h)
        if type == 1:  # ridged
            signal = (offset - n.abs()) ** 2 * feedback
            feedback = torch.clamp(2.0 * signal, 0.0, 1.0)
            out = out + weight * signal
        elif type == 2:  # billow
            out = out + weight * (2.0 * n.abs() - 1.0)
        else:
            out = out + weight * n
        total += weight
        weight *= gain
        frequency *= lacunarity
        c, s = c * _TURN[0] - s * _TURN[1], s * _TURN[0] + c * _TURN[1]
    if type == 1:
        ridge = max(offset, 1.0 - offset)
        return 2.0 * out / (ridge * ridge * total) - 1.0
    return out / total


def _stack2(fractals, x, y):
    """A stack of enabled, added fractals."""
    height = torch.zeros_like(x)
    for f in fractals:
        px, py = x, y
        if float(f["warpAmplitude"]) > 0.0:
            seed = _pcg(int(f["seed"]) ^ 0x5BD1E995)
            wave, amp = float(f["warpWavelength"]), float(f["warpAmplitude"])
            px = x + amp * _fractal2(x, y, seed, wave, 4)
            py = y + amp * _fractal2(x, y, _pcg(seed), wave, 4)
        height = height + float(f["amplitude"]) * _fractal2(
            px, py, int(f["seed"]), float(f["wavelength"]), int(f["octaves"]), float(f["gain"]),
            float(f["lacunarity"]), int(f["basis"]), int(f["type"]), float(f["offset"]))
    return height


def _axes(grid):
    c = torch.arange(grid.width, device="cuda", dtype=torch.float64)
    r = torch.arange(grid.height, device="cuda", dtype=torch.float64)
    return grid.x0 + (c + 0.5) * grid.pixel, grid.y0 - (r + 0.5) * grid.pixel


def _by_rows(grid, at):
    """`at`(xs, ys) over the grid's cells, some rows at a time."""
    xs, ys = _axes(grid)
    rows = max(1, (1 << 21) // grid.width)
    return torch.cat([at(*torch.broadcast_tensors(xs[None, :], ys[k:k + rows, None]))
                      for k in range(0, grid.height, rows)])


def _perlin3(x, y, z, seed):
    c = [torch.floor(v) for v in (x, y, z)]
    f = [v - w for v, w in zip((x, y, z), c)]
    i = [v.long() for v in c]
    key = _pcg(seed)
    corners = []
    for n in range(8):
        d = (n & 1, (n >> 1) & 1, n >> 2)
        h = _pcg3d((i[0] + d[0]) & _M, (i[1] + d[1]) & _M, (i[2] + d[2] + key) & _M)[0] & 15
        gx, gy, gz = (a - b for a, b in zip(f, d))
        u = torch.where(h < 8, gx, gy)
        v = torch.where(h < 4, gy, torch.where((h == 12) | (h == 14), gx, gz))
        corners.append(torch.where((h & 1) == 0, u, -u) + torch.where((h & 2) == 0, v, -v))
    u, v, w = (_fade(t) for t in f)
    near = _lerp(v, _lerp(u, corners[0], corners[1]), _lerp(u, corners[2], corners[3]))
    far = _lerp(v, _lerp(u, corners[4], corners[5]), _lerp(u, corners[6], corners[7]))
    return torch.clamp(_lerp(w, near, far), -1.0, 1.0)


def _body_source(f, lon, lat, radius):
    lon, lat = torch.deg2rad(lon), torch.deg2rad(lat)
    p = [torch.cos(lat) * torch.cos(lon) * radius, torch.cos(lat) * torch.sin(lon) * radius,
         torch.sin(lat) * radius]
    t = torch.eye(3, dtype=torch.float64)
    frequency, weight, total = 1.0 / float(f["wavelength"]), 1.0, 0.0
    out = torch.zeros_like(p[0])
    for o in range(int(f["octaves"])):
        h, h1, h2 = _pcg3d(int(f["seed"]), o, 0)
        g = _pcg3d(int(f["seed"]), o, 1)[0]
        r = [sum(float(t[k, m]) * p[m] for m in range(3)) * frequency for k in range(3)]
        out = out + weight * _perlin3(r[0] + _unit(h1), r[1] + _unit(h2), r[2] + _unit(g), h)
        total += weight
        weight *= float(f["gain"])
        frequency *= float(f["lacunarity"])
        t = _TURN3 @ t
    return float(f["amplitude"]) * out / total


def _pairs(c0, c1, r0, r1, most=1 << 22):
    """(feature, col, row) of every cell of the boxes [c0, c1) x [r0, r1), some features at a
    time."""
    wide = (c1 - c0).clamp(min=0)
    n = wide * (r1 - r0).clamp(min=0)
    ends = torch.cumsum(n, 0)
    total = int(ends[-1]) if len(ends) else 0
    starts = ends - n
    for p in range(0, total, most):
        k = torch.arange(p, min(p + most, total), device=n.device)
        i = torch.searchsorted(ends, k, right=True)
        local = k - starts[i]
        yield i, c0[i] + local % wide[i], r0[i] + local // wide[i]


def _window(grid, x, y, reach):
    c = [(x - reach - grid.x0) / grid.pixel, (x + reach - grid.x0) / grid.pixel]
    r = [(grid.y0 - y - reach) / grid.pixel, (grid.y0 - y + reach) / grid.pixel]
    return (c[0].floor().clamp(0, grid.width).long(), c[1].ceil().clamp(0, grid.width).long(),
            r[0].floor().clamp(0, grid.height).long(), r[1].ceil().clamp(0, grid.height).long())


def _smooth(t):
    t = torch.clamp(t, 0.0, 1.0)
    return t * t * (3.0 - 2.0 * t)


def _ft_shape(x, rim, fresh_rim, depth):
    """The Fassett-Thomson profile (diameters) at x radii."""
    inside = -0.228809953 + x * (0.227533882 + x * (0.083116795 - x * 0.039499407))

    def outside(start):
        poly = 0.188253307 + x * (-0.187050452 + x * (0.01844746 + x * 0.01505647))
        return poly * (1.0 - ((x - start) / (1.5 - start)) ** 2)

    if rim == 2:
        h = torch.where(x <= 0.98, inside, torch.where(x <= 1.02, fresh_rim, outside(1.02)))
    else:
        edge = 0.98 if rim == 0 else 1.0
        h = torch.where(x <= 0.2, -0.181, torch.where(x <= edge, inside, outside(edge)))
    return torch.where(x > 1.5, 0.0, torch.maximum(h, fresh_rim - depth))


def _mpd_height(distance, diameter, fresh_rim, depth, rim):
    """The Martin-Parkes-Dunstan profile (meters)."""
    depth, rim, fresh = depth * diameter, rim * diameter, fresh_rim * diameter
    radius = 0.5 * diameter
    x = distance / radius - 1.0
    k = fresh - rim + depth
    alpha = (rim - fresh) / k
    es = 0.14 * radius ** 0.74
    es = torch.where(fresh > 0.0, es * rim / fresh, es)
    beta = torch.clamp(1.5 * (fresh - rim) / k, max=1.0)

    def exterior(u):
        offset = rim - es
        slope = -es / 8.0 - offset
        r = 1.0 / (u + 1.0)
        law, fall, taper = es * r ** 3 + offset + slope * u, -3.0 * es * r ** 4 + slope, 1.0 - u * u
        return law * taper, fall * taper - 2.0 * u * law

    join, slope = exterior(beta)
    drop = rim - join
    slope = torch.where(drop > 0.0, torch.maximum(slope, -3.0 * drop / beta), slope)
    t = x / beta
    near = rim + (join - rim) * t * t * (3.0 - 2.0 * t) + beta * slope * t * t * (t - 1.0)
    h = torch.where(x <= beta, near, exterior(x)[0])
    h = torch.where(x <= 0.0, k * (alpha + 1.0) / alpha * x * x + rim, h)
    h = torch.where(x <= alpha, (k * x + 2.0 * k) * x + fresh, h)
    return torch.where(x >= 1.0, 0.0, h)


def _kilometers(coefficient, exponent, diameter):
    return coefficient * (diameter / 1000.0) ** exponent


def _crater_sum(batch, grid):
    """The sum over the batch's craters of what each adds at the grid's cells, in 64 bits: the
    closed-form profiles with ellipses, outline harmonics, wall terraces and massif peaks."""
    kernel, records, data, footprints = batch
    for name in ("tableCount", "markCount", "hasDatum"):
        assert not records[name].any(), "none under these cases' options"
    total = torch.zeros(grid.height * grid.width, dtype=torch.float64, device="cuda")
    if not len(records):
        return total.view(grid.height, grid.width)
    p = kernel["profile"]
    f = {k: torch.from_numpy(records[k].astype(np.float64)).cuda()
         for k in ("x", "xLow", "y", "yLow", "diameter", "resolution", "freshDepth", "freshRim",
                   "currentDepth", "currentRim", "ellipticity", "heading")}
    count = torch.from_numpy(records["harmonicCount"].astype(np.int64)).cuda()
    first = torch.from_numpy(records["firstHarmonic"].astype(np.int64)).cuda()
    offset = torch.from_numpy(records["harmonicOffset"].astype(np.int64)).cuda()
    peaks = torch.from_numpy(records["peakCount"].astype(np.int64)).cuda()
    peak_at = torch.from_numpy(records["peakOffset"].astype(np.int64)).cuda()
    terraces = torch.from_numpy(records["terraceCount"].astype(np.int64)).cuda()
    terrace_at = torch.from_numpy(records["terraceOffset"].astype(np.int64)).cuda()
    d = torch.from_numpy(data.astype(np.float64)).cuda()
    d = torch.cat([d, torch.zeros(512, dtype=torch.float64, device="cuda")])
    foot = torch.from_numpy(footprints).cuda().view(-1, 3)
    x, y = f["x"] + f["xLow"], f["y"] + f["yLow"]
    reach_radii = float(kernel["reachRadii"])
    most = int(count.max())
    complex_ = (f["diameter"] >= float(p["transitionDiameter"])) & (int(p["complex"]) == 1)
    # Simple craters of a complex profile end at their own profile's reach.
    simple_reach = 2.0 if int(p["simple"]) == 1 else 1.5
    reach = torch.where(complex_ | (int(p["complex"]) != 1), foot[:, 2],
                        foot[:, 2] * (simple_reach / reach_radii))
    fitted = f["diameter"]
    if float(p["peakFitMaxDiameter"]) > 0.0:
        fitted = torch.clamp(fitted, max=float(p["peakFitMaxDiameter"]))
    peak_height = 1e3 * _kilometers(float(p["peakHeightCoefficient"]),
                                    float(p["peakHeightExponent"]), fitted)
    width = _kilometers(float(p["peakWidthCoefficient"]), float(p["peakWidthExponent"]), fitted)
    peak_base = (torch.sqrt(3.0 * 1e9 * width / (math.pi * peak_height))
                 if int(p["peakFromVolume"]) == 1 else 500.0 * width) * f["diameter"] / fitted
    floor = torch.clamp(1e3 * _kilometers(float(p["floorCoefficient"]),
                                          float(p["floorExponent"]), f["diameter"]) /
                        f["diameter"], max=0.9)
    worn = torch.where(f["freshRim"] > 0.0,
                       torch.clamp(f["currentRim"] / f["freshRim"], 0.0, 1.0), 1.0)
    kept_depth = torch.where(f["freshDepth"] > 0.0, f["currentDepth"] / f["freshDepth"], 1.0)
    xs, ys = _axes(grid)
    for i, col, row in _pairs(*_window(grid, x, y, reach)):
        dx, dy = xs[col] - x[i], ys[row] - y[i]
        diameter = f["diameter"][i]
        radius = 0.5 * diameter
        r = torch.sqrt(dx * dx + dy * dy)
        theta = torch.atan2(dy, dx)
        share = _smooth(r / radius) * worn[i]
        wobble = torch.ones_like(r)
        for h in range(most):
            order = (first[i] + h).double()
            at = offset[i] + 2 * h
            wave = share ** (0.5 * order) * d[at] * torch.cos(order * theta + d[at + 1])
            wobble = wobble + torch.where((h < count[i]) & (share > 0.0), wave, 0.0)
        along = torch.sqrt(f["ellipticity"][i])
        turn = theta - f["heading"][i]
        stretch = 1.0 / torch.sqrt((torch.cos(turn) / along) ** 2 + (torch.sin(turn) * along) ** 2)
        distance = r / (stretch * wobble)
        for n in torch.unique(i[terraces[i] > 0]).tolist():
            at = torch.nonzero(i == n).view(-1)
            distance[at] = _terraced(d[terrace_at[n]:terrace_at[n] + 512], int(terraces[n]),
                                     distance[at] / radius[at], theta[at]) * radius[at]
        fresh_rim, depth, rim = f["freshRim"][i], f["currentDepth"][i], f["currentRim"][i]
        if int(p["simple"]) == 1:
            height = _mpd_height(distance, diameter, fresh_rim, depth, rim)
        else:
            height = _ft_shape(distance / radius, int(p["rim"]), fresh_rim, depth) * diameter
        at = torch.nonzero(complex_[i]).view(-1)
        if len(at):
            n = i[at]
            height[at] = _complex(p, distance[at], radius[at], depth[at], rim[at], floor[n],
                                  kept_depth[n], peak_height[n], peak_base[n])
            at = at[peaks[i[at]] > 0]
            n = i[at]
            reach2 = (2.6 * peak_base[n] * torch.clamp(d[peak_at[n] + 5], min=1.0)) ** 2
            at = at[r[at] ** 2 < reach2]
            if len(at):
                n = i[at]
                height[at] += kept_depth[n] * (
                    _massifs(d, peak_at[n], peaks[n], peak_height[n], peak_base[n], dx[at], dy[at])
                    - _dome(peak_height[n], peak_base[n], distance[at]))
        shaped = torch.where(distance < reach_radii * radius, f["resolution"][i] * height, 0.0)
        total.index_add_(0, row * grid.width + col, shaped)
    return total.view(grid.height, grid.width)


def _terraced(d, count, radii, theta):
    """One crater's profile distance (radii) after its wall terraces; `d` its terraces' data:
    a header of 20, 8 for each of the count - 1 scarps, 3 for each step."""
    d = d.tolist()

    def turned(at, offset):
        turns = d[at] * theta / (2.0 * math.pi) + d[offset]
        return turns, 1.0 - (2.0 * (turns - torch.floor(turns)) - 1.0) ** 2 - 2.0 / 3.0

    def blocks(s, salt, gaps):
        turns, _ = turned(s + 2, s + 3)
        key = int(d[s + 7]) ^ ((salt * 0x85EBCA6B) & _M)
        cell = torch.floor(turns)
        u, cell = turns - cell, cell.long()

        def value(k):
            h = _unit(_pcg((key + (k % int(d[s + 2])) * 0x9E3779B9) & _M)).double()
            return h if gaps < 0.0 else (h >= gaps).double()

        edge = torch.minimum(u, 1.0 - u)
        b = torch.where(edge < 0.3, _smooth(0.5 + 0.5 * edge / 0.3), 1.0)
        beside = value(torch.where(u < 0.5, cell - 1, cell + 1))
        return beside * (1.0 - b) + value(cell) * b

    def base(k):
        return 0.0 if k == 0 else 1.0 if k >= count else d[20 + 8 * (k - 1)]

    def scarp(k):
        if k == 0 or k >= count:
            return torch.full_like(radii, base(k))
        s = 20 + 8 * (k - 1)
        return (d[s] + d[s + 1] * turned(s + 2, s + 3)[1] +
                d[s + 4] * torch.cos(3.0 * theta + d[s + 5]) +
                d[s + 6] * (2.0 * blocks(s, 0, -1.0) - 1.0))

    def ease(v):
        steepest = 1.0 / (1.0 - 0.5 * d[3])
        return torch.where(v < d[3], steepest * v * v / (2.0 * d[3]), steepest * (v - 0.5 * d[3]))

    rim = 1.0 + d[16] * turned(17, 18)[1]
    radii = radii / (1.0 + (rim - 1.0) * _smooth(radii))
    inner = d[0]
    t = (radii - inner) / (1.0 - inner)
    scarps = [scarp(k) for k in range(count + 1)]
    step = torch.zeros_like(radii, dtype=torch.long)
    for k in range(1, count):
        step = torch.where((step == k - 1) & (t >= scarps[k]), k, step)
    out = radii.clone()
    for k in range(count):
        low, high = scarps[k], scarps[k + 1]
        within = torch.clamp((t - low) / (high - low), 0.0, 1.0)
        strength = torch.full_like(t, d[2])
        if d[4] > -1.5:
            arcs = sum(d[6 + 2 * n] * torch.cos((2 + n) * (theta + 2.39996323 * k) + d[7 + 2 * n])
                       for n in range(5))
            strength = strength * _smooth((arcs - d[4]) / d[5])
        if count > 1:
            top = k + 1 >= count
            strength = strength * blocks(20 + 8 * ((k if top else k + 1) - 1), 2 if top else 1,
                                         d[19])
        level, width, share = d[20 + 8 * (count - 1) + 3 * k:][:3]
        strength = strength * share
        lower, upper = width * level, width * (1.0 - level)
        stair = torch.full_like(t, level)
        stair = torch.where(within > 1.0 - upper,
                            level + (1.0 - level) * ease((within - (1.0 - upper)) / upper), stair)
        stair = torch.where(within < lower, level * (1.0 - ease(1.0 - within / lower)), stair)
        rise = d[1] * within + (1.0 - d[1]) * stair
        shaped = within + strength * (rise - within)
        at = (step == k) & (radii > inner) & (radii < 1.0)
        out = torch.where(at, inner + (base(k) + shaped * (base(k + 1) - base(k))) * (1.0 - inner),
                          out)
    return out


def _dome(height, base, distance):
    return torch.where(distance < base, height * (1.0 - (distance / base) ** 2) ** 2, 0.0)


def _complex(p, distance, radius, depth, rim, floor, kept, peak_height, peak_base):
    x = distance / radius
    depth, rim = depth * 2.0 * radius, rim * 2.0 * radius
    far, law = float(p["complexReachRadii"]), float(p["ejectaExponent"])
    edge = far ** -law
    out = torch.where(x >= far, 0.0, rim * (torch.clamp(x, min=1.0) ** -law - edge) / (1.0 - edge))
    t = torch.clamp((x - floor) / (1.0 - floor), min=0.0)
    inside = rim - depth + depth * t * t + kept * _dome(peak_height, peak_base, distance)
    return torch.where(x >= 1.0, out, inside)


def _massifs(d, o, count, height, base, dx, dy):
    """A complex crater's massif peak: warped cones, the tallest, roughened by ridges."""
    height, base = height * d[o + 4], base * d[o + 5]
    px, py = dx / base, dy / base
    rough, wave, warp, key = d[o], d[o + 1], d[o + 2], d[o + 3].long()
    wx = _fractal2(px, py, (key + 1) & _M, 2.0 * wave, 3)
    wy = _fractal2(px + 17.31, py - 9.73, (key + 1) & _M, 2.0 * wave, 3)
    px, py = px + warp * wx, py + warp * wy
    best = torch.zeros_like(px)
    for n in range(int(count.max())):
        m = torch.where(n < count, o + 6 + 11 * n, o + 6)
        ex, ey, radius, stretch = px - d[m], py - d[m + 1], d[m + 2], d[m + 3]
        qx = (ex * d[m + 4] + ey * d[m + 5]) / (radius * stretch)
        qy = (ey * d[m + 4] - ex * d[m + 5]) * stretch / radius
        squared = qx * qx + qy * qy
        pull = 1.0 - squared
        sx, sy = qx - d[m + 8] * pull, qy - d[m + 9] * pull
        r = torch.clamp(torch.sqrt(sx * sx + sy * sy), max=1.0)
        cone = d[m + 6] * (1.0 - r ** d[m + 7]) ** d[m + 10]
        best = torch.maximum(best, torch.where(squared < 1.0, cone, 0.0))
    ridges = _fractal2(px, py, key, wave, 5, type=1)
    return height * torch.where(best > 0.0, best * (1.0 + rough * ridges), best)


def _boulder_max(stones, grid, base):
    """Each boulder's dome, averaged over a sample width, max-composited on `base`."""
    if not len(stones):
        return base
    best = base.clone().view(-1)
    x, y, diameter, exposed, weight = stones.unbind(1)
    width = grid.pixel
    xs, ys = _axes(grid)
    for i, col, row in _pairs(*_window(grid, x, y, 0.5 * (diameter + width))):
        distance, radius = torch.hypot(xs[col] - x[i], ys[row] - y[i]), 0.5 * diameter[i]

        def area(u):
            u = torch.clamp(u, -1.0, 1.0)
            return 0.5 * (u * torch.sqrt(1.0 - u * u) + torch.asin(u))

        lift = exposed[i] * (area((distance + 0.5 * width) / radius) -
                             area((distance - 0.5 * width) / radius)) * radius / width
        at = row * grid.width + col
        drawn = torch.where((weight[i] > 0.0) & (lift > 0.0), base.view(-1)[at] + weight[i] * lift,
                            -math.inf)
        best.scatter_reduce_(0, at, drawn, "amax")
    return best.view_as(base)


def _philox(c0, c1, c2, k0, k1):
    c3 = torch.zeros_like(c0)
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57  # the low 64 bits of 32 x 32-bit products
        c0, c1, c2, c3 = (((p1 >> 32) & _M) ^ c1 ^ k0, p1 & _M, ((p0 >> 32) & _M) ^ c3 ^ k1,
                          p0 & _M)
        k0, k1 = (k0 + 0x9E3779B9) & _M, (k1 + 0xBB67AE85) & _M
    return c0, c1, c2, c3


def _node_normal(col, row, level, seed):
    high = ((col >> 32) ^ (row >> 32)) & _M
    a, b, c, e = _philox(col & _M, row & _M, (level | (high << 5)) & _M, seed, 0x524D4450)
    u1 = ((a >> 5) * 2 ** 26 + (b >> 6)).double() * 2.0 ** -53
    u2 = ((c >> 5) * 2 ** 26 + (e >> 6)).double() * 2.0 ** -53
    return torch.sqrt(-2.0 * torch.log1p(-u1)) * torch.cos(2.0 * math.pi * u2)


def _refined(state, grid, dimension=2.2, scale=1.5):
    """Diamond-square over the whole grid, level by level, read at its cells."""
    posts, pg, spline = state["posts"].double(), state["post_grid"], state["interp"] == 1
    levels = max(0, math.ceil(math.log2(pg.pixel / grid.pixel) - 1e-9))
    step = pg.pixel / 2.0 ** levels
    xs, ys = _axes(grid)
    u = (xs - (pg.x0 + 0.5 * pg.pixel)) / step
    v = (ys - (pg.y0 - 0.5 * pg.pixel)) / step
    reach, before, after = (3, 1, 2) if spline else (1, 0, 1)
    mid = torch.tensor([-1.0, 9.0, 9.0, -1.0], device="cuda", dtype=torch.float64) / 16.0
    boxes = {levels: [math.floor(float(u.min())) - 2, math.ceil(float(u.max())) + after + 1,
                      math.floor(float(v.min())) - 2, math.ceil(float(v.max())) + after + 1]}
    for n in range(levels, 0, -1):
        c0, c1, r0, r1 = boxes[n]
        boxes[n - 1] = [(c0 - reach) // 2 - before - 1, (c1 + reach) // 2 + after + 1,
                        (r0 - reach) // 2 - before - 1, (r1 + reach) // 2 + after + 1]
    c0, c1, r0, r1 = boxes[0]
    pc = torch.arange(c0, c1 + 1, device="cuda").clamp(0, pg.width - 1)
    pr = (-torch.arange(r0, r1 + 1, device="cuda")).clamp(0, pg.height - 1)
    nodes = posts[pr[:, None], pc[None, :]]
    factor = 2.0 ** (-(3.0 - dimension) / 2.0)
    seed = state["seed"]

    def normals(cols, rows, level):
        at = torch.broadcast_tensors(cols[None, :], rows[:, None])
        return torch.cat([_node_normal(a, b, level, seed)
                          for a, b in zip(at[0].split(512), at[1].split(512))])

    for n in range(1, levels + 1):
        pc0, _, pr0, _ = boxes[n - 1]
        c0, c1, r0, r1 = 2 * pc0, 2 * (pc0 + nodes.shape[1]) - 1, 2 * pr0, \
            2 * (pr0 + nodes.shape[0]) - 1
        wide = torch.zeros((r1 - r0 + 1, c1 - c0 + 1), device="cuda", dtype=torch.float64)
        wide[0::2, 0::2] = nodes
        cols = torch.arange(c0, c1 + 1, device="cuda")
        rows = torch.arange(r0, r1 + 1, device="cuda")

        def mean4(a, axis):  # the value between entries k and k + 1 (edges repeat their end)
            k = torch.arange(a.shape[axis], device="cuda")
            taps = [a.index_select(axis, (k + t).clamp(0, a.shape[axis] - 1))
                    for t in ((-1, 0, 1, 2) if spline else (0, 1))]
            if spline:
                return sum(m * t for m, t in zip(mid, taps))
            return 0.5 * (taps[0] + taps[1])

        square = mean4(mean4(nodes, 1), 0)
        wide[1::2, 1::2] = square + scale * factor ** (2 * n - 1) * normals(cols[1::2], rows[1::2],
                                                                           n)
        diamond = scale * factor ** (2 * n)
        even, odd = wide[0::2, 0::2], wide[1::2, 1::2]

        def shifted(a, axis):  # as mean4, between entries k - 1 and k
            return torch.roll(mean4(a, axis), 1, axis)

        # (odd col, even row): even nodes along x, odd nodes along y; and the other way round.
        east = 0.5 * (mean4(even, 1) + shifted(odd, 0))
        north = 0.5 * (shifted(odd, 1) + mean4(even, 0))
        wide[0::2, 1::2] = east + diamond * normals(cols[1::2], rows[0::2], n)
        wide[1::2, 0::2] = north + diamond * normals(cols[0::2], rows[1::2], n)
        b = boxes[n]
        nodes = wide[b[2] - r0:b[3] - r0 + 1, b[0] - c0:b[1] - c0 + 1].contiguous()
    c0, _, r0, _ = boxes[levels]

    def taps(t, lo):
        near = torch.round(t)
        t = torch.where((t - near).abs() <= 1e-6, near, t)
        k = torch.floor(t)
        share, k = t - k, k.long() - lo
        if not spline:
            return [(k, 1.0 - share), (torch.where(share > 0.0, k + 1, k), share)]

        def weight(z):
            z = z.abs()
            return torch.where(z <= 1.0, (1.5 * z - 2.5) * z * z + 1.0,
                               torch.where(z < 2.0, ((-0.5 * z + 2.5) * z - 4.0) * z + 2.0, 0.0))

        return [(k + j, weight(share - j)) for j in (-1, 0, 1, 2)]

    lines = sum(w[None, :] * nodes[:, k] for k, w in taps(u, c0))
    return sum(w[:, None] * lines[k] for k, w in taps(v, r0))


def _near(mask, radius):
    return torch.nn.functional.max_pool2d(mask[None, None].half(), 2 * radius + 1, 1,
                                          radius)[0, 0] > 0


def _chained(state, mode, decay):
    """The chain's heights with each link's field solved by conjugate gradients in 64 bits."""
    chain, patches, grid = state["chain"], state["patches"], state["grid"]
    nan = float("nan")
    whole = torch.full((grid.height, grid.width), nan, dtype=torch.float64, device="cuda")
    whole[state["windows"][0].slices()] = patches[0].double()
    dx = grid.pixel
    reach = 3.0 * decay
    for k in range(1, len(patches)):
        later = torch.full_like(whole, nan)
        later[state["windows"][k].slices()] = patches[k].double()
        win, _ = chain.lattice(k)
        h, w = win.height, win.width
        r0, r1 = max(0, win.row0), min(grid.height, win.row0 + h)
        c0, c1 = max(0, win.col0), min(grid.width, win.col0 + w)
        part = (slice(r0 - win.row0, r1 - win.row0), slice(c0 - win.col0, c1 - win.col0))
        a = torch.full((h, w), nan, dtype=torch.float64, device="cuda")
        b = a.clone()
        a[part], b[part] = whole[r0:r1, c0:c1], later[r0:r1, c0:c1]
        data = ~a.isnan()
        keep = data & _near(~data, 3) & ~b.isnan()
        fixed = torch.where(keep, a - b, 0.0)
        # The chamfer distance to data, as far as the solve reaches.
        dist = torch.where(data, 0.0, math.inf).double()
        for _ in range(int(math.ceil(reach / dx)) + 1):
            pad = torch.nn.functional.pad(dist, (1, 1, 1, 1), value=math.inf)
            for j in range(3):
                for i in range(3):
                    step = dx * math.hypot(i - 1, j - 1)
                    dist = torch.minimum(dist, pad[j:j + h, i:i + w] + step)
        unknown = ~data & (dist <= reach * (1.0 + 1e-9))
        unknown[:3], unknown[-3:], unknown[:, :3], unknown[:, -3:] = False, False, False, False
        mask = unknown.double()
        centre = 4.0 / dx ** 2 + 1.0 / decay ** 2

        def laplace(v):
            out = centre * v
            out[1:] -= v[:-1] / dx ** 2
            out[:-1] -= v[1:] / dx ** 2
            out[:, 1:] -= v[:, :-1] / dx ** 2
            out[:, :-1] -= v[:, 1:] / dx ** 2
            return out

        def apply(v):
            return laplace(laplace(v)) if mode == "slope" else laplace(v)

        x = torch.zeros_like(fixed)
        r = -mask * apply(fixed)
        p, rr = r.clone(), (r * r).sum()
        goal = float(rr) * 1e-22
        for n in range(60000):
            if n % 50 == 0 and float(rr) <= goal:
                break
            ap = mask * apply(p)
            alpha = rr / (p * ap).sum()
            x += alpha * p
            r -= alpha * ap
            new = (r * r).sum()
            p = r + (new / rr) * p
            rr = new
        field = torch.full_like(whole, 0.0)
        field[r0:r1, c0:c1] = (fixed + x)[part]
        whole = torch.where(whole.isnan(), later + field, whole)
    return whole


def exact(case, seed):
    kind = case["kind"]
    if kind == "seams" and case["mode"] == "feather":
        # A feathered post carries the value of the nearest post with data; between equally near
        # ones the scan order decides, which 64-bit arithmetic does not define.
        return None
    state = prepare(case, seed)
    if kind == "seams":
        return _chained(state, case["mode"], case["overlap"] * case["pixel"] / 3.0)
    if kind == "tiles":
        return _tiles(state)
    grid = state["grid"]
    if kind == "body":
        f = state["fractals"][0]
        return _by_rows(grid, lambda x, y: _body_source(f, x, y, 1737400.0))
    if kind == "refine":
        return _refined(state, grid)
    if kind == "layer":
        n = int(state["kernel"]["count"])
        return state["base"].double() + _by_rows(
            grid, lambda x, y: _stack2(state["kernel"]["fractals"][:n], x, y))
    if kind in ("source", "terrain"):
        height = _by_rows(grid, lambda x, y: _stack2(state["fractals"], x, y))
    else:
        height = state["base"].double()
    if kind in ("craters", "terrain"):
        height = height + _crater_sum(state["host"], grid)
    if kind in ("boulders", "terrain"):
        height = _boulder_max(state["boulders"].view(-1, 5), grid, height)
    return height


def _tiles(state):
    ts = state["tiles"]
    out = torch.zeros(ts.output_floats, dtype=torch.float64, device="cuda")
    for grid, t in zip(ts.grids, ts.tiles):
        c0, c1 = int(t["crater_begin"]), int(t["crater_begin"]) + int(t["crater_count"])
        b0, b1 = int(t["boulder_begin"]), int(t["boulder_begin"]) + int(t["boulder_count"])
        end = len(ts.crater_data) if c1 == len(ts.crater_records) else None
        data = ts.crater_data[int(t["data_begin"]):end]
        height = _by_rows(grid, lambda x, y: _stack2(ts.fractals, x, y))
        height = height + _crater_sum((ts.crater_kernel, ts.crater_records[c0:c1], data,
                                       ts.crater_footprints[3 * c0:3 * c1]), grid)
        height = _boulder_max(torch.from_numpy(ts.boulders[b0:b1]).cuda(), grid, height)
        rows = out[int(t["height_offset"]):]
        rows.as_strided((grid.height, grid.width), (int(t["pitch"]), 1)).copy_(height)
    return out
