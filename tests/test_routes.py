"""Which calls go by shortened programs: the rules weigh what a call could save against what building
them costs, and both sides were measured where a test here draws the line.  No GPU needed."""

import ctypes as C
import math

import numpy as np
import pytest

from tangerine_gb300 import _lib, sdf
from tangerine_gb300 import workloads as W

U, D, I, BU, BD, BI = W.UNION, W.DIFF, W.INTER, W.BLEND_UNION, W.BLEND_DIFF, W.BLEND_INTER
BLENDS = ((U, 0.3), (D, 0.2), (I, 0.05), (BU, 0.25), (BD, 0.1), (BI, 0.1))
EXPORT, LATTICE, CLOUD, RENDER = range(4)


def _tree(prims, seed, blends=False):
    kw = {"ops": BLENDS} if blends else {}
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, **kw))):
        seed += 7919
    return sdf.from_spec(spec)


def _by_tapes(lib, tree, call, grid=None, pixels=0):
    answer = lib.tg_debug_goes_by_tapes(tree.handle, call, C.byref(grid) if grid is not None else None, pixels)
    assert answer >= 0
    return bool(answer)


# Measured without / with tapes, us an image.
@pytest.mark.parametrize("prims,seed,blends,width,height,tapes", [
    (1, 3, False, 1920, 1080, False),       # 168 / 238
    (1, 2, False, 400, 300, False),         # 211 / 279
    (2, 3, False, 1920, 1080, False),       # 256 / 270
    (4, 4, True, 128, 96, False),           # 122 / 177
    (8, 6, True, 64, 48, False),            # 152 / 193
    (8, 4, True, 128, 96, True),            # 237 / 221
    (4, 3, False, 800, 500, True),          # 385 / 260
    (16, 3, False, 64, 48, False),          # 191 / 227
    (8, 2, False, 200, 150, True),          # 627 / 441
    (32, 6, True, 128, 96, True),           # 459 / 283
    (64, 3, False, 64, 48, True),           # 382 / 237
    (256, 2, False, 64, 48, True),          # 1757 / 667
])
def test_render(lib, prims, seed, blends, width, height, tapes):
    assert _by_tapes(lib, _tree(prims, seed, blends), RENDER, pixels=width * height) == tapes


# Measured by whole programs / by tapes, us a call.
@pytest.mark.parametrize("prims,seed,blends,n,tapes", [
    (1, 4, True, 300, False),               # 163 / 177
    (2, 4, True, 300, False),               # 182 / 188
    (4, 3, False, 300, True),               # 251 / 208
    (16, 3, False, 150, False),             # 110 / 115
    (16, 3, False, 190, True),              # 189 / 134
    (32, 4, True, 150, True),               # 378 / 137
    (128, 2, False, 190, True),             # 329 / 244
    (256, 2, False, 64, False),             # 269 / 448
    (512, 3, False, 110, False),            # 314 / 471
    (512, 4, True, 64, False),              # 1455 / 2244
    (512, 4, True, 110, True),              # 2764 / 2175
])
def test_lattice(lib, prims, seed, blends, n, tapes):
    grid = _lib.Grid(-1.6, -1.6, -1.6, 3.2 / (n - 1), n, n, n)
    assert _by_tapes(lib, _tree(prims, seed, blends), LATTICE, grid) == tapes


def test_lattice_of_long_programs_and_few_points(lib):
    """125 primitives of some 300 quads: 250 us by whole programs, 482 by tapes."""
    spec = W.random_tree(11 * 1000003 + 125, 125)
    assert sdf.has_export_octree(sdf.from_spec(spec))
    n = (34, 318, 59)
    step = [3.2 / (k - 1) for k in n]
    assert not _by_tapes(lib, sdf.from_spec(spec), LATTICE, _lib.Grid(-1.6, -1.6, -1.6, step[0], *n, step[1], step[2]))


# Measured by whole programs / by tapes, us an export to the device.
@pytest.mark.parametrize("prims,seed,blends,res,tapes", [
    (1, 2, False, 900, False),              # 264 / 270
    (16, 3, False, 512, False),             # 164 / 197
    (16, 3, False, 900, False),             # 249 / 271
    (16, 4, True, 720, False),              # 215 / 233
    (32, 3, False, 720, False),             # 255 / 285
    (64, 4, True, 400, False),              # 169 / 222
    (64, 2, False, 900, True),              # 922 / 820
    (128, 2, False, 720, True),             # 948 / 779
    (256, 2, False, 400, False),            # 546 / 587
    (256, 2, False, 512, True),             # 755 / 658
    (512, 4, True, 320, False),             # 902 / 1011
    (512, 6, True, 450, True),              # 1029 / 817
])
def test_export(lib, prims, seed, blends, res, tapes):
    grid = sdf._grid(W.export_grid(resolution=res))
    assert _by_tapes(lib, _tree(prims, seed, blends), EXPORT, grid) == tapes


# Measured without / with tapes, us a call.
@pytest.mark.parametrize("prims,seed,blends,step,tapes", [
    (1, 3, False, 0.03, False),             # 124 / 141
    (8, 2, False, 0.03, False),             # 213 / 225
    (8, 2, False, 0.015, True),             # 322 / 243
    (64, 4, True, 0.04, False),             # 422 / 569
    (64, 3, False, 0.02, True),             # 338 / 241
    (128, 3, False, 0.03, False),           # 495 / 604
    (256, 2, False, 0.02, True),            # 1705 / 1056
    (512, 4, True, 0.06, False),            # 2299 / 7287
    (512, 4, True, 0.04, False),            # 2585 / 4712
    (512, 4, True, 0.02, True),             # 5552 / 2038
    (512, 6, True, 0.06, False),            # 845 / 3471
])
def test_cloud(lib, prims, seed, blends, step, tapes):
    n = math.ceil(3.2 / step)
    grid = _lib.Grid(-1.6, -1.6, -1.6, step, n, n, n)
    assert _by_tapes(lib, _tree(prims, seed, blends), CLOUD, grid) == tapes


# Wide scenes build eight times as many tapes: without / with, us an image.
@pytest.mark.parametrize("width,height,tapes", [(640, 360, False), (1920, 1080, True)])      # 566 / 815, 1453 / 1024
def test_render_of_wide_scenes(lib, width, height, tapes):
    rng = np.random.default_rng(4)
    tree = None
    for i in range(60):
        a = rng.uniform(0.5, 1.0)
        q = rng.normal(size=4)
        brush = (sdf.sphere(a), sdf.box(a, 0.7 * a, 0.9 * a), sdf.torus(a, 0.3 * a))[i % 3].rotate(*[float(v) for v in q / np.linalg.norm(q)])
        brush.move(*[float(v) for v in rng.uniform(-6, 6, 3)])
        tree = brush if tree is None else sdf.union(tree, brush)
    assert _by_tapes(lib, tree, RENDER, pixels=width * height) == tapes
