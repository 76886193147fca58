"""Shortened programs (tg_tape.cuh) against whole ones: a tape leaves out only operands that
lose everywhere in its box, so every value it gives is the whole program's, bit for bit (the
tolerance is 0)."""

import ctypes as C

import numpy as np
import pytest

from conftest import golden_names
from tangerine_gb300 import _lib, sdf
from tangerine_gb300 import workloads as W

pytestmark = pytest.mark.gpu

ALL_OPS = ((W.UNION, 0.2), (W.DIFF, 0.2), (W.INTER, 0.1), (W.BLEND_UNION, 0.2), (W.BLEND_DIFF, 0.15), (W.BLEND_INTER, 0.15))
# Coarse (bricks larger than octree cells, many parts a brick), fine, cut bricks on every
# axis, a step per axis, one brick, one cell.
GRIDS = {
    "coarse": (-2.0, -2.0, -2.0, 0.11, 38, 38, 38),
    "fine": (-0.75, -0.6, -0.4, 0.004, 150, 142, 129),
    "ragged": (-1.9, -1.7, -2.0, 0.021, 173, 120, 191, 0.027, 0.019),
    "brick": (-0.3, -0.2, -0.3, 0.03, 8, 8, 8),
    "cell": (0.1, 0.1, 0.1, 0.5, 2, 2, 2),
}


def _same(a, b):
    for x, y in ((a.vertices, b.vertices), (a.cubes, b.cubes), (a.faces, b.faces), (a.normals, b.normals)):
        np.testing.assert_array_equal(x, y)
    assert (a.colors is None) == (b.colors is None)
    if a.colors is not None:
        np.testing.assert_array_equal(a.colors, b.colors)


@pytest.mark.parametrize("grid", sorted(GRIDS))
@pytest.mark.parametrize("prims,ops,paint", [(1, ALL_OPS, True), (2, ALL_OPS, True), (40, ALL_OPS, True), (150, W.OPS_60_20_10_10, True),
                                             (60, ALL_OPS, False)])
def test_brick_tapes_equal_dense_export(lib, grid, prims, ops, paint):
    seed = 3
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops, paint=paint))):
        seed += 1
    with sdf.compile(sdf.from_spec(spec)) as prog:
        g = _lib.Grid(*GRIDS[grid])
        _same(prog.export_mesh(g, dense=True), prog.export_mesh(g, tapes=True))


@pytest.mark.parametrize("name", golden_names())
def test_brick_tapes_equal_dense_export_fixture_trees(lib, golden, name):
    """Every brush and operator (ellipsoids, cones, stencils, scales, flates, unpainted brushes)."""
    g = golden[name]
    if "octree_nodes" not in g:
        pytest.skip("no octree")
    with sdf.compile(sdf.from_spec(g["spec"])) as prog:
        info = prog.info()
        lo, hi = np.asarray(info.bounds_min[:]), np.asarray(info.bounds_max[:])
        for cells in (20, 130):
            step = float(np.max(hi - lo)) * 1.1 / cells
            n = [int(np.ceil((h - l) * 1.1 / step)) + 3 for l, h in zip(lo, hi)]
            start = [float(l - 0.05 * (h - l) - step) for l, h in zip(lo, hi)]
            grid = _lib.Grid(*start, step, *n)
            _same(prog.export_mesh(grid, dense=True), prog.export_mesh(grid, tapes=True))


def test_brick_tapes_far_large_and_stretched_operands(lib):
    """Operands whose own float error is large (a sphere of radius 3000 seen near its surface),
    a thin blend, and rotations that are not unit quaternions (never shortened)."""
    cut = sdf.sphere(3000.0).move(0.0, 0.0, -2999.9)
    body = sdf.blend_union(0.003, sdf.box(0.5, 0.4, 0.6), sdf.torus(0.5, 0.1).move(0.2, 0.1, 0.3))
    tree = sdf.inter(sdf.blend_diff(0.05, body, sdf.sphere(0.3).move(0.4, 0.3, 0.2)), cut)
    stretched = sdf.union(sdf.box(0.4, 0.2, 0.3).rotate(0.1, 0.3, 0.2, 1.4), sdf.cylinder(0.2, 0.5).move(0.3, 0.0, 0.0))
    grid = _lib.Grid(-0.9, -0.8, -0.8, 0.013, 140, 120, 131)
    for t in (tree, stretched):
        with sdf.compile(t) as prog:
            whole = prog.export_mesh(grid, brick=6)
            assert whole.vertices.shape[0] > 1000
            _same(whole, prog.export_mesh(grid, tapes=True))


@pytest.mark.parametrize("prims,ops,grid", [(1, ALL_OPS, 1.0), (30, ALL_OPS, 5.0), (30, ALL_OPS, 16.0), (120, W.OPS_60_20_10_10, 17.0),
                                            (200, ALL_OPS, 33.0)])
def test_voxel_blocks_match_oracle(lib, port, prims, ops, grid):
    """Lattices smaller than a 4^3 box, of whole and of cut 16^3 and 64^3 blocks."""
    seed = 11
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops))):
        seed += 1
    h = port.build(spec)
    try:
        want, size, _ = port.vox(h, grid, 3)
    finally:
        port.free(h)
    with sdf.compile(sdf.from_spec(spec)) as prog:
        vox, gsize, _ = prog.export_voxels(grid, 3)
    np.testing.assert_array_equal(vox, want)
    assert gsize == size


@pytest.mark.parametrize("prims,ops,paint,step,refine", [(200, ALL_OPS, True, (0.021, 0.027, 0.019), 4), (200, W.OPS_60_20_10_10, False, 0.021, 0),
                                                         (100, ALL_OPS, True, 0.02, 1)])
def test_point_cloud_tapes_match_oracle(lib, port, prims, ops, paint, step, refine):
    """Lattices past the size from which the cloud goes by tapes, bricks cut on every axis;
    refined points leave their voxel's brick and its parts on the way."""
    seed = 21
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops, paint=paint))):
        seed += 1
    h = port.build(spec)
    o = port.octree(h)
    try:
        b = port.bounds(h)
        points, cells = port.point_cloud(o, b[:3], b[3:], step, refine)
        normals, colors = port.vertex_attributes(o, points)
    finally:
        port.octree_free(o)
        port.free(h)
    with sdf.compile(sdf.from_spec(spec)) as prog:
        bricks = np.prod(np.ceil((b[3:] - b[:3]) / np.asarray(step) / 8))
        quads = prog.info().distance_quads / prog.info().octree_cells
        assert bricks * (quads - 12) > 45000
        m = prog.export_point_cloud(b[:3], b[3:], step, refine)
    assert points.shape[0] > 1000
    np.testing.assert_array_equal(m.cubes, cells.astype(np.uint32))
    np.testing.assert_array_equal(m.vertices, points)
    np.testing.assert_array_equal(m.normals, normals)
    if paint:
        np.testing.assert_array_equal(m.colors, colors)
    else:
        assert m.colors is None


def _large_cells(prims, ops, paint):
    """A tree with long programs in most of its space: few cells, so few of them were split."""
    seed = 31
    for seed in range(31, 400):
        spec = W.random_tree(seed, prims, ops=ops, paint=paint)
        if not sdf.has_export_octree(sdf.from_spec(spec)):
            continue
        with sdf.compile(sdf.from_spec(spec)) as prog:
            info = prog.info()
        if info.distance_quads >= 100 * info.octree_cells:
            return spec
    raise AssertionError("no such tree")


@pytest.mark.parametrize("prims,ops,large,paint", [(3, ALL_OPS, False, True), (150, ALL_OPS, False, True), (600, W.OPS_60_20_10_10, False, True),
                                                   (400, W.OPS_60_20_10_10, True, True), (400, ALL_OPS, True, True),
                                                   (300, W.OPS_60_20_10_10, True, False)])
def test_render_by_tapes_equals_render_without(lib, prims, ops, large, paint):
    """Enough pixels together go by the root cube's tapes (built by way of larger bricks' where
    the cells are large); the same poses one by one do not.  Odd image sides, a camera inside
    the root cube, one that misses it."""
    if large:
        spec = _large_cells(prims, ops, paint)
    else:
        seed = 31
        while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops))):
            seed += 1
    poses = np.concatenate([W.camera_poses(7, 7), [[0.3, 0.2, 0.1], [60.0, 50.0, 70.0]]]).astype(np.float32)
    with sdf.compile(sdf.from_spec(spec)) as prog:
        depth, normals, colors = prog.render(sdf.cameras(poses), 83, 61)
        assert poses.shape[0] * 83 * 61 >= 32 ** 3 / 4 > 83 * 61 and np.isfinite(depth).any()
        for i, p in enumerate(poses):
            d, n, c = prog.render(sdf.cameras(p[None]), 83, 61)
            np.testing.assert_array_equal(d[0], depth[i])
            np.testing.assert_array_equal(n[0], normals[i])
            np.testing.assert_array_equal(c[0], colors[i])


def _chain(seed, prims):
    """A left-deep tree (a script's n-ary operators fold left): one operator a level."""
    words = []
    rng = W._Words(seed)
    for i in range(prims):
        W._emit_primitive(rng, words, True)
        if i:
            words += [W.UNION] if i % 5 else [W.BLEND_UNION, 0.05]
        if i % 7 == 6:
            words += [W.FLATE, 0.01]
    return np.asarray(words, np.float32)


@pytest.mark.parametrize("spec", [W.random_tree(5, 1), W.random_tree(6, 2), W.random_tree(8, 33, ops=ALL_OPS), W.random_tree(9, 257, ops=ALL_OPS),
                                  _chain(3, 90)], ids=["1", "2", "33", "257", "chain"])
def test_teams_equal_a_thread_each(lib, spec):
    """Whole-tree queries by a block, a warp and a thread each: counts of one, around the
    teams' sizes, and past their limit give the same bits."""
    rng = np.random.default_rng(4)
    many = 70000
    points = rng.uniform(-1.3, 1.3, (many, 3)).astype(np.float32)
    origins = rng.normal(size=(many, 3))
    origins = (4.0 * origins / np.linalg.norm(origins, axis=1, keepdims=True)).astype(np.float32)
    dirs = (rng.uniform(-1, 1, origins.shape) - origins).astype(np.float32)
    with sdf.compile(sdf.from_spec(spec)) as prog:
        values, gradients, (hit, travel, position) = prog.eval_tree(points), prog.gradient_tree(points), prog.ray_march(origins, dirs)
        for n in (1, 2, 31, 160, 1500):
            np.testing.assert_array_equal(prog.eval_tree(points[:n]), values[:n])
            np.testing.assert_array_equal(prog.gradient_tree(points[:n]), gradients[:n])
            h, t, p = prog.ray_march(origins[:n], dirs[:n])
            np.testing.assert_array_equal(h, hit[:n])
            np.testing.assert_array_equal(t, travel[:n])
            np.testing.assert_array_equal(p, position[:n])


@pytest.mark.parametrize("bricks", [(7, 8), (1, 7), (2, 3), (15, 4)])
def test_batch_of_fixture_trees_equals_dense_exports(lib, golden, bricks):
    """Brick blocks and cell passes of every kind of tree (distorting ones are classified a
    brick at a time), bricks with and without a box in shared memory in one batch."""
    specs = [golden[n]["spec"] for n in golden_names() if "octree_nodes" in golden[n]]
    programs = [sdf.compile(sdf.from_spec(s)) for s in specs]
    grids = []
    for i, prog in enumerate(programs):
        info = prog.info()
        lo, hi = np.asarray(info.bounds_min[:]), np.asarray(info.bounds_max[:])
        step = float(np.max(hi - lo)) * 1.1 / (9 + 5 * (i % 7))
        n = [int(np.ceil((h - l) * 1.1 / step)) + 3 for l, h in zip(lo, hi)]
        grids.append(_lib.Grid(*[float(l - 0.05 * (h - l) - step) for l, h in zip(lo, hi)], step, *n))
    with sdf.Batch(programs, grids) as b:
        b.set_tuning([bricks[i % 2] for i in range(len(programs))], [(1, 2, 4)[i % 3] for i in range(len(programs))])
        b.run()
        for m, (prog, grid) in enumerate(zip(programs, grids)):
            _same(b.mesh(m), prog.export_mesh(grid, dense=True))
    for p in programs:
        p.close()


@pytest.mark.parametrize("prims,ops,shape", [(64, ALL_OPS, (257, 193, 209)), (256, W.OPS_60_20_10_10, (241, 999, 50)), (30, ALL_OPS, (1025, 1025, 66)),
                                             (1, ALL_OPS, (353, 320, 300))])
def test_large_lattices_equal_their_pieces(lib, prims, ops, shape):
    """A large lattice (by tapes, in slabs) against small ones cut out of it (by whole
    programs): coordinates are multiples of 2^-7, the same in both, and so are the values."""
    seed = 21
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops))):
        seed += 1
    step = 1.0 / 64.0 if max(shape) < 500 else 1.0 / 128.0
    low = [-round(n * step / 2 / step) * step for n in shape]
    rng = np.random.default_rng(8)
    with sdf.compile(sdf.from_spec(spec)) as prog:
        whole = prog.eval_grid(_lib.Grid(*low, step, *shape))
        for cut in range(24):
            size = [min(n, int(rng.integers(2, 70))) for n in shape]
            at = [0 if cut == 0 else n - s if cut == 1 else int(rng.integers(0, n - s + 1)) for n, s in zip(shape, size)]
            piece = prog.eval_grid(_lib.Grid(*[l + a * step for l, a in zip(low, at)], step, *size))
            np.testing.assert_array_equal(piece, whole[at[2]:at[2] + size[2], at[1]:at[1] + size[1], at[0]:at[0] + size[0]])


@pytest.mark.parametrize("name", golden_names())
def test_point_queries_match_oracle(lib, port, golden, name):
    """Whole-tree values and gradients in counts around a warp's 64 and 16 points, for every
    kind of tree."""
    spec = golden[name]["spec"]
    try:
        prog = sdf.compile(sdf.from_spec(spec))
    except Exception:
        pytest.skip("no octree for this tree")
    rng = np.random.default_rng(6)
    points = rng.uniform(-1.5, 1.5, (20005, 3)).astype(np.float32)
    points[5000:] = points[rng.integers(0, 1500, 15005)]
    handle = port.build(spec)
    values, gradients = port.eval(handle, points), port.gradient(handle, points)
    with prog:
        for n in (1, 15, 16, 17, 63, 65, 20005):
            np.testing.assert_array_equal(prog.eval_tree(points[:n]), values[:n])
            np.testing.assert_array_equal(prog.gradient_tree(points[:n]), gradients[:n])


@pytest.mark.parametrize("log2_table", [14, 15])
def test_gradient_arrays_are_the_callers_own(lib, log2_table):
    """Gradients come in page-locked blocks that the library reuses: not while an array views them."""
    with sdf.Surrogate(log2_table=log2_table) as net:
        rng = np.random.default_rng(2)
        a, b = (np.concatenate([rng.uniform(-1, 1, (n, 3)), rng.uniform(-0.5, 0.5, (n, 1))], 1).astype(np.float32) for n in (700, 300))
        table, mlp, loss = net.gradients(a)
        kept = table.copy(), mlp.copy()
        other = net.gradients(b)
        assert not np.shares_memory(other[0], table) and not np.shares_memory(other[1], mlp)
        np.testing.assert_array_equal(table, kept[0])
        np.testing.assert_array_equal(mlp, kept[1])
        table[:] = 0.0          # writable, and nobody else's
        assert np.any(other[0]) and not np.array_equal(other[1], kept[1])


def _unit(*q):
    q = np.asarray(q, np.float64)
    return [float(v) for v in (q / np.linalg.norm(q)).astype(np.float32)]


def _tilted():
    """A slab whose top crosses z = 0.1 at a slight slant."""
    return sdf.box(0.9, 0.9, 0.5).rotate(*_unit(0.0, 0.02, 0.0, 0.9998)).move(0.0, 0.0, -0.4)


@pytest.mark.parametrize("scale", [1e4, 3e4, 1e5])
def test_brick_tapes_of_large_scales(lib, scale):
    """A brush's own rounding grows with its scale: the top of a unit sphere or box scaled to 1e4
    and more lies in steps of some thousandths, across a slab's that it crosses slowly."""
    grid = _lib.Grid(-0.43, -0.41, -0.1, 0.0021, 410, 391, 150)
    for big in (lambda: sdf.sphere(1.0), lambda: sdf.box(1.0, 0.9, 1.0), lambda: sdf.cylinder(1.0, 1.0)):
        cut = big().rotate(*_unit(0.3, 0.1, 0.2, 0.927)).scale(scale)
        # The brush's extent along z by the tree's own distance: the cut's top goes to 0.1.
        lo, hi = 0.0, 2.0 * scale
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if cut.eval(0.0, 0.0, mid) < 0.0 else (lo, mid)
        tree = sdf.inter(sdf.box(0.4, 0.38, 0.5), sdf.union(cut.move(0.0, 0.0, 0.1 - lo), _tilted()))
        with sdf.compile(tree) as prog:
            whole = prog.export_mesh(grid, staged=True)
            assert whole.vertices.shape[0] > 1000
            _same(whole, prog.export_mesh(grid, tapes=True))


def test_shortened_programs_of_large_steps_between(lib):
    """Operators that go far from the surface and back (a flate by 2e6 and one by -2e6; a blend
    8e6 wide, a quarter of that below its operands, lifted again) leave distances in steps of
    1/8: a step may lie between the points that are looked at and the others."""
    step, n = 1.0 / 256.0, 330
    block = lambda w: sdf.box(w, 0.8, 0.3).rotate(*_unit(0.02, 0.05, 0.3, 1.0))
    slab = lambda: sdf.box(0.7, 0.7, 0.2).rotate(*_unit(0.3, 0.1, 0.2, 1.0))
    for far in (sdf.flate(sdf.flate(block(0.8), 2e6), -2e6), sdf.flate(sdf.blend_union(8e6, block(0.8), block(0.7)), -2e6)):
        with sdf.compile(sdf.diff(sdf.union(far, slab()), sdf.sphere(0.2).move(0.1, 0.1, 0.1))) as prog:
            whole = prog.eval_grid(_lib.Grid(-n // 2 * step, -n // 2 * step, -n // 2 * step, step, n, n, n))
            for z in range(0, n, 55):
                for y in range(0, n, 55):
                    piece = prog.eval_grid(_lib.Grid(-n // 2 * step, (y - n // 2) * step, (z - n // 2) * step, step, n, 55, 55))
                    np.testing.assert_array_equal(piece, whole[z:z + 55, y:y + 55])


def _top_at(make, z):
    """The brush moved along z until its top over the origin is at z, by the tree's own distance."""
    shape, (lo, hi) = make(), (0.0, 1e3)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if shape.eval(0.0, 0.0, mid) < 0.0 else (lo, mid)
    return shape.move(0.0, 0.0, z - lo)


@pytest.mark.parametrize("norm", [0.9992, 1.0009])
@pytest.mark.parametrize("size", [4.0, 40.0])
def test_brick_tapes_of_rotations_off_the_unit(lib, norm, size):
    """Rotations typed with three digits: the distance program's inverse matrix and the surface
    program's inverse quaternion then place a brush some thousandths of its extent apart, and
    the normals are those of the surface program."""
    grid = _lib.Grid(-0.43, -0.41, -0.1, 0.0021, 410, 391, 150)
    for axis in ((0.3, 0.1, 0.2, 0.927), (0.1, -0.2, 0.4, 0.8), (0.05, 0.04, 0.6, 0.8)):
        q = [norm * v for v in _unit(*axis)]
        for lift in (-0.02, 0.0, 0.02):
            big = _top_at(lambda: sdf.box(size, 0.9 * size, size).rotate(*q), 0.1 + lift)
            with sdf.compile(sdf.inter(sdf.box(0.4, 0.38, 0.5), sdf.union(big, _tilted()))) as prog:
                whole = prog.export_mesh(grid, staged=True)
                assert whole.vertices.shape[0] > 1000
                _same(whole, prog.export_mesh(grid, tapes=True))


def _call(kind, prog):
    """A call that goes by tapes or blocks where there is room, and what it returns."""
    if kind == "mesh":
        m = prog.export_mesh(W.export_grid(resolution=150), tapes=True)
        return m.vertices, m.faces, m.cubes, m.normals, m.colors
    if kind == "cloud":
        m = prog.export_point_cloud((-1.6,) * 3, (1.6,) * 3, 0.013, 2)
        return m.vertices, m.cubes, m.normals, m.colors
    if kind == "voxels":
        voxels, size, _ = prog.export_voxels(40.0, 3)
        return voxels, np.asarray(size)
    if kind == "render":
        return prog.render(sdf.cameras(W.camera_poses(7, 2)), 210, 190)
    return (prog.eval_grid(_lib.Grid(-1.6, -1.6, -1.6, 3.2 / 219, 220, 220, 220)),)


CALLS = ("mesh", "cloud", "voxels", "render", "lattice")


@pytest.mark.parametrize("kind", CALLS)
def test_calls_go_without_tapes_where_memory_ends(lib, kind):
    """Device memory that ends at any point of a call: from the least that the call needs on, all
    of it or a part by whole programs, it returns the same."""
    with sdf.compile(sdf.from_spec(W.random_tree(1, 256))) as prog:
        try:
            lib.tg_debug_device_limit(0, 1)
            want = _call(kind, prog)
            full = int(lib.tg_debug_device_limit(0, 0))
            fits = []
            for limit in np.linspace(full // 64, full, 90, dtype=np.int64):
                lib.tg_debug_device_limit(int(limit), 1)
                try:
                    got = _call(kind, prog)
                except _lib.TangerineError:
                    fits.append(False)
                    continue
                fits.append(True)
                for a, b in zip(got, want):
                    np.testing.assert_array_equal(a, b)
        finally:
            lib.tg_debug_device_limit(0, 1)
    least = fits.index(True)
    assert 0 < least < 80       # the limit bites, and the call goes without something
    assert all(fits[least:]), [i for i in range(least, len(fits)) if not fits[i]]


def test_kept_tapes_give_way_to_other_calls(lib):
    """What a call keeps to be faster the next time takes no other call's room."""
    with sdf.compile(sdf.from_spec(W.random_tree(1, 256))) as prog:
        try:
            lib.tg_debug_device_limit(0, 1)
            _call("mesh", prog)
            lib.tg_debug_device_limit(int(lib.tg_debug_device_limit(0, 0)), 0)
            depth, _, _ = prog.render(sdf.cameras(W.camera_poses(7, 1)), 640, 360, exact=True)
            with sdf.compile(sdf.from_spec(W.random_tree(2, 16))) as other:
                assert other.export_mesh(W.export_grid(resolution=32)).vertices.shape[0] > 0
        finally:
            lib.tg_debug_device_limit(0, 1)
    assert np.isfinite(depth).any()


def test_page_locked_results_are_bounded(lib):
    """Blocks for results that callers may keep: at most 2 GB in use, none far larger than asked
    for, and room again once they are given back."""
    C = _lib.C

    def take(size):
        ptr = C.c_void_p()
        return ptr.value if lib.tg_host_take(size, C.byref(ptr)) == 0 else None

    taken = []
    try:
        while len(taken) < 12 and (block := take(200 << 20)):
            taken.append(block)
        assert 8 <= len(taken) <= 10            # an eighth more is pinned than asked for
        lib.tg_host_give(taken[0])
        small = take(1 << 20)
        assert small and small != taken[0]
        assert take(200 << 20) == taken[0]
        lib.tg_host_give(small)
    finally:
        for block in taken:
            lib.tg_host_give(block)


@pytest.mark.parametrize("prims,cells", [(1200, 130), (1500, 150), (1900, 200)])
def test_voxel_blocks_with_full_lists_equal_bricks(lib, prims, cells):
    """Trees with more records in a block than its list holds (all of the tree in one or a few,
    and a far sphere), against the same without room for the blocks' scratch."""
    seed = 11
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims))):
        seed += 1
    tree = sdf.union(sdf.from_spec(spec).scale(0.2), sdf.sphere(0.1).move(1.2, 1.0, 1.1))
    with sdf.compile(tree) as prog:
        info = prog.info()
        grid = cells / float(np.max(np.asarray(info.bounds_max[:]) - np.asarray(info.bounds_min[:])))
        voxels, size, _ = prog.export_voxels(grid, 3)
        blocks, words = int(np.prod([-(-n // 64) for n in size])), int(np.prod(size)) // 4
        try:        # room for the words and their ranks, and for less than the blocks' 41.7 KB each
            lib.tg_debug_device_limit(int(lib.tg_debug_device_limit(0, 1)) + words + blocks * 41000, 0)
            want, want_size, _ = prog.export_voxels(grid, 3)
        finally:
            lib.tg_debug_device_limit(0, 1)
    assert size == want_size and voxels.shape[0] > 500
    np.testing.assert_array_equal(voxels, want)


@pytest.mark.parametrize("whole", [True, False])
def test_voxels_around_the_first_blocks_match_oracle(lib, port, whole):
    """The largest lattices of at most 4096 boxes of 4^3 go box by box, larger ones by blocks."""
    seed = 11
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, 90, ops=ALL_OPS))):
        seed += 1
    with sdf.compile(sdf.from_spec(spec)) as prog:
        def boxes(grid):
            return int(np.prod([-(-n // 4) for n in prog.export_voxels(grid, 3)[1]]))
        grid = 4.0
        while boxes(grid + 0.25) <= 4096:
            grid += 0.25
        grid += 0.0 if whole else 0.25
        voxels, size, _ = prog.export_voxels(grid, 3)
    h = port.build(spec)
    try:
        want, want_size, _ = port.vox(h, grid, 3)
    finally:
        port.free(h)
    assert size == want_size
    np.testing.assert_array_equal(voxels, want)


def _by_whole_programs(lib, room, call):
    """A call with `room` bytes of device memory beside what is held: not enough for tapes."""
    try:
        lib.tg_debug_device_limit(int(lib.tg_debug_device_limit(0, 1)) + room, 0)
        return call()
    finally:
        lib.tg_debug_device_limit(0, 1)


@pytest.mark.parametrize("prims,ops,large,paint", [(24, ALL_OPS, False, True), (150, ALL_OPS, False, True), (600, W.OPS_60_20_10_10, False, True),
                                                   (400, W.OPS_60_20_10_10, True, True), (300, W.OPS_60_20_10_10, True, False)])
def test_render_by_tapes_equals_whole_programs(lib, prims, ops, large, paint):
    """The same images with room for the tapes (by way of larger bricks' where the cells are
    large) and without.  Odd image sides, a camera inside the root cube, one that misses it."""
    seed = 31
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops, paint=paint))):
        seed += 1
    if large:
        spec = _large_cells(prims, ops, paint)
    width, height = 83, 61
    poses = np.concatenate([W.camera_poses(7, 7), [[0.3, 0.2, 0.1], [60.0, 50.0, 70.0]]]).astype(np.float32)
    pixels = len(poses) * width * height
    assert lib.tg_debug_goes_by_tapes(sdf.from_spec(spec).handle, 3, None, pixels) == 1
    with sdf.compile(sdf.from_spec(spec)) as prog:
        images = prog.render(sdf.cameras(poses), width, height)
        want = _by_whole_programs(lib, 19 * pixels + (1 << 20), lambda: prog.render(sdf.cameras(poses), width, height))
    assert np.isfinite(images[0]).any()
    for a, b in zip(images, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("prims,ops,shape", [(5, ALL_OPS, (353, 320, 300)), (64, ALL_OPS, (257, 193, 209)), (64, ALL_OPS, (15, 633, 641)),
                                             (200, W.OPS_60_20_10_10, (33, 17, 9000)), (200, ALL_OPS, (1601, 16, 241)), (90, ALL_OPS, (129, 3001, 14)),
                                             (100, ALL_OPS, (1025, 1025, 66)), (500, ALL_OPS, (190, 191, 193))])
def test_lattices_by_tapes_equal_whole_programs(lib, prims, ops, shape):
    """Lattices with remainders of bricks on every axis, one brick thin on some, in one and in
    several slabs, by levels one and two at a time: with room for the tapes and without."""
    seed = 21
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops))):
        seed += 1
    steps = [3.2 / n for n in shape]
    grid = _lib.Grid(-1.6, -1.6, -1.6, steps[0], *shape, steps[1], steps[2])
    assert lib.tg_debug_goes_by_tapes(sdf.from_spec(spec).handle, 1, C.byref(grid), 0) == 1
    with sdf.compile(sdf.from_spec(spec)) as prog:
        lattice = prog.eval_grid(grid)
        want = _by_whole_programs(lib, 4 * int(np.prod(shape)) + (1 << 18), lambda: prog.eval_grid(grid))
    np.testing.assert_array_equal(lattice, want)


@pytest.mark.parametrize("prims,ops,paint,step,refine", [(200, ALL_OPS, True, (0.014, 0.017, 0.012), 4), (200, W.OPS_60_20_10_10, False, 0.013, 0),
                                                         (100, ALL_OPS, True, 0.012, 1), (20, ALL_OPS, True, 0.011, 6)])
def test_clouds_by_tapes_equal_whole_programs(lib, prims, ops, paint, step, refine):
    """The same points, normals and colours with room for the tapes and without; bricks cut on
    every axis, refined points that leave their voxel's brick and its parts on the way."""
    seed = 21
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ops, paint=paint))):
        seed += 1
    step = [float(v) for v in np.broadcast_to(np.asarray(step, np.float32), (3,))]
    with sdf.compile(sdf.from_spec(spec)) as prog:
        info = prog.info()
        lo, hi = np.asarray(info.bounds_min[:]), np.asarray(info.bounds_max[:])
        shape = [int(np.ceil((h - l) / s)) for l, h, s in zip(lo, hi, step)]
        grid = _lib.Grid(*[float(v) for v in lo], step[0], *shape, step[1], step[2])
        assert lib.tg_debug_goes_by_tapes(sdf.from_spec(spec).handle, 2, C.byref(grid), 0) == 1
        cloud = prog.export_point_cloud(lo, hi, step, refine)
        count = cloud.vertices.shape[0]
        want = _by_whole_programs(lib, int(4.5 * np.prod(shape)) + 31 * count + (1 << 20), lambda: prog.export_point_cloud(lo, hi, step, refine))
    assert count > 1000
    for a, b in ((cloud.vertices, want.vertices), (cloud.cubes, want.cubes), (cloud.normals, want.normals)):
        np.testing.assert_array_equal(a, b)
    assert (cloud.colors is None) == (want.colors is None) == (not paint)
    if paint:
        np.testing.assert_array_equal(cloud.colors, want.colors)


@pytest.mark.parametrize("kind", CALLS)
@pytest.mark.parametrize("parts,events", [(1, 1), (100, 0), (3001, 0), (0, 100), (0, 5003)])
def test_calls_with_little_room_for_tapes(lib, kind, parts, events):
    """Bricks whose parts and parts whose events found no room go by whole programs."""
    with sdf.compile(sdf.from_spec(W.random_tree(1, 256))) as prog:
        want = _call(kind, prog)
        lib.tg_debug_tape_room(parts, events)
        try:
            got = _call(kind, prog)
        finally:
            lib.tg_debug_tape_room(0, 0)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


def test_more_long_parts_than_are_listed(lib):
    """A tree whose few cells all have long programs, and more bricks than the list of long parts
    holds (16384): the others are built in their turn."""
    blends = ((W.UNION, 0.3), (W.DIFF, 0.2), (W.INTER, 0.05), (W.BLEND_UNION, 0.25), (W.BLEND_DIFF, 0.1), (W.BLEND_INTER, 0.1))
    seed = 6
    while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, 256, ops=blends))):
        seed += 7919
    n = 430
    grid = _lib.Grid(-1.6, -1.6, -1.6, 3.2 / n, n, n, n)
    with sdf.compile(sdf.from_spec(spec)) as prog:
        info = prog.info()
        assert info.octree_cells <= 4 and info.distance_quads > 300 * info.octree_cells
        lattice = prog.eval_grid(grid)
        want = _by_whole_programs(lib, 4 * n ** 3 + (1 << 18), lambda: prog.eval_grid(grid))
    np.testing.assert_array_equal(lattice, want)


def test_queries_at_special_points(lib, port):
    """Zeros, denormal, huge and infinite coordinates, NaN: the oracle's values by a block, a warp
    and half a lane a point."""
    v = np.asarray([0, -0.0, 1e-40, -1e-30, 1e10, -1e30, 3e38, np.inf, -np.inf, np.nan, 0.3, -0.7], np.float32)
    points = np.stack(np.meshgrid(v, v, v, indexing="ij"), -1).reshape(-1, 3)
    for prims in (1, 3, 60):
        seed = 4
        while not sdf.has_export_octree(sdf.from_spec(spec := W.random_tree(seed, prims, ops=ALL_OPS))):
            seed += 1
        handle = port.build(spec)
        try:
            values, gradients = port.eval(handle, points), port.gradient(handle, points)
        finally:
            port.free(handle)
        with sdf.compile(sdf.from_spec(spec)) as prog:
            for n in (100, 1728, 40000):
                np.testing.assert_array_equal(prog.eval_tree(np.resize(points, (n, 3))), np.resize(values, n))
                np.testing.assert_array_equal(prog.gradient_tree(np.resize(points, (n, 3))), np.resize(gradients, (n, 3)))


def test_culled_exports_of_deflated_trees_equal_dense(lib):
    """The reference's bounds of a flate by a negative radius are too small by it: the surface leaves
    the octree's cube, by way of the compiled program, the root's alone (export_tree) and a batch."""
    def trees():
        yield sdf.flate(sdf.union(sdf.sphere(0.5), sdf.box(0.4, 0.3, 0.6).move(0.2, 0.1, 0.0)), -0.08)
        yield sdf.union(sdf.flate(sdf.torus(0.5, 0.2).rotate(0.6, 0.0, 0.0, 0.8), -0.03).scale(1.3), sdf.sphere(0.2).move(0.1, 0.0, 0.0))
        yield sdf.flate(sdf.flate(sdf.blend_union(0.1, sdf.cylinder(0.4, 0.5), sdf.sphere(0.3).move(0.3, 0.2, 0.1)), 0.02), -0.06).paint(0.2, 0.4, 0.6)
    lo, hi, step = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0), 0.011
    programs = [sdf.compile(t) for t in trees()]
    grid = sdf.export_grid(lo, hi, step)
    for tree, prog in zip(trees(), programs):
        dense = prog.export_mesh(grid, dense=True)
        info = prog.info()
        assert (dense.vertices.max(0) > np.asarray(info.bounds_max[:])).any()
        for brick in (3, 7, 16):
            _same(dense, prog.export_mesh(grid, brick=brick))
        _same(dense, prog.export_mesh(grid, tapes=True))
        _same(dense, sdf.export_tree(tree, lo, hi, step))
    with sdf.Batch(programs, [grid] * len(programs)) as batch:
        batch.run()
        for i, prog in enumerate(programs):
            _same(prog.export_mesh(grid, dense=True), batch.mesh(i))
    for prog in programs:
        prog.close()


def _deflated(seed, prims=8):
    """Few brushes with flates by negative radii at any depth."""
    rng = np.random.default_rng(seed)
    def build(n):
        if n == 1:
            a, b, c = (float(v) for v in rng.uniform(0.2, 0.6, 3))
            t = (sdf.sphere(a), sdf.box(a, b, c), sdf.cylinder(a, b))[int(rng.integers(3))].move(*[float(v) for v in rng.uniform(-0.8, 0.8, 3)])
        else:
            m = int(rng.integers(1, n))
            l, r = build(m), build(n - m)
            x = rng.uniform()
            t = sdf.union(l, r) if x < 0.5 else sdf.diff(l, r) if x < 0.7 else sdf.inter(l, r) if x < 0.8 else sdf.blend_union(0.1, l, r)
        return sdf.flate(t, float(rng.uniform(-0.1, -0.02))) if rng.uniform() < 0.3 else t
    return build(prims)


@pytest.mark.parametrize("seed", [20, 74, 121, 159, 220, 351])
def test_culled_exports_below_negative_flates_equal_dense(lib, seed):
    """Below a negative flate the octree's clips hold in less than their sphere: cells that hold a
    brick's ball by less than that decide nothing about it.  All cells where the tree's own sign
    changes are kept, whatever the bricks (the clip's errors put others into the dense mesh)."""
    with sdf.compile(_deflated(seed)) as prog:
        grid = sdf.export_grid((-1.5, -1.5, -1.5), (1.5, 1.5, 1.5), 0.02)
        dense = prog.export_mesh(grid, dense=True)
        _same(dense, prog.export_mesh(grid))
        _same(dense, prog.export_mesh(grid, tapes=True))
        c = dense.cubes.astype(np.int64)
        at = np.stack([c % (grid.nx - 1), c // (grid.nx - 1) % (grid.ny - 1), c // ((grid.nx - 1) * (grid.ny - 1))], 1)
        corners = at[:, None] + np.asarray(list(np.ndindex(2, 2, 2)))
        points = (np.float32([grid.x0, grid.y0, grid.z0]) + corners.astype(np.float32) * np.float32(grid.step)).reshape(-1, 3)
        inside = (prog.eval_tree(points) < 0).reshape(-1, 8)
        surface = dense.cubes[inside.any(1) & ~inside.all(1)]
        for brick in (2, 4, 15, 32):
            assert np.isin(surface, prog.export_mesh(grid, brick=brick).cubes).all()
