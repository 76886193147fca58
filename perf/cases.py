"""The work a user of the framework has it do, as cases that can be timed.

Every case is a call through the public Python face (tangerine_gb300.sdf) or, for images
rendered into device memory, through the C ABI below it.  The models are the repository's
seeded random CSG trees (tangerine_gb300.workloads.random_tree: spheres, boxes, tori and
cylinders joined by union, difference, intersection and blended union), the lattices its
export grids over [-2, 2]^3.  A case names its kind and its sizes:

  export_tree   the whole export a modeller runs: tree handle in, host mesh out
  mesh_device   a compiled model exported again (another resolution, another pass of a
                pipeline) to a mesh that stays on the GPU
  eval_grid     the dense distance lattice, for consumers that want the field itself
  gradient      whole-tree gradients at scattered points (scripts, physics queries)
  rays          exact whole-tree ray casts: picking in the editor, one ray or a viewport of them
  render        depth, normal and colour images of camera poses
  batch         many independent models exported by one launch (an asset library)
  sodapop       the editor's interactive meshing of a model at a density
  cloud         point-cloud export with refinement
  voxels        MagicaVoxel export
  net           one training gradient (forward and backward) of the learned distance bound
"""

import math

import numpy as np
import torch

from tangerine_gb300 import _lib, sdf
from tangerine_gb300 import workloads as W

BOX = ((-2.0, -2.0, -2.0), (2.0, 2.0, 2.0))
CLOUD_BOX = ((-1.6, -1.6, -1.6), (1.6, 1.6, 1.6))
RAY_STEPS, RAY_EPSILON = 100, 1e-3          # the ray casts' defaults
RENDER_STEPS, RENDER_EPSILON = 256, 1e-4    # the benchmark's render settings
LEVELS, NET_PARAMS = 16, 10497              # the learned bound's hash levels and network size


def listed():
    return [
        # A small model at the coarse setting used while modelling: launches and latency.
        {"name": "export_tree_16_128", "kind": "export_tree", "prims": 16, "res": 128},
        # The benchmark's headline export, tree to host mesh.
        {"name": "export_tree_256_512", "kind": "export_tree", "prims": 256, "res": 512},
        # The largest export: a detailed model at production resolution, mesh kept on the GPU.
        {"name": "mesh_device_256_1024", "kind": "mesh_device", "prims": 256, "res": 1024},
        # A ragged dense lattice with a step per axis.
        {"name": "eval_grid_64_301", "kind": "eval_grid", "prims": 64, "nx": 301, "ny": 257, "nz": 193},
        # Gradients at a hundred thousand scattered points.
        {"name": "gradient_64_100k", "kind": "gradient", "prims": 64, "count": 100003},
        # The editor's mouse pick: a single ray.
        {"name": "pick_64_1", "kind": "rays", "prims": 64, "count": 1},
        # Two full-HD views of a large scene.
        {"name": "render_1024_2x1080p", "kind": "render", "prims": 1024, "width": 1920, "height": 1080, "poses": 2},
        # An asset library: mixed sizes of model and lattice.
        {"name": "batch_32", "kind": "batch", "models": 32, "max_prims": 512, "max_res": 256},
        # The editor's own meshing at its default density.
        {"name": "sodapop_256_20", "kind": "sodapop", "prims": 256, "density": 20.0},
        # A fine point cloud with the default five refinement steps.
        {"name": "cloud_256_0.01", "kind": "cloud", "prims": 256, "step": 0.01, "refine": 5},
        # Voxels at 64 a unit.
        {"name": "voxels_256_64", "kind": "voxels", "prims": 256, "grid_size": 64.0},
        # One training batch of the learned bound at its default table and batch size.
        {"name": "net_gradient_2e18", "kind": "net", "log2_table": 18, "count": 262144},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["export_tree", "mesh_device", "eval_grid", "gradient", "rays", "render", "batch", "sodapop", "cloud", "voxels",
                       "net"])
    if kind in ("export_tree", "mesh_device"):
        return {"kind": kind, "prims": _log(rng, 8, 256), "res": _log(rng, 48, 800)}
    if kind == "eval_grid":
        return {"kind": kind, "prims": _log(rng, 8, 256), "nx": _log(rng, 20, 320), "ny": _log(rng, 20, 320), "nz": _log(rng, 20, 320)}
    if kind == "gradient":
        return {"kind": kind, "prims": _log(rng, 8, 256), "count": _log(rng, 1, 200000)}
    if kind == "rays":
        return {"kind": kind, "prims": _log(rng, 8, 128), "count": _log(rng, 1, 16384)}
    if kind == "render":
        return {"kind": kind, "prims": _log(rng, 8, 1024), "width": _log(rng, 200, 1920), "height": _log(rng, 150, 1080),
                "poses": rng.randint(1, 2)}
    if kind == "batch":
        return {"kind": kind, "models": rng.randint(2, 32), "max_prims": _log(rng, 16, 512), "max_res": rng.choice([64, 128, 192, 256])}
    if kind == "sodapop":
        return {"kind": kind, "prims": _log(rng, 8, 256), "density": round(rng.uniform(5.0, 24.0), 2)}
    if kind == "cloud":
        return {"kind": kind, "prims": _log(rng, 8, 256), "step": round(math.exp(rng.uniform(math.log(0.01), math.log(0.08))), 5),
                "refine": rng.randint(0, 6)}
    if kind == "voxels":
        return {"kind": kind, "prims": _log(rng, 8, 256), "grid_size": float(rng.randint(6, 64))}
    return {"kind": kind, "log2_table": rng.randint(14, 18), "count": _log(rng, 500, 262144)}


# ---- models and inputs ------------------------------------------------------------------

def _valid(spec):
    return sdf.has_export_octree(sdf.from_spec(spec))


def _spec(prims, seed):
    """A seeded tree that leaves something to export (intersections can leave nothing)."""
    tree_seed = (1000003 * (seed % 2000) + prims) & 0x7FFFFFFF
    while not _valid(spec := W.random_tree(tree_seed, prims)):
        tree_seed += 7919
    return spec


def _painted(spec, seed):
    """The tree with every primitive's paint drawn from the seed."""
    rng = np.random.default_rng(seed)
    spec, i = spec.copy(), 0
    while i < spec.size:
        op = int(spec[i])
        if op == W.PAINT:
            spec[i + 1:i + 4] = rng.random(3, dtype=np.float32)
        i += 1 + W.ARITY[op]
    return spec


# A mesh's size follows the model's geometry, and passes over several seeds return the same
# shapes: the mesh kinds' geometry is the benchmark's model of that size, and the seed paints it.
MODEL_SEED = 1


def _points(case, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1.25, 1.25, (case["count"], 3)).astype(np.float32)


def _rays(case, seed):
    """Casts from around the model toward it."""
    rng = np.random.default_rng(seed)
    o = rng.normal(size=(case["count"], 3))
    o = (4.0 * o / np.linalg.norm(o, axis=1, keepdims=True)).astype(np.float32)
    return o, (rng.uniform(-1.0, 1.0, o.shape) - o).astype(np.float32)


def _net_inputs(case, seed):
    """Table and network values of a bound in training, and samples (x, y, z, distance)."""
    rng = np.random.default_rng(seed)
    table = rng.uniform(-0.3, 0.3, LEVELS * 2 * (1 << case["log2_table"])).astype(np.float32)
    mlp = np.zeros(NET_PARAMS, np.float32)
    at = 0
    for rows, cols in ((64, 32), (64, 64), (64, 64), (1, 64)):
        limit = math.sqrt(6.0 / (rows + cols))
        mlp[at:at + rows * cols] = rng.uniform(-limit, limit, rows * cols)
        mlp[at + rows * cols:at + rows * cols + rows] = rng.uniform(-0.05, 0.05, rows)
        at += rows * cols + rows
    n = case["count"]
    samples = np.concatenate([rng.uniform(-2.0, 2.0, (n, 3)), rng.uniform(-0.5, 0.5, (n, 1))], 1).astype(np.float32)
    return table, mlp, samples


def _lattice(case):
    """A lattice over the model with a step per axis."""
    n = [case["nx"], case["ny"], case["nz"]]
    step = [np.float32(3.2 / (k - 1)) for k in n]
    return _lib.Grid(-1.6, -1.6, -1.6, float(step[0]), n[0], n[1], n[2], float(step[1]), float(step[2]))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "net":
        table, mlp, s["samples"] = _net_inputs(case, seed)
        s["net"] = sdf.Surrogate(log2_table=case["log2_table"])
        s["net"].set_params(table, mlp)
        return s
    if kind == "batch":
        res = tuple(r for r in W.BATCH_RESOLUTIONS if r <= case["max_res"])
        load = W.batch_workload(MODEL_SEED, case["models"], max_prims=case["max_prims"], resolutions=res, valid=_valid)
        programs = [sdf.compile(sdf.from_spec(_painted(W.random_tree(t, p), seed + i))) for i, (t, p, _) in enumerate(load)]
        s["batch"] = sdf.Batch(programs, [W.export_grid(resolution=r) for _, _, r in load])
        return s
    if kind in ("eval_grid", "gradient", "rays", "render"):
        tree = sdf.from_spec(_spec(case["prims"], seed))
    else:
        tree_seed = MODEL_SEED
        while not _valid(spec := W.random_tree(tree_seed, case["prims"])):
            tree_seed += 7919
        tree = sdf.from_spec(_painted(spec, seed))
    if kind in ("export_tree", "sodapop"):
        s["tree"] = tree
        return s
    s["program"] = sdf.compile(tree)
    if kind == "mesh_device":
        s["grid"] = W.export_grid(resolution=case["res"])
    elif kind == "eval_grid":
        s["grid"] = _lattice(case)
        s["out"] = torch.empty(case["nz"], case["ny"], case["nx"], dtype=torch.float32, device="cuda")
    elif kind == "voxels":
        s["color"] = 1 + seed % 255
    elif kind == "gradient":
        s["points"] = _points(case, seed)
    elif kind == "rays":
        s["rays"] = _rays(case, seed)
    elif kind == "render":
        s["cameras"] = sdf.cameras(W.camera_poses(seed % 100000, case["poses"]))
        px = case["poses"] * case["height"] * case["width"]
        s["images"] = (torch.empty(px, dtype=torch.float32, device="cuda"), torch.empty(px, 3, dtype=torch.float32, device="cuda"),
                       torch.empty(px, 3, dtype=torch.uint8, device="cuda"))
    return s


# ---- one pass ---------------------------------------------------------------------------

class _DeviceArray:
    """A block of the library's device memory; keeps its owner alive while tensors view it."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _device(owner, ptr, shape, typestr, dtype):
    if not ptr or not shape[0]:
        return torch.empty((0,) + shape[1:], dtype=dtype, device="cuda")
    return torch.as_tensor(_DeviceArray(owner, ptr, shape, typestr), device="cuda")


def _device_mesh(owner, m, vertices, faces):
    return {"vertices": _device(owner, m.vertices, (vertices, 3), "<f4", torch.float32),
            "normals": _device(owner, m.normals, (vertices, 3), "<f4", torch.float32),
            "colors": _device(owner, m.colors, (vertices, 3), "|u1", torch.uint8),
            "faces": _device(owner, m.faces, (faces, 3), "<i4", torch.int32),
            "cubes": _device(owner, m.cubes, (vertices,), "<i4", torch.int32)}


def _host_mesh(m):
    return {"vertices": m.vertices, "normals": m.normals, "colors": m.colors, "faces": m.faces.view(np.int32),
            "cubes": m.cubes.view(np.int32)}


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "export_tree":
        return _host_mesh(sdf.export_tree(s["tree"], *BOX, 4.0 / case["res"]))
    if kind == "mesh_device":
        m = s["program"].export_mesh_device(s["grid"])
        return _device_mesh(s["program"], m, int(m.vertex_count), int(m.face_count))
    if kind == "eval_grid":
        s["program"].eval_grid_device(s["grid"], s["out"].data_ptr())
        return s["out"]
    if kind == "gradient":
        return s["program"].gradient_tree(s["points"])
    if kind == "rays":
        hit, travel, position = s["program"].ray_march(*s["rays"], iterations=RAY_STEPS, epsilon=RAY_EPSILON)
        return {"hit": hit, "travel": travel, "position": position}
    if kind == "render":
        depth, normals, colors = s["images"]
        ptr = _lib.C.c_void_p
        _lib.check(_lib.load().tg_render(s["program"].ptr, s["cameras"], case["poses"], case["width"], case["height"], RENDER_STEPS,
                                         RENDER_EPSILON, 0, ptr(depth.data_ptr()), ptr(normals.data_ptr()), ptr(colors.data_ptr()), 1,
                                         None), "tg_render")
        return {"depth": depth, "normals": normals, "colors": colors}
    if kind == "batch":
        s["batch"].run()
        # The models' meshes lie one after the other: all of them from the first one's start.
        info = s["batch"].info()
        return _device_mesh(s["batch"], s["batch"].mesh_device(0), int(info.vertices), int(info.faces))
    if kind == "sodapop":
        d = s["tree"].sodapop_mesh(case["density"])
        return {"positions": d.positions, "normals": d.normals, "colors": d.colors, "faces": d.faces.view(np.int32),
                "cells": d.cells.view(np.int32), "grid": d.grid}
    if kind == "cloud":
        m = s["program"].export_point_cloud(*CLOUD_BOX, case["step"], case["refine"])
        return {"vertices": m.vertices, "normals": m.normals, "colors": m.colors, "cubes": m.cubes.view(np.int32)}
    if kind == "voxels":
        voxels, size, radius = s["program"].export_voxels(case["grid_size"], s["color"])
        return {"voxels": voxels, "size": list(size), "radius": radius}
    table, mlp, loss = s["net"].gradients(s["samples"])
    return {"table": table, "mlp": mlp, "loss": loss}


# ---- what a pass cannot do without ------------------------------------------------------

BRUSH_FLOPS = 45                # a 3x4 transform and a primitive's distance


def _area(prims):
    """Surface area of the models, in square units: seeded trees of these sizes measure about this."""
    return 25.0 if prims < 32 else 50.0 if prims < 128 else 75.0


def work(case):
    kind = case["kind"]
    if kind in ("export_tree", "mesh_device"):
        # A vertex, its normal, colour and cell, and two triangles per lattice cell on the
        # surface; one distance and the gradient's four and the colour's one evaluation each.
        n = _area(case["prims"]) * (case["res"] / 4.0) ** 2
        return {"bytes": 55 * n, "flops": 6 * BRUSH_FLOPS * n}
    if kind == "eval_grid":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4 * n, "flops": BRUSH_FLOPS * n}
    if kind == "gradient":
        return {"bytes": 24 * case["count"], "flops": 4 * BRUSH_FLOPS * case["prims"] * case["count"]}
    if kind == "rays":
        return {"bytes": 41 * case["count"], "flops": 10 * BRUSH_FLOPS * case["prims"] * case["count"]}
    if kind == "render":
        n = case["poses"] * case["width"] * case["height"]
        return {"bytes": 19 * n, "flops": 5 * BRUSH_FLOPS * n}
    if kind == "batch":
        res = [r for r in W.BATCH_RESOLUTIONS if r <= case["max_res"]]
        n = case["models"] * 40.0 * sum((r / 4.0) ** 2 for r in res) / len(res)
        return {"bytes": 55 * n, "flops": 6 * BRUSH_FLOPS * n}
    if kind == "sodapop":
        n = _area(case["prims"]) * case["density"] ** 2
        return {"bytes": 68 * n, "flops": 5 * BRUSH_FLOPS * n}
    if kind == "cloud":
        n = 1.2 * _area(case["prims"]) / case["step"] ** 2
        return {"bytes": 31 * n, "flops": (6 + 5 * case["refine"]) * BRUSH_FLOPS * n}
    if kind == "voxels":
        n = 1.2 * _area(case["prims"]) * case["grid_size"] ** 2
        return {"bytes": 16 * n, "flops": BRUSH_FLOPS * n}
    # Samples in, table in, table and network gradients out; three passes of the products.
    return {"bytes": 16 * case["count"] + 2 * 4 * LEVELS * 2 * (1 << case["log2_table"]) + 8 * NET_PARAMS,
            "flops": 6 * (32 * 64 + 64 * 64 + 64 * 64 + 64) * case["count"]}


# ---- the same in 64 bits ----------------------------------------------------------------

def _rotate(q, v):
    """Rows of v rotated by the quaternion (x, y, z, w), whatever its norm's rounding."""
    u, w = q[:3], q[3]
    uv = torch.linalg.cross(u.expand_as(v), v)
    return v + 2.0 * (uv * w + torch.linalg.cross(u.expand_as(v), uv))


def _quaternion_product(a, b):
    ax, ay, az, aw = a
    bx, by, bz, bw = b
    return (aw * bx + ax * bw + ay * bz - az * by, aw * by + ay * bw + az * bx - ax * bz,
            aw * bz + az * bw + ax * by - ay * bx, aw * bw - ax * bx - ay * by - az * bz)


def _brush(op, prm, q, t, p):
    n = sum(x * x for x in q)
    inverse = torch.tensor([-q[0] / n, -q[1] / n, -q[2] / n, q[3] / n], dtype=torch.float64, device=p.device)
    v = _rotate(inverse, p - torch.tensor(t, dtype=torch.float64, device=p.device))
    if op == W.SPHERE:
        return v.norm(dim=1) - prm[0]
    if op == W.BOX:
        a = v.abs() - torch.tensor(prm, dtype=torch.float64, device=p.device)
        return a.clamp(min=0.0).norm(dim=1) + a.max(dim=1).values.clamp(max=0.0)
    ring = v[:, :2].norm(dim=1)
    if op == W.TORUS:
        return torch.hypot(ring - prm[0], v[:, 2]) - prm[1]
    a = torch.stack([ring - prm[0], v[:, 2].abs() - prm[1]], 1)
    return a.max(dim=1).values.clamp(max=0.0) + a.clamp(min=0.0).norm(dim=1)


def _parse(spec):
    """The spec as a postfix list of brushes (op, parameters, rotation, translation) and set
    operators; the transforms of a random tree follow its brushes."""
    out, i, words = [], 0, [float(v) for v in spec]
    while i < len(words):
        op = int(words[i])
        a = words[i + 1:i + 1 + W.ARITY[op]]
        i += 1 + len(a)
        if op in (W.SPHERE, W.BOX, W.TORUS, W.CYLINDER):
            out.append([op, a, (0.0, 0.0, 0.0, 1.0), [0.0, 0.0, 0.0]])
        elif op == W.ROTATE:
            out[-1][2] = _quaternion_product(a, out[-1][2])
        elif op == W.MOVE:
            out[-1][3] = [x + y for x, y in zip(out[-1][3], a)]
        elif op in (W.UNION, W.DIFF, W.INTER, W.BLEND_UNION):
            out.append([op, a])
    return out


def _distance(tree, p):
    stack = []
    for e in tree:
        if len(e) == 4:
            stack.append(_brush(*e, p))
            continue
        r, l = stack.pop(), stack.pop()
        if e[0] == W.UNION:
            d = torch.minimum(l, r)
        elif e[0] == W.INTER:
            d = torch.maximum(l, r)
        elif e[0] == W.DIFF:
            d = torch.maximum(l, -r)
        else:
            h = (e[1][0] - (l - r).abs()).clamp(min=0.0)
            d = torch.minimum(l, r) - h * h * 0.25 / e[1][0]
        stack.append(d)
    return stack[0]


def _exact_gradient(case, seed):
    tree = _parse(_spec(case["prims"], seed))
    p = torch.from_numpy(_points(case, seed)).cuda().double()
    h = float(np.float32(0.0001))
    g = torch.zeros_like(p)
    for corner in ((h, -h, -h), (-h, -h, h), (-h, h, -h), (h, h, h)):
        k = torch.tensor(corner, dtype=torch.float64, device="cuda")
        g += k * _distance(tree, p + k)[:, None]
    return (g / g.norm(dim=1, keepdim=True)).cpu().numpy()


def _exact_rays(case, seed):
    tree = _parse(_spec(case["prims"], seed))
    o, d = (torch.from_numpy(a).cuda().double() for a in _rays(case, seed))
    d = d / d.norm(dim=1, keepdim=True)
    travel = torch.zeros(o.shape[0], dtype=torch.float64, device="cuda")
    hit = torch.zeros(o.shape[0], dtype=torch.bool, device="cuda")
    for _ in range(RAY_STEPS):
        f = _distance(tree, o + d * travel[:, None])
        hit |= f <= RAY_EPSILON
        travel = torch.where(hit, travel, travel + f)
    position = o + d * travel[:, None]
    return {"hit": None, "travel": torch.where(hit, travel, math.inf).cpu().numpy(), "position": position.cpu().numpy()}


def _exact_net(case, seed):
    """The bound's gradient by automatic differentiation: hash-grid encoding (Mueller et al.
    2022) with the cells picked in float32 as any float32 caller would, then the 32-64-64-64-1
    network and the mean squared error against the clamped distances."""
    table, mlp, samples = _net_inputs(case, seed)
    size = 1 << case["log2_table"]
    lo, hi, base, top, clamp = np.float32(-2.0), np.float32(2.0), 16, 1024, 0.5      # the default options
    unit = np.clip((samples[:, :3] - lo) * (np.float32(1.0) / (hi - lo)), np.float32(0.0), np.float32(1.0)).astype(np.float32)
    u = torch.from_numpy(unit).cuda()
    t = torch.from_numpy(table).cuda().double().reshape(LEVELS, size, 2).requires_grad_()
    m = torch.from_numpy(mlp).cuda().double().requires_grad_()
    growth = math.exp((math.log(top) - math.log(base)) / (LEVELS - 1))
    features = []
    for level in range(LEVELS):
        res = int(math.floor(base * growth ** level + 1e-6))
        x = u * float(res)
        c = x.floor().long().clamp(0, res - 1)
        f = (x - c.float()).double()
        blend = 0.0
        for k in range(8):
            d = (k & 1, (k >> 1) & 1, k >> 2)
            cx, cy, cz = (c[:, a] + d[a] for a in range(3))
            if (res + 1) ** 3 <= size:
                at = cx + (res + 1) * (cy + (res + 1) * cz)
            else:
                at = (cx ^ (cy * 2654435761) ^ (cz * 805459861)) & (size - 1)
            w = math.prod(f[:, a] if d[a] else 1.0 - f[:, a] for a in range(3))
            blend = blend + w[:, None] * t[level][at]
        features.append(blend)
    h, at = torch.cat(features, 1), 0
    for rows, cols in ((64, 32), (64, 64), (64, 64), (1, 64)):
        w = m[at:at + rows * cols].reshape(rows, cols)
        b = m[at + rows * cols:at + rows * cols + rows]
        at += rows * cols + rows
        h = h @ w.T + b
        if rows > 1:
            h = h.relu()
    target = torch.from_numpy(samples[:, 3]).cuda().double().clamp(-clamp, clamp)
    squared = (h[:, 0] - target).square()
    squared.mean().backward()
    return {"table": t.grad.reshape(-1).cpu().numpy(), "mlp": m.grad.cpu().numpy(), "loss": float(squared.sum())}


def exact(case, seed):
    """Gradients, ray casts and the bound's gradient have values in 64 bits.  The others do
    not: an export's lattice, voxels, mesh and refined points follow the octree's clipped
    programs in float32 (which operand a cell keeps, which cells the surface crosses and where
    an iteration stops all hang on float32 comparisons), and so do a bounded render's steps."""
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    if case["kind"] == "rays":
        return _exact_rays(case, seed)
    if case["kind"] == "net":
        return _exact_net(case, seed)
    return None
