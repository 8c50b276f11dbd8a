"""The work this library is measured on: the calls that a cloth simulation makes of it.

The reference-format calls build a tree from the step's triangles and query it, as a caller
of the reference extension does in every step (the tree is rebuilt because the triangles
move).  The engine cases keep their meshes, trees and captured step, as its users do.  All
inputs are this repository's seeded workloads (``cccollisions_b200.workloads``) at their own
sizes and at sizes around them.

The library returns collision rows in the order its thread blocks finish, padded with -1 up
to the capacity.  A caller takes the rows that are there; here they are put in mesh order
(first triangle, second triangle, sub-test, time) in place, so that two runs can be compared.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cccollisions_b200 as C
from cccollisions_b200 import _native, workloads as W
from cccollisions_b200.engine import Engine
from cccollisions_b200.serve import Request, Server

# capacities per triangle of the full-size workloads: no candidate and no row is dropped
CANDIDATES, ROWS = 32, 16
# distinct continuous sub-tests per triangle of the cloth over the sphere, and of the folds,
# whose layers interpenetrate; double-precision operations of one (coefficients, cubic, filter)
SUBTESTS = {"cloth_sphere": 16, "fold": 40}
SUBTEST_FLOPS = 252
DEV = "cuda:0"


def listed():
    return [
        # one garment panel in a simulation loop: the smallest call, all launch latency
        dict(name="panel_impulses", kind="impulses", n=23, batch=1, dtype="float64"),
        # the crumpled 64 x 64 cloth folded through itself: self-intersections of a pose
        dict(name="pose_intersections", kind="intersections", n=64, batch=1, dtype="float32", threshold=0.0),
        # self-proximity of a larger pose, as a repulsion force asks for it
        dict(name="pose_proximity", kind="proximity", n=121, batch=1, dtype="float32", threshold=0.002),
        # intersection contours of a pose (edges crossing triangles), in double precision
        dict(name="pose_contour", kind="contour", n=75, batch=1, dtype="float64"),
        # the 128 x 128 cloth dropped on a level-5 icosphere: one continuous step
        dict(name="cloth_sphere", kind="continuous", nx=128, ny=128, level=5, batch=1, dtype="float64", masked=0.0),
        # a batch of equal garments in single precision, re-checked where they were corrected
        dict(name="batch_recheck", kind="continuous", nx=61, ny=47, level=3, batch=6, dtype="float32", masked=0.3),
        # the 256 x 256 fold: impulses of one step of a large cloth
        dict(name="fold_impulses", kind="impulses", n=256, batch=1, dtype="float64"),
        # impulses of collision rows that the caller kept (and filtered) from an earlier query
        dict(name="kept_rows", kind="kept_rows", n=129, batch=1, dtype="float32"),
        # the resident engine on a handful of small meshes: a captured step, latency bound
        dict(name="engine_few", kind="step", meshes=5, lo=300, hi=3000, level=2, dtype="float32", rebuild=False),
        # topology changed: trees built again, then a step that was not captured
        dict(name="engine_rebuild", kind="step", meshes=12, lo=1000, hi=50000, level=4, dtype="float64", rebuild=True),
        # the batched workload: 64 cloth-over-sphere meshes of 1e3 to 1e5 cloth triangles
        dict(name="engine_batched", kind="step", meshes=64, lo=1000, hi=100000, level=5, dtype="float64",
             rebuild=False),
        # impulse requests served to convergence (folds whose layers start apart)
        dict(name="served", kind="served", requests=10, lo=2000, hi=50000, dtype="float64"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    dtype = rng.choice(["float32", "float64"])
    kind = rng.choice(["impulses", "intersections", "proximity", "contour", "continuous", "kept_rows", "step", "served"])
    if kind == "continuous":
        return dict(kind=kind, nx=size(20, 128), ny=size(20, 128), level=rng.randint(2, 5), batch=rng.choice([1, 1, 2, 3]),
                    dtype=dtype, masked=rng.choice([0.0, 0.0, 0.1, 0.5]))
    if kind == "step":
        # (cloth much finer than the 0.005 it is jittered by collides with itself in more rows
        # than the capacity holds, unless the sphere's triangles make up for it)
        lo, level = size(200, 2000), rng.randint(1, 5)
        return dict(kind=kind, meshes=size(2, 40), lo=lo, hi=min(lo * size(2, 50), 100000 if level == 5 else 15000),
                    level=level, dtype=dtype, rebuild=rng.random() < 0.3)
    if kind == "served":
        lo = size(500, 5000)
        return dict(kind=kind, requests=size(2, 10), lo=lo, hi=lo * size(2, 10), dtype=dtype)
    n = size(20, 256 if kind == "impulses" else 160)
    case = dict(kind=kind, n=n, batch=rng.choice([1, 1, 2, 4]) if n < 100 else 1, dtype=dtype)
    if kind in ("intersections", "proximity"):
        case["threshold"] = rng.choice([0.0, 0.005]) if kind == "intersections" else rng.choice([0.001, 0.002])
    return case


# ---------------------------------------------------------------------------------------
# sizes

def _spread(case, count):
    """Triangle counts of `count` meshes, even over the logarithm of [lo, hi], small and large
    mixed, and the grids (nx, ny) closest to them with the aspects 0.6, 0.9, 1.3, 1.8 in turn."""
    out = []
    for i in range(count):
        u = ((i * 7) % count + 0.5) / count
        cells = case["lo"] * (case["hi"] / case["lo"]) ** u / 2
        nx = max(2, round(math.sqrt(cells * (0.6, 0.9, 1.3, 1.8)[i % 4])))
        out.append((nx + 1, max(2, round(cells / nx)) + 1))
    return out


def _grid_triangles(nx, ny):
    return 2 * (nx - 1) * (ny - 1)


def _triangles(case):
    """Triangles of one pass."""
    if case["kind"] == "step":
        return sum(_grid_triangles(*g) + 20 * 4 ** case["level"] for g in _spread(case, case["meshes"]))
    if case["kind"] == "served":
        return sum(_grid_triangles(*g) for g in _spread(case, case["requests"]))
    if case["kind"] == "continuous":
        return case["batch"] * (_grid_triangles(case["nx"], case["ny"]) + 20 * 4 ** case["level"])
    return case["batch"] * _grid_triangles(case["n"], case["n"])


def work(case):
    t, b, kind = _triangles(case), 4 if case["dtype"] == "float32" else 8, case["kind"]
    tree = (2 * t) * (6 * b + 4 * 8)                      # boxes and tree rows written by the build
    soup, corner_sums = 9 * b * t, (2 * 9 * b + 3 * 4) * t
    subtests = SUBTESTS["cloth_sphere" if kind in ("continuous", "step") else "fold"] * t
    if kind == "impulses":
        return dict(bytes=2 * soup + 3 * b * t + tree + corner_sums, flops=subtests * SUBTEST_FLOPS)
    if kind == "continuous":
        share = case["masked"] or 1.0
        return dict(bytes=2 * soup + tree + t * ROWS * (24 + b), flops=share * subtests * SUBTEST_FLOPS)
    if kind == "intersections":
        return dict(bytes=soup + tree + t * ROWS * 16, flops=6 * 400 * t)
    if kind == "proximity":
        return dict(bytes=soup + tree + t * ROWS * 24, flops=6 * 900 * t)
    if kind == "contour":
        return dict(bytes=soup + tree + t * ROWS * (32 + b), flops=6 * 600 * t)
    if kind == "kept_rows":
        rows = 4 * t
        return dict(bytes=rows * (24 + b) + 2 * soup + 3 * b * t + corner_sums, flops=rows * 300)
    if kind == "step":
        return dict(bytes=2 * soup + 3 * t * (24 + b), flops=subtests * SUBTEST_FLOPS)
    # served: a check and a correction an iteration, some 20 of them
    return dict(bytes=20 * (2 * soup + 3 * b * t), flops=20 * subtests * SUBTEST_FLOPS)


# ---------------------------------------------------------------------------------------
# inputs

def _gpu(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV).to(getattr(torch, dtype))


def _fold_meshes(case, seed):
    """Batched jittered folds: x0, x1 (B, F, 3, 3) and unequal corner masses (B, F, 3)."""
    parts = [W.impulse_fold(seed=1000 * seed + b, n=case["n"]) for b in range(case["batch"])]
    x0, x1 = (_gpu(np.concatenate([p[k] for p in parts]), case["dtype"]) for k in (0, 1))
    mass = W.rng(seed).uniform(0.5, 2.0, parts[0][2].shape[1:])
    return x0, x1, _gpu(np.stack([mass] * case["batch"]), case["dtype"])


def prepare(case, seed):
    kind, dtype = case["kind"], case["dtype"]
    state = dict(case=case)
    if kind in ("intersections", "proximity", "contour"):
        poses = [W.static_fold(seed=1000 * seed + b, n=case["n"], dtype=np.float64) for b in range(case["batch"])]
        state["x0"] = _gpu(np.concatenate(poses), dtype)
    elif kind == "impulses":
        state["x0"], state["x1"], state["mass"] = _fold_meshes(case, seed)
    elif kind == "kept_rows":
        x0, x1, mass = state["x0"], state["x1"], state["mass"] = _fold_meshes(case, seed)
        bboxes, tree = C.bvh_motion(x0, x1)
        rows, times = C.find_collisions_continuous(bboxes, tree, x0, x1, CANDIDATES, ROWS)
        # every second collision in mesh order, as (B, N) padded with -1
        kept = [[v[::2] for v in _mesh_order(r, t, (x0.shape[1],) * 2)] for r, t in _rows_there(rows, times)]
        most = max(max(r.shape[0] for r, _ in kept), 1)
        state["rows"] = torch.full((len(kept), most, 3), -1, dtype=torch.int64, device=DEV)
        state["times"] = torch.full((len(kept), most, 1), -1.0, dtype=x0.dtype, device=DEV)
        for b, (r, t) in enumerate(kept):
            state["rows"][b, :len(r)], state["times"][b, :len(r), 0] = r, t
    elif kind == "continuous":
        parts = [W.cloth_sphere(seed=1000 * seed + b, nx=case["nx"], ny=case["ny"], level=case["level"])
                 for b in range(case["batch"])]
        state["x0"], state["x1"] = (_gpu(np.concatenate([p[k] for p in parts]), dtype) for k in (0, 1))
        if case["masked"]:
            shape = tuple(state["x0"].shape[:2])
            state["mask"] = torch.from_numpy(W.rng(seed).random(shape) < case["masked"]).to(DEV)
    elif kind == "step":
        meshes = [W.cloth_sphere(seed=1000 * seed + i, nx=nx, ny=ny, level=case["level"])
                  for i, (nx, ny) in enumerate(_spread(case, case["meshes"]))]
        sizes = state["sizes"] = [x0.shape[1] for x0, _ in meshes]
        eng = state["engine"] = Engine(tri_capacity=sum(sizes), mesh_capacity=len(sizes), dtype=getattr(torch, dtype),
                                       max_candidates_per_triangle=CANDIDATES, max_collisions_per_triangle=ROWS)
        sids = state["sids"] = [eng.add_mesh(f) for f in sizes]
        for sid, (x0, x1) in zip(sids, meshes):
            eng.upload_soup(sid, x0[0], x1[0])
        eng.set_active(sids)
        eng.build(sids)
        state["base"] = torch.tensor(np.cumsum([0] + sizes[:-1]), dtype=torch.int64, device=DEV)
        state["packed"] = (torch.full((sum(sizes) * ROWS, 3), -1, dtype=torch.int64, device=DEV),
                           torch.full((sum(sizes) * ROWS,), -1.0, dtype=eng.dtype, device=DEV),
                           torch.empty(2 * len(sizes) + 2, dtype=torch.int32, device=DEV))
        if not case["rebuild"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                eng.capture(_native.ENGINE_OP_CCD, stream=side)
    elif kind == "served":
        state["server"] = Server(budget_bytes=4 << 30, dtype=getattr(torch, dtype))
        np_dtype = np.dtype(dtype).type
        state["requests"] = [
            Request(*W.impulse_fold_mesh(1000 * seed + i, nx, ny, dtype=np_dtype, **W.SEPARATED_FOLD), rid=i)
            for i, (nx, ny) in enumerate(_spread(case, case["requests"]))]
    return state


# ---------------------------------------------------------------------------------------
# one pass

def _rows_there(rows, times=None):
    """Views of each mesh's (rows, times) without the -1 padding, which follows them."""
    count = (rows[:, :, 0] >= 0).sum(1).tolist()
    return [(rows[b, :n], None if times is None else times[b, :n, 0]) for b, n in enumerate(count)]


def _mesh_order(rows, times, ids):
    """Rows (i, j, sub-test) in the order of their columns, then of their times; `ids`: what
    the first and second column stay below."""
    key = rows[:, 0] * ids[1] + rows[:, 1]
    if rows.shape[1] > 2:
        key = key * 16 + rows[:, 2]
    if times is None:
        return rows[torch.sort(key)[1]], None
    spare = 62 - (ids[0] * ids[1] * 16).bit_length()
    key = (key << spare) + (times.double() * ((1 << spare) - 1)).long()
    key, order = torch.sort(key)
    rows, times = rows[order], times[order]
    # roots of one sub-test too close for the key's spare bits: the earlier first
    key >>= spare
    tie = (key[1:] == key[:-1]) & (times[1:] < times[:-1])
    first = torch.where(tie, times[1:], times[:-1])
    times[1:] = torch.where(tie, times[:-1], times[1:])
    times[:-1] = first
    return rows, times


def _contour_order(rows, coefs, ids):
    order = torch.sort((rows[:, 0] * ids[1] + rows[:, 1]) * 16 + rows[:, 2])[1]
    return rows[order], coefs[order]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("intersections", "proximity", "contour"):
        x0 = state["x0"]
        bboxes, tree = C.bvh(x0)
        ids = (x0.shape[1],) * 2
        if kind == "contour":
            rows, coefs = C.find_triangle_edge_collisions(bboxes, tree, x0, max_collisions=ROWS)
            for r, c in _rows_there(rows, coefs):
                r[:], c[:] = _contour_order(r, c, ids)
            return dict(bboxes=bboxes, tree=tree, rows=rows, coefs=coefs)
        if kind == "intersections":
            rows = C.find_collisions(bboxes, tree, x0, threshold=case["threshold"], max_collisions=ROWS)
        else:
            (rows,) = C.find_proximity(bboxes, tree, x0, case["threshold"], ROWS)
        for r, _ in _rows_there(rows):
            r[:], _ = _mesh_order(r, None, ids)
        return dict(bboxes=bboxes, tree=tree, rows=rows)
    if kind == "impulses":
        bboxes, tree = C.bvh_motion(state["x0"], state["x1"])
        dv, dx, count = C.compute_impulses(bboxes, tree, state["x0"], state["x1"], state["mass"], CANDIDATES, ROWS)
        return dict(bboxes=bboxes, tree=tree, dv=dv, dx=dx, count=count)
    if kind == "kept_rows":
        dv, dx, count = C.compute_impulses_from_collisions(state["rows"], state["times"], state["x0"], state["x1"],
                                                           state["mass"])
        return dict(dv=dv, dx=dx, count=count)
    if kind == "continuous":
        x0, x1 = state["x0"], state["x1"]
        bboxes, tree = C.bvh_motion(x0, x1)
        if "mask" in state:
            rows, times = C.find_collisions_continuous_partial(bboxes, tree, x0, x1, state["mask"], CANDIDATES, ROWS)
        else:
            rows, times = C.find_collisions_continuous(bboxes, tree, x0, x1, CANDIDATES, ROWS)
        for r, t in _rows_there(rows, times):
            r[:], t[:] = _mesh_order(r, t, (x0.shape[1],) * 2)
        return dict(bboxes=bboxes, tree=tree, rows=rows, times=times)
    if kind == "step":
        eng, sids = state["engine"], state["sids"]
        rows, times, meta = state["packed"]
        if case["rebuild"]:
            eng.build(sids)
            eng.ccd()
        else:
            eng.replay(_native.ENGINE_OP_CCD)
        eng.pack_rows(rows, times, meta)
        at = meta.tolist()
        meshes = len(sids)
        if at[-1]:
            raise RuntimeError(f"engine status {at[-1]:#x}")
        total = at[meshes]
        base = torch.repeat_interleave(state["base"], torch.diff(meta[:meshes + 1]), output_size=total)
        # the first column numbers the batch's triangles, so that one sort orders every mesh
        rows[:total, 0] += base
        rows[:total], times[:total] = _mesh_order(rows[:total], times[:total], (_triangles(case), max(state["sizes"])))
        return dict(offsets=meta[:meshes + 1], rows=rows, times=times)
    stats = state["server"].run(state["requests"], realtime=False)
    done = state["requests"]
    return dict(verts=np.concatenate([r.verts1_out for r in done]),
                iterations=np.array([r.iterations for r in done]), requests=stats["requests"])


# ---------------------------------------------------------------------------------------
# the same in 64 bits, without the library

def exact(case, seed):
    """Boxes and impulses in 64 bits.  The collision rows, their times and what follows from
    them have no such value: which sub-tests have a row hangs on the last bits of the
    reference's cubic solver, which the library repeats operation by operation."""
    kind = case["kind"]
    if kind in ("step", "served"):
        return None
    state = prepare(case, seed)
    host = {k: v.cpu().numpy().astype(np.float64) for k, v in state.items() if k in ("x0", "x1", "mass", "times")}
    if kind == "kept_rows":
        return _exact_impulses(state["rows"].cpu().numpy(), **host)
    x0 = host["x0"]
    lo, hi = x0.min(2), x0.max(2)
    if "x1" in host:
        lo, hi = np.minimum(lo, host["x1"].min(2)), np.maximum(hi, host["x1"].max(2))
    out = dict(bboxes=np.stack([_tree_boxes(np.concatenate([a, b], 1)) for a, b in zip(lo, hi)]), tree=None)
    if kind == "impulses":
        return dict(out, dv=None, dx=None, count=None)
    return dict(out, rows=None, **({} if kind in ("intersections", "proximity") else
                                   {"coefs" if kind == "contour" else "times": None}))


def _tree_boxes(leaf):
    """Boxes of the radix tree over the positions 0 .. n - 1 (Karras 2012; the keys are the
    positions themselves): n - 1 internal nodes, then the n leaves."""
    n = len(leaf)
    i = np.arange(n - 1)

    def prefix(j):
        bits = np.frexp((i ^ np.clip(j, 0, n - 1)).astype(np.float64))[1]
        return np.where((j < 0) | (j > n - 1), -1, 64 - bits)

    d = np.where(prefix(i + 1) >= prefix(i - 1), 1, -1)
    least = prefix(i - d)
    length = np.zeros(n - 1, np.int64)
    step = 1 << int(n).bit_length()
    while step:
        length += step * (prefix(i + (length + step) * d) > least)
        step >>= 1
    first, last = np.minimum(i, i + length * d), np.maximum(i, i + length * d)
    # minima and maxima of the ranges [first, last] from those of 2^k leaves
    level = np.frexp((last - first + 1).astype(np.float64))[1] - 1
    box, table = np.empty((n - 1, 6)), np.concatenate([leaf[:, :3], -leaf[:, 3:]], 1)
    for k in range(int(level.max()) + 1):
        at = level == k
        box[at] = np.minimum(table[first[at]], table[last[at] + 1 - (1 << k)])
        table[:n - (1 << k)] = np.minimum(table[:n - (1 << k)], table[1 << k:])
    box[:, 3:] *= -1
    return np.concatenate([box, leaf])


def _exact_impulses(rows, x0, x1, mass, times):
    """Impulses of given collisions: the contact's points, normal and normal velocity, then the
    velocity change of the four corners that keeps the pair's momentum."""
    dv, dx, count = np.zeros_like(x0), np.zeros_like(x0), np.zeros(mass.shape, np.int32)
    edges = ((0, 1), (0, 2), (1, 2))

    def dot(a, b):
        return (a * b).sum(-1)

    for b in range(len(rows)):
        for k in range(15):
            at = rows[b, :, 2] == k
            i, j, t = rows[b, at, 0], rows[b, at, 1], times[b, at]
            if k < 9:           # edge against edge
                points = [(i, c) for c in edges[k // 3]] + [(j, c) for c in edges[k % 3]]
            elif k < 12:        # face of the first against a vertex of the second
                points = [(i, 0), (i, 1), (i, 2), (j, k - 9)]
            else:               # face of the second against a vertex of the first
                points = [(j, 0), (j, 1), (j, 2), (i, k - 12)]
            x = [x0[b, tri, c] for tri, c in points]
            move = [x1[b, tri, c] - x0[b, tri, c] for tri, c in points]
            m = [mass[b, tri, c] for tri, c in points]
            p = [a + v * t for a, v in zip(x, move)]
            if k < 9:
                da, db, dc = p[1] - p[0], p[3] - p[2], p[2] - p[0]
                n = np.cross(da, db)
                flat = dot(n, n) < 1e-15
                with np.errstate(all="ignore"):
                    s = np.where(flat, 0.5, dot(np.cross(dc, db), n) / dot(n, n))
                    r = np.where(flat, 0.5, dot(np.cross(dc, da), n) / dot(n, n))
                first, second, side = [1 - s, s, 0 * s, 0 * s], [0 * r, 0 * r, 1 - r, r], (0, 0, 1, 1)
            else:
                e1, e2, ep = p[0] - p[1], p[2] - p[1], p[3] - p[1]
                d00, d01, d11, d20, d21 = dot(e1, e1), dot(e1, e2), dot(e2, e2), dot(ep, e1), dot(ep, e2)
                area = d00 * d11 - d01 * d01
                flat = np.abs(area) < 1e-15
                with np.errstate(all="ignore"):
                    u = np.where(flat, 1 / 3, (d11 * d20 - d01 * d21) / area)
                    w = np.where(flat, 1 / 3, (d00 * d21 - d01 * d20) / area)
                first, second, side = [u, 1 - u - w, w, 0 * u], [0 * u, 0 * u, 0 * u, 1 + 0 * u], (0, 0, 0, 1)

            def blend(weights, values):
                return sum((q[:, None] if v.ndim > 1 else q) * v for q, v in zip(weights, values))

            normal = np.cross(p[1] - p[0], p[2] - p[0])
            normal /= np.sqrt(dot(normal, normal))[:, None]
            normal *= np.where(dot(blend(second, x) - blend(first, x), normal) < 0, -1, 1)[:, None]
            speed = dot(blend(second, move) - blend(first, move), normal)
            m0, m1 = blend(first, m), blend(second, m)
            with np.errstate(all="ignore"):
                early = np.clip(np.where(np.abs(speed) < 1e-15, 0.1, 4e-3 / -speed), 0, 1)
            keep = 1 - np.maximum(t[:, 0] - early, 0)
            for (tri, c), one in zip(points, side):
                change = normal * (-speed * m0 if one else speed * m1)[:, None] / (m0 + m1)[:, None]
                np.add.at(dv[b, :, c], tri, change)
                np.add.at(dx[b, :, c], tri, change * keep[:, None])
                np.add.at(count[b, :, c], tri, 1)
    return dict(dv=dv, dx=dx, count=None)
