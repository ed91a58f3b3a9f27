"""Performance cases of the GMorpho path, each through the public Python API
(`broxy_gb300.api`): voxelization, closing, meshing, the host-buffer update,
the frame field and its closing, the batched form and the edit server.

Solids are the benchmark's sums of 200 Gaussian blobs classified at level
0.5, sampled on the box that the blobs fill with a small margin (a mesh is
fitted to its box the same way).  Radii are the benchmark's field
r = 2 + floor(30 s(x)) at 1024 fine voxels per axis and as large against the
solid on other grids, or a uniform radius within that range.
"""
import math
import os
import re

import numpy as np
import torch

import broxy_gb300
from broxy_gb300 import _lib as L
from broxy_gb300 import api, synth

_ROWS = 12  # rows kept for a mesh's vertices, per squared fine edge of its grid (twice that for its triangles)
_MARGIN = 0.05  # world units added around a mesh's box
_SPAN = (0.06, 0.94)  # the part of the unit cube that the blob solids are sampled on


def listed():
    return [
        # 64 icospheres (82k triangles) into 128^3: the smallest load
        {"name": "voxelize_spheres_128", "kind": "voxelize", "shape": "spheres", "count": 64, "level": 3, "res": 64},
        # the benchmark's 4.0M-triangle isosurface into 1024^3: a large load
        {"name": "voxelize_iso_1024", "kind": "voxelize", "shape": "iso", "samples": 672, "res": 512},
        # one update of a small grid, launch-bound: closing, mesh, 20 filter iterations
        {"name": "update_128_r4", "kind": "update", "res": 64, "radius": 4, "iters": 20},
        # closing at the benchmark's middle size and uniform radius
        {"name": "close_512_r12", "kind": "close", "res": 256, "radius": 12, "se": "sphere", "mode": "ref"},
        # the headline closing: 1024^3 with a radius per voxel
        {"name": "close_1024_field", "kind": "close", "res": 512, "radius": 0, "se": "sphere", "mode": "ref"},
        # a ragged box (slab, crop) with the cube element and the one-level mode
        {"name": "close_box_cube_exact", "kind": "box", "rx": 208, "ry": 144, "rz": 272, "radius": 0, "se": "cube",
         "mode": "exact"},
        # meshing of the closed 1024^3 grid with the 20 filter iterations
        {"name": "mesh_1024", "kind": "mesh", "res": 512, "iters": 20},
        # a whole update of host buffers, copies included
        {"name": "update_host_512", "kind": "update_host", "res": 256, "radius": 0, "filter": True},
        # the frame field's solve on the lattice of a 1024^3 grid
        {"name": "frame_field_32", "kind": "frame_field", "n": 32, "points": 4},
        # the frame-field closing
        {"name": "rotcube_512_field", "kind": "rotcube", "res": 256, "qres": 16, "radius": 0},
        # many uneven grids in one call
        {"name": "batch_16", "kind": "batch", "count": 16, "hi": 384, "lanes": 4},
        # brush edits on a resident grid: painted, then reset
        {"name": "serve_1024", "kind": "serve", "res": 512, "edits": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["voxelize", "voxelize", "update", "close", "close", "box", "mesh", "mesh", "update_host",
                       "frame_field", "rotcube", "batch", "serve"])
    se, mode = rng.choice(["sphere", "sphere", "cube"]), rng.choice(["ref", "ref", "exact"])
    res = rng.choice([64, 128, 256, 512])
    radius = rng.choice([0, _log(rng, 2, max(4, res // 16))])
    if kind == "voxelize":
        if rng.random() < 0.5:
            return {"kind": kind, "shape": "spheres", "count": _log(rng, 8, 96), "level": rng.choice([2, 3, 4]),
                    "res": rng.choice([64, 128, 256])}
        return {"kind": kind, "shape": "iso", "samples": _log(rng, 60, 560), "res": res}
    if kind == "update":
        return {"kind": kind, "res": min(res, 256), "radius": radius, "iters": rng.randint(1, 30)}
    if kind == "close":
        return {"kind": kind, "res": res, "radius": radius, "se": se, "mode": mode}
    if kind == "box":
        return {"kind": kind, "rx": 16 * _log(rng, 3, 26), "ry": 16 * _log(rng, 3, 26), "rz": 16 * _log(rng, 3, 26),
                "radius": radius, "se": se, "mode": mode}
    if kind == "mesh":
        return {"kind": kind, "res": res, "iters": rng.randint(0, 24)}
    if kind == "update_host":
        return {"kind": kind, "res": min(res, 256), "radius": radius, "filter": rng.random() < 0.8}
    if kind == "frame_field":
        return {"kind": kind, "n": _log(rng, 6, 36), "points": rng.randint(1, 20)}
    if kind == "rotcube":
        return {"kind": kind, "res": min(res, 256), "qres": _log(rng, 3, 32), "radius": min(radius, 16)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 16), "hi": 32 * rng.randint(4, 12),
                "lanes": rng.choice([1, 4, 8])}
    return {"kind": kind, "res": rng.choice([128, 256]), "edits": rng.randint(2, 16)}


# ------------------------------------------------------------------ inputs

def _solid(dims, seed, level=0.5):
    """Packed grid (dims = cells x, y, z) of the blob solid, its longest edge
    spanning _SPAN on every axis."""
    centres, sigmas, weights = synth.blob_params(seed)
    big = max(dims)
    c, s, w = (torch.as_tensor(a, device="cuda") for a in (centres, sigmas, weights))

    def axis(a):
        n = 2 * dims[a]
        x = _SPAN[0] + (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * (_SPAN[1] - _SPAN[0]) / (2 * big)
        return torch.exp(-(x[None, :] - c[:, a:a + 1]) ** 2 / (2 * s[:, None] ** 2))

    gx, gy, gz = axis(0) * w[:, None], axis(1), axis(2)
    out = torch.empty((dims[2], dims[1], dims[0]), dtype=torch.uint8, device="cuda")
    for z in range(0, dims[2], 8):
        occ = torch.einsum("kz,ky,kx->zyx", gz[:, 2 * z:2 * z + 16], gy, gx) >= level
        n = occ.shape[0] // 2
        o = occ.reshape(n, 2, dims[1], 2, dims[0], 2).to(torch.uint8)
        acc = torch.zeros((n, dims[1], dims[0]), dtype=torch.uint8, device="cuda")
        for k in range(8):
            acc |= o[:, k >> 2, :, (k >> 1) & 1, :, k & 1] << k
        out[z:z + n] = acc
    return out.reshape(-1)


def _radii(dims, seed):
    """The benchmark's radius field on a box of cells, its largest radius in
    proportion to the box."""
    span = max(4, 30 * max(dims) // 512)
    centres, widths, amps = synth.radius_params(seed)
    c, s, a = (torch.as_tensor(v, device="cuda") for v in (centres, widths, amps))

    def axis(k):
        n = 2 * dims[k]
        x = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
        return torch.exp(-(x[None, :] - c[:, k:k + 1]) ** 2 / (2 * s[:, None] ** 2))

    gx, gy, gz = axis(0) * a[:, None], axis(1), axis(2)
    out = torch.empty((2 * dims[2], 2 * dims[1], 2 * dims[0]), dtype=torch.int8, device="cuda")
    for z in range(0, 2 * dims[2], 16):
        f = torch.einsum("kz,ky,kx->zyx", gz[:, z:z + 16], gy, gx)
        out[z:z + 16] = (2 + torch.floor(span * f.clamp(0.0, 1.0))).to(torch.int8)
    return out.reshape(-1)


def _quats(n, seed):
    """A smooth field of unit quaternions on the n^3 lattice (x fastest)."""
    rng = np.random.default_rng(seed)
    x = np.stack(np.meshgrid(*([np.arange(n) / n] * 3), indexing="ij"), -1).reshape(-1, 3)[:, ::-1]
    axis = np.sin(x @ rng.uniform(-4, 4, (3, 3)) + rng.uniform(0, 6, 3)) + rng.normal(size=3)
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    half = 0.5 * (0.8 + 0.6 * np.sin(x @ rng.uniform(-3, 3, 3) + rng.uniform(0, 6)))
    q = np.concatenate([np.sin(half)[:, None] * axis, np.cos(half)[:, None]], 1)
    return torch.as_tensor(q.astype(np.float32), device="cuda")


def _constraints(case, seed):
    """Hard-constrained lattice nodes (distinct) and their twists."""
    rng = np.random.default_rng(seed)
    n, k = case["n"], case["points"]
    node = rng.choice(n ** 3, size=k, replace=False)
    pos = np.stack([node % n, node // n % n, node // (n * n)], 1) + 0.5
    twist = rng.normal(size=(k, 3))
    twist *= rng.uniform(0.2, 2.5, (k, 1)) / np.linalg.norm(twist, axis=1, keepdims=True)
    return node, (pos / n).astype(np.float32), twist.astype(np.float32)


def _instances(case, seed):
    """The benchmark's uneven grids, their edges and radii the case's own and
    their solids the seed's."""
    plan = synth.batch_instances(case["count"] + case["hi"], case["count"], 64, case["hi"], device="cuda")
    for i, g in enumerate(plan):
        E = g["edge"]
        X = torch.zeros((g["res"],) * 3, dtype=torch.uint8, device="cuda")
        X[:E // 2, :E // 2, :E // 2] = _solid((E // 2,) * 3, seed * 100 + i).view((E // 2,) * 3)
        g["X"] = X.reshape(-1)
        g["radius"] = min(g["radius"], max(2, E // 16))
    return plan


def _keep_mesh(s, n, **where):
    """The program's own copy of a mesh (the context's lasts until its next
    mesh), with room for any mesh of such a grid."""
    s["V"], s["N"] = (torch.zeros((_ROWS * n * n, 3), dtype=torch.float32, **where) for _ in range(2))
    s["T"] = torch.zeros((2 * _ROWS * n * n, 3), dtype=torch.int32, **where)
    return s


def _kept(s, mesh):
    V, N, T = mesh
    s["V"][:V.shape[0]].copy_(V)
    s["N"][:N.shape[0]].copy_(N)
    s["T"][:T.shape[0]].copy_(T.view(torch.int32))
    return {"V": s["V"], "N": s["N"], "T": s["T"], "vertices": V.shape[0], "triangles": T.shape[0]}


_context = None


def _ctx():
    """The context that a program keeps for its lifetime."""
    global _context
    if _context is None:
        _context = api.Context(0)
    return _context


def _se(case):
    return L.GM_SE_CUBE if case.get("se") == "cube" else L.GM_SE_SPHERE


def _mode(case):
    return L.GM_EXACT if case.get("mode") == "exact" else L.GM_REF


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case, "ctx": _ctx()}
    if kind == "voxelize":
        if case["shape"] == "spheres":
            P, T = synth.spheres_mesh(seed, case["count"], case["level"])
            P, T = torch.as_tensor(P, device="cuda"), torch.as_tensor(T.astype(np.int32), device="cuda")
        else:
            P, T = synth.blob_mesh(case["samples"], seed)
        ends = torch.stack([P.amin(0), P.amax(0)]).cpu().numpy()  # the box is all that the attributes read
        s["desc"] = api.grid_attributes(ends, case["res"], _MARGIN)
        s["P"], s["T"] = P, T
        s["out"] = torch.zeros(case["res"] ** 3, dtype=torch.uint8, device="cuda")
    elif kind in ("close", "update", "rotcube", "box"):
        dims = (case["rx"], case["ry"], case["rz"]) if kind == "box" else (case["res"],) * 3
        s["X"] = _solid(dims, seed)
        s["R"] = _radii(dims, seed) if case["radius"] == 0 else None
        s["out"] = torch.empty_like(s["X"])
        s["desc"] = api.make_box(dims, cell_size=1.0 / max(dims)) if kind == "box" else api.make_desc(case["res"])
        if kind == "update":
            _keep_mesh(s, 2 * case["res"], device="cuda")
        if kind == "rotcube":
            s["Q"] = _quats(case["qres"], seed)
    elif kind == "mesh":
        s["C"] = _solid((case["res"],) * 3, seed)
        s["desc"] = api.make_desc(case["res"])
        _keep_mesh(s, 2 * case["res"], device="cuda")
    elif kind == "update_host":
        dims = (case["res"],) * 3
        s["X"] = _solid(dims, seed).cpu().pin_memory()
        s["R"] = _radii(dims, seed).cpu().pin_memory() if case["radius"] == 0 else None
        s["desc"] = api.make_desc(case["res"])
        _keep_mesh(s, 2 * case["res"], pin_memory=True)
    elif kind == "frame_field":
        _, pos, twist = _constraints(case, seed)
        s["ff"] = api.FrameField(s["ctx"], (0.0,) * 3, (1.0,) * 3, case["n"])
        for p, t in zip(pos, twist):
            s["ff"].add_point(p, t)
    elif kind == "batch":
        s["ctx"] = api.Context(0)  # its lanes and captured work belong to this set of grids
        s["items"], s["meshes"] = [], []
        for g in _instances(case, seed):
            s["items"].append((api.make_desc(g["res"], g["data_res"]), g["X"], None, g["radius"],
                               torch.empty_like(g["X"])))
            s["meshes"].append(_keep_mesh({}, 2 * g["res"], device="cuda"))
    elif kind == "serve":
        res = case["res"]
        rng = np.random.default_rng(seed)
        desc, cs = api.make_desc(res), 0.5 / res
        R = torch.full(((2 * res) ** 3,), 8, dtype=torch.int8, device="cuda")
        s["server"] = api.Server(desc, _solid((res,) * 3, seed), R, slots=4, max_crop_res=min(res, 512), rmax=32)
        s["R"], s["edits"] = R, []
        for _ in range(case["edits"]):
            reach = float(rng.uniform(16, min(128, res / 2)))
            r = int(rng.integers(8, 33))
            core = min(r, reach - 1)
            support = (core + (reach - core) * math.sqrt(1 - math.sqrt(0.5))) * cs
            s["edits"].append((rng.uniform(0.2, 0.8, 3), r * cs, support))
        s["base"] = 8.5 * cs
    else:
        raise ValueError(kind)
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["kind"]
    if kind == "voxelize":
        return ctx.voxelize(s["desc"], s["P"], s["T"], out=s["out"])
    if kind == "close":
        return ctx.close(s["desc"], s["X"], s["R"], case["radius"], _mode(case), _se(case), out=s["out"])
    if kind == "box":
        return ctx.close_box(s["desc"], s["X"], s["R"], case["radius"], _mode(case), _se(case), out=s["out"])
    if kind == "rotcube":
        return ctx.close_rotcube(s["desc"], s["X"], s["Q"], case["qres"], s["R"], case["radius"], out=s["out"])
    if kind == "update":
        C = ctx.close(s["desc"], s["X"], s["R"], case["radius"], out=s["out"])
        return {"closing": C, **_kept(s, ctx.mesh(s["desc"], C, case["iters"]))}
    if kind == "mesh":
        return _kept(s, ctx.mesh(s["desc"], s["C"], case["iters"]))
    if kind == "update_host":
        scale = (case["radius"] + 0.5) * 0.5 * s["desc"].cell_size if case["radius"] else 0.5
        nv, nt = ctx.update_to_host(s["desc"], s["X"], s["R"], scale, s["V"], s["N"], s["T"], bilateral=case["filter"])
        return {"V": s["V"], "N": s["N"], "T": s["T"], "vertices": nv, "triangles": nt}
    if kind == "frame_field":
        s["ff"].generate()
        return _of(s["ff"], s["ff"].quats())
    if kind == "batch":
        meshes = ctx.batch_close_mesh(s["items"], lanes=case["lanes"])
        return [[it[4], *list(_kept(kept, mesh).values())[:3]]
                for it, kept, mesh in zip(s["items"], s["meshes"], meshes)]
    srv = s["server"]
    for c, scale, support in s["edits"]:
        srv.submit(c, scale, support, 0.0, L.GM_BRUSH_MAX)
    srv.drain()
    for c, scale, support in s["edits"]:
        srv.submit(c, scale, support, s["base"], L.GM_BRUSH_ZERO)
    srv.drain()
    return {"closing": _of(srv, srv.closing()), "radii": s["R"]}


def _of(owner, view):
    """A view of memory that `owner` frees when it goes: the view keeps it."""
    view.owner = owner
    return view


# ------------------------------------------------------------------ the work

def _mesh_bytes(n):
    return 24 * 7 * n * n + 12 * 14 * n * n  # about 7 n^2 vertices with normals and 14 n^2 triangles


def work(case):
    kind = case["kind"]
    if kind == "voxelize":
        if case["shape"] == "spheres":
            nt = case["count"] * 20 * 4 ** case["level"]
            mesh = 12 * (nt / 2) + 12 * nt
        else:
            mesh = 48 * 8.9 * case["samples"] ** 2  # three vertices of its own and their indices per triangle
        return {"bytes": mesh + case["res"] ** 3, "flops": 0}
    if kind == "frame_field":
        return {"bytes": 16 * case["n"] ** 3, "flops": 0}
    if kind == "box":
        cells = case["rx"] * case["ry"] * case["rz"]
        return {"bytes": cells * (2 + (8 if case["radius"] == 0 else 0)), "flops": 0}
    if kind == "batch":
        cells = case["count"] * 0.4 * (case["hi"] / 2) ** 3
        return {"bytes": 2 * cells + case["count"] * 0.5 * _mesh_bytes(case["hi"]), "flops": 0}
    if kind == "serve":
        edge = 2 * min(72, case["res"] / 4)  # fine voxels of an average dirty box
        return {"bytes": 2 * case["edits"] * edge ** 3 * (1 + 1 / 4), "flops": 0}
    res = case["res"]
    cells = res ** 3
    b = 2 * cells + (8 * cells if case.get("radius", 0) == 0 else 0)
    if kind == "mesh":
        b = cells + _mesh_bytes(2 * res)
    elif kind == "update":
        b += cells + _mesh_bytes(2 * res)
    elif kind == "update_host":
        b += _mesh_bytes(2 * res)
    elif kind == "rotcube":
        b += 16 * case["qres"] ** 3
    return {"bytes": b, "flops": 0}


# ------------------------------------------------------------------ 64-bit values

def exact(case, seed):
    if case["kind"] == "mesh":
        return _exact_mesh(_solid((case["res"],) * 3, seed), case["res"], case["iters"])
    if case["kind"] == "frame_field":
        return _exact_field(case, seed)
    return None  # bytes, or a mesh of such bytes


def _exact_field(case, seed):
    """The biharmonic system (L^T L + S) q = b by conjugate gradients to
    (nearly) the last bit."""
    n = case["n"]
    node, _, twist = _constraints(case, seed)
    half = 0.5 * np.linalg.norm(twist.astype(np.float64), axis=1, keepdims=True)
    q = np.concatenate([np.sin(half) * twist / (2 * half), np.cos(half)], 1).astype(np.float32).astype(np.float64)
    node = torch.as_tensor(node, device="cuda")
    b = torch.zeros((n ** 3, 4), dtype=torch.float64, device="cuda")
    b[node] = torch.as_tensor(q, device="cuda")
    S = torch.zeros((n ** 3, 1), dtype=torch.float64, device="cuda")
    S[node] = 1.0

    def spread(v):  # the sum over the six neighbours
        v = v.view(n, n, n, -1)
        o = torch.zeros_like(v)
        for a in range(3):
            o.narrow(a, 1, n - 1).add_(v.narrow(a, 0, n - 1))
            o.narrow(a, 0, n - 1).add_(v.narrow(a, 1, n - 1))
        return o.view(n ** 3, -1)

    w = 1.0 / spread(torch.ones((n ** 3, 1), dtype=torch.float32, device="cuda"))  # entries in 32 bits
    w = w.double()

    def apply(p):
        y = p - w * spread(p)
        return y - spread(w * y) + S * p

    x = torch.zeros_like(b)
    r, p = b.clone(), b.clone()
    rr = (r * r).sum(0)
    bb = rr.clone()
    for it in range(60 * n * n):
        Ap = apply(p)
        a = torch.where(rr > 0, rr / (p * Ap).sum(0), 0.0)
        x += a * p
        r -= a * Ap
        new = (r * r).sum(0)
        p = r + torch.where(rr > 0, new / rr, 0.0) * p
        rr = new
        if it % 64 == 0 and bool((rr <= 1e-26 * bb).all()):
            break
    return x


def _triangle_tables():
    """Edge ids per cube value, the triangles' count and the slots a value takes."""
    path = os.path.join(os.path.dirname(broxy_gb300.__file__), "csrc", "mc_tables.inc")
    text = open(path).read()
    rows = []
    for name in ("GM_MC_TRI_PACKED_INIT", "GM_MC_TRI_LEN_INIT", "GM_MC_TRI_COUNT_INIT"):
        body = text[text.index(name):].split("}")[0].split("{")[1]
        rows.append([int(v.rstrip("UL"), 0) for v in re.findall(r"0x[0-9a-fA-F]+ULL|\b\d+\b", body)])
    edges = [[(v >> (4 * k)) & 15 for k in range(15)] for v in rows[0]]
    return [torch.tensor(t, device="cuda") for t in (edges, rows[1], rows[2])]


def _morton(p):
    """30-bit Morton codes of points (x, y, z)."""
    code = torch.zeros(p.shape[0], dtype=torch.int64, device="cuda")
    for bit in range(11):
        for a in range(3):
            code |= ((p[:, a] >> bit) & 1) << (3 * bit + a)
    return code


# the edge's owner cube (offset from the cube) and its direction, by edge id
_OWNER = [(0, 0, 0, 0), (1, 0, 0, 1), (0, 1, 0, 0), (0, 0, 0, 1), (0, 0, 1, 0), (1, 0, 1, 1), (0, 1, 1, 0),
          (0, 0, 1, 1), (0, 0, 0, 2), (1, 0, 0, 2), (1, 1, 0, 2), (0, 1, 0, 2)]
_CORNER = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _exact_mesh(C, res, iters):
    """Vertices and normals of the contour marching cubes with `iters`
    bilateral iterations; the triangles are whole numbers (None)."""
    n = 2 * res
    c = C.view(res, res, res)
    occ = torch.empty((res, 2, res, 2, res, 2), dtype=torch.bool, device="cuda")
    for k in range(8):
        occ[:, k >> 2, :, (k >> 1) & 1, :, k & 1] = ((c >> k) & 1).bool()
    occ = occ.view(n, n, n)
    inner = slice(2, n - 2)  # cubes of cells 1 .. res - 2
    at = occ[inner, inner, inner]
    keys, place, high = [], [], []
    for a in range(3):
        sl = [inner] * 3
        sl[2 - a] = slice(3, n - 1)
        beyond = occ[tuple(sl)]
        p = torch.nonzero(at ^ beyond).flip(1) + 2
        keys.append(_morton(p) * 3 + a)
        place.append(p)
        high.append(beyond[p[:, 2] - 2, p[:, 1] - 2, p[:, 0] - 2])
    axis = torch.cat([torch.full_like(k, a) for a, k in enumerate(keys)])
    keys, order = torch.cat(keys).sort()
    place, high, axis = torch.cat(place)[order], torch.cat(high)[order], axis[order]
    iso, cell = float(np.float32(0.95)), float(np.float32(0.5) * np.float32(1.0 / res))
    V = place.double() * cell
    V[torch.arange(len(axis), device="cuda"), axis] += torch.where(high, iso, 1 - iso) * cell
    # mixed cubes in Morton order
    cubes, values = [], []
    for z in range(2, n - 2, 32):
        z1 = min(z + 32, n - 2)
        v = torch.zeros((z1 - z, n - 4, n - 4), dtype=torch.uint8, device="cuda")
        for k, (dx, dy, dz) in enumerate(_CORNER):
            v |= occ[z + dz:z1 + dz, 2 + dy:n - 2 + dy, 2 + dx:n - 2 + dx].to(torch.uint8) << k
        p = torch.nonzero((v != 0) & (v != 255))
        values.append(v[p[:, 0], p[:, 1], p[:, 2]].long())
        cubes.append(p.flip(1) + torch.tensor([2, 2, z], device="cuda"))
    cubes, values = torch.cat(cubes), torch.cat(values)
    order = _morton(cubes).sort()[1]
    cubes, values = cubes[order], values[order]
    edges, length, count = _triangle_tables()
    owner = torch.tensor(_OWNER, device="cuda")
    first = count[values].cumsum(0) - count[values]
    T = torch.zeros((int(count[values].sum()), 3), dtype=torch.int64, device="cuda")
    for late in (False, True):  # a triangle past its cube's slots is written over the next cube's first
        for t in range(5):
            have = (length[values] > t) & ((count[values] <= t) == late) & (first + t < T.shape[0])
            where = torch.nonzero(have)[:, 0]
            for j in range(3):
                o = owner[edges[values[where], 3 * t + j]]
                key = _morton(cubes[where] + o[:, :3]) * 3 + o[:, 3]
                i = torch.searchsorted(keys, key).clamp_(max=len(keys) - 1)
                T[first[where] + t, 2 - j] = torch.where(keys[i] == key, i, 0)
    P = [V[T[:, j]] for j in range(3)]
    area = torch.linalg.cross(P[1] - P[0], P[2] - P[0])
    N = torch.zeros_like(V)
    for j in range(3):
        N.index_add_(0, T[:, j], area)
    N /= N.norm(dim=1, keepdim=True)
    for it in range(iters):
        sigma2 = float((np.float32(1e10) if it < 2 else np.float32(0.2)) ** 2)
        M = torch.zeros_like(N)
        for a, b in ((0, 1), (1, 0), (0, 2), (2, 0), (1, 2), (2, 1)):
            nb = N[T[:, b]]
            d = ((P[a] - P[b]) ** 2).sum(1) + ((N[T[:, a]] - nb) ** 2).sum(1) / sigma2
            M.index_add_(0, T[:, a], torch.exp(-d)[:, None] * nb)
        N = M / M.norm(dim=1, keepdim=True)
    rows = torch.zeros((_ROWS * n * n - V.shape[0], 3), dtype=torch.float64, device="cuda")
    return {"V": torch.cat([V, rows]), "N": torch.cat([N, rows]), "T": None, "vertices": None, "triangles": None}
