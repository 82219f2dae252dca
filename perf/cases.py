"""Measured workloads of the mesh -> SDF bake, each through a public entry point of the binding
(italy-rs_gb300/sdfb): what a program that bakes distance fields calls, from one small prop to a
512^3 scene, from device and from host buffers, one mesh at a time, in batches and through the
server. Sizes are those of the tests, the benchmark and the tuning table.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "italy-rs_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import sdfb  # noqa: E402
from sdfb import meshgen as mg  # noqa: E402

# ---------------------------------------------------------------------------------------------
# Cases.


def listed():
    return [
        # One small prop on a coarse grid from device buffers: the call's latency is what counts.
        {"name": "prop_32", "kind": "device", "mesh": "sphere", "tris": 1280, "nx": 32, "ny": 32, "nz": 32},
        # The reference's sign-test sphere (4,096 triangles, welded) at its plain-bake size.
        {"name": "uv_sphere_64", "kind": "device", "mesh": "uv", "tris": 4096, "nx": 64, "ny": 64, "nz": 64},
        # A mesh in host memory on an odd, non-cubic grid, into page-locked outputs.
        {"name": "host_ragged", "kind": "host", "mesh": "torus", "tris": 5500, "nx": 97, "ny": 61, "nz": 43},
        # The everyday asset: 81,920 triangles at 256^3 (the benchmark's single-mesh workload).
        {"name": "asset_256", "kind": "device", "mesh": "sphere", "tris": 81920, "nx": 256, "ny": 256, "nz": 256},
        # A scanned or sculpted mesh far denser than its grid: a million triangles at 128^3.
        {"name": "dense_mesh_128", "kind": "device", "mesh": "torus", "tris": 1048576, "nx": 128, "ny": 128,
         "nz": 128},
        # The drop-in bakeSdf(MeshAsset, resolution): a soup with holes in pageable host memory
        # (weld, watertight gate, winding-number sign, padded odd grid).
        {"name": "bake_soup_100", "kind": "soup", "mesh": "open", "tris": 10000, "res": 100},
        # A large scene with holes: 500k triangles at 512^3, signed by the winding number.
        {"name": "open_scene_512", "kind": "device", "mesh": "open", "tris": 500000, "nx": 512, "ny": 512, "nz": 512},
        # The benchmark's batch: 64 meshes of 1e3..1e6 triangles, grids 32^3..256^3, one call.
        {"name": "batch_64", "kind": "batch", "count": 64, "tri_lo": 1000, "tri_hi": 1000000, "n_lo": 32, "n_hi": 256},
        # Occupancy alone (a collision or culling grid) of the everyday asset.
        {"name": "occupancy_256", "kind": "occupancy", "mesh": "sphere", "tris": 81920, "nx": 256, "ny": 256,
         "nz": 256},
        # The sparse voxelizer on a million-triangle soup at 512 (the benchmark's sparse workload).
        {"name": "sparse_512", "kind": "sparse", "mesh": "torus", "tris": 1048576, "res": 512},
        # Per-cell materials of a textured soup on its bake grid.
        {"name": "materials_96", "kind": "materials", "mesh": "sphere", "tris": 20480, "res": 96},
        # A client of the server: registers eight meshes, submits a bake of each, waits for all.
        {"name": "serve_8", "kind": "serve", "count": 8, "tri_lo": 1000, "tri_hi": 82000, "n_lo": 32, "n_hi": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A grid whose longest axis is log-uniform in [lo, hi], the others 0.4..1 of it."""
    n = [_log(rng, lo, hi)] * 3
    if rng.random() < 0.6:
        n = [max(4, int(round(a * rng.uniform(0.4, 1.0)))) for a in n]
    return {"nx": n[0], "ny": n[1], "nz": n[2]}


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "open", "soup", "batch", "occupancy", "sparse",
                       "materials", "serve"])
    closed = rng.choice(["sphere", "torus"])
    if kind == "device":
        return {"kind": "device", "mesh": closed, "tris": _log(rng, 300, 600000), **_grid(rng, 24, 256)}
    if kind == "host":
        return {"kind": "host", "mesh": closed, "tris": _log(rng, 300, 100000), **_grid(rng, 24, 128)}
    if kind == "open":
        return {"kind": "device", "mesh": "open", "tris": _log(rng, 3000, 300000), **_grid(rng, 48, 320)}
    if kind == "soup":
        return {"kind": "soup", "mesh": rng.choice(["open", closed]), "tris": _log(rng, 3000, 100000),
                "res": _log(rng, 32, 160)}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(5, 32), "tri_lo": 1000, "tri_hi": _log(rng, 5000, 300000),
                "n_lo": 32, "n_hi": rng.choice([64, 128, 160])}
    if kind == "occupancy":
        return {"kind": "occupancy", "mesh": closed, "tris": _log(rng, 1000, 500000), **_grid(rng, 32, 320)}
    if kind == "sparse":
        return {"kind": "sparse", "mesh": closed, "tris": _log(rng, 1000, 500000), "res": _log(rng, 48, 400)}
    if kind == "materials":
        return {"kind": "materials", "mesh": closed, "tris": _log(rng, 1000, 100000), "res": _log(rng, 32, 128)}
    return {"kind": "serve", "count": rng.randint(3, 16), "tri_lo": 1000, "tri_hi": _log(rng, 5000, 80000),
            "n_lo": 32, "n_hi": rng.choice([64, 96, 128])}


# ---------------------------------------------------------------------------------------------
# Meshes: (verts float32[V, 3], idx uint32[T, 3]) in [-0.5, 0.5]^3, shaped by the seed.

_icosphere = functools.lru_cache(maxsize=8)(mg.icosphere)


def _level(tris):
    return max(1, min(7, int(round(math.log(max(tris, 20) / 20.0, 4)))))


def _torus_dims(tris):
    nv = max(3, int(round(math.sqrt(tris / 6.0))))
    return max(3, int(round(tris / (2.0 * nv)))), nv


def _sphere(tris, seed, radius=0.35, center=(0.0, 0.0, 0.0)):
    v, f = _icosphere(_level(tris))
    c = np.asarray(center, np.float64)
    return mg._f32(mg.displace(c + v * radius, c, np.random.default_rng(seed), 0.05), f)


def _torus(tris, seed, R=0.28, r=0.1, center=(0.0, 0.0, 0.0)):
    nu, nv = _torus_dims(tris)
    return mg.displaced_torus(nu, nv, R, r, seed, center=center)


def _open(tris, seed):
    """Five displaced spheres and three tori at seeded places, 2% of the faces deleted."""
    rng = np.random.default_rng(seed)
    parts = []
    for _ in range(5):
        r = rng.uniform(0.14, 0.2)
        c = rng.uniform(-0.5 + r * 1.1, 0.5 - r * 1.1, size=3)
        parts.append(_sphere(tris / 6.0, int(rng.integers(1 << 30)), r, c))
    left = max(300, tris - sum(len(f) for _, f in parts))
    for _ in range(3):
        R, r = rng.uniform(0.17, 0.23), rng.uniform(0.045, 0.065)
        c = rng.uniform(-0.5 + (R + r) * 1.1, 0.5 - (R + r) * 1.1, size=3)
        parts.append(_torus(left / 3.0, int(rng.integers(1 << 30)), R, r, c))
    v, f = mg.concat(parts)
    return mg.delete_faces(v, f, 0.02, int(rng.integers(1 << 30)))


def _mesh(kind, tris, seed):
    if kind == "uv":  # the reference's sphere: its radius varies with the seed
        lat = max(4, int(round(math.sqrt(tris / 4.0))))
        return mg.uv_sphere_mesh(0.36 + 0.08 * np.random.default_rng(seed).random(), 2 * lat, lat)
    return {"sphere": _sphere, "torus": _torus, "open": _open}[kind](tris, seed)


def _batch_sizes(case):
    """(mesh kind, triangles, grid edge) of each mesh: counts spread over the logarithm of the range,
    grid edges over the powers of two from n_lo to n_hi (and n_hi)."""
    edges = [e for e in (32, 64, 128, 256) if case["n_lo"] <= e < case["n_hi"]] + [case["n_hi"]]
    out, ratio = [], math.log(case["tri_hi"] / case["tri_lo"])
    for k in range(case["count"]):
        u = (0.5 + k * 0.6180339887498949) % 1.0
        out.append(("sphere" if k % 2 else "torus", int(round(case["tri_lo"] * math.exp(ratio * u))),
                    edges[(k * 5 + k // len(edges)) % len(edges)]))
    return out


def _unit_grid(nx, ny, nz):
    """The grid of nx x ny x nz cells centred on the origin whose longest edge is 1."""
    h = 1.0 / max(nx, ny, nz)
    return sdfb.make_grid((-0.5 * nx * h, -0.5 * ny * h, -0.5 * nz * h), h, (nx, ny, nz))


def _mesh_for(case, seed):
    """The case's mesh, squeezed into its grid's box."""
    v, f = _mesh(case["mesh"], case["tris"], seed)
    n = np.array([case["nx"], case["ny"], case["nz"]], np.float64)
    return np.ascontiguousarray(v * (n / n.max()).astype(np.float32)), f


# ---------------------------------------------------------------------------------------------
# States.

@functools.lru_cache(maxsize=1)
def _context():
    return sdfb.Context(0)  # a program keeps one context


@functools.lru_cache(maxsize=1)
def _server():
    return sdfb.Server(sdfb.Context(0), hbm_budget_bytes=64 << 30)  # and one server


def _dev(a):
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


def _pinned(shape, dtype):
    return torch.empty(tuple(shape), dtype=dtype).pin_memory().numpy()


# The bounds that a soup is stored with (a MeshAsset's boundsMin / boundsMax): not a cube.
_BOUNDS = np.array([0.5, 0.41, 0.47], np.float32)


def _soup(case, seed):
    """(positions float32[3T, 3], bounds minimum, bounds maximum) of the case's mesh as a soup."""
    v, f = _mesh(case["mesh"], case["tris"], seed)
    return np.ascontiguousarray((v * (2.0 * _BOUNDS))[f.reshape(-1)]), -_BOUNDS, _BOUNDS


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("device", "occupancy"):
        v, f = _mesh_for(case, seed)
        s["grid"] = _unit_grid(case["nx"], case["ny"], case["nz"])
        s["v"], s["f"] = _dev(v), _dev(f)
        s["opts"] = sdfb.make_opts(no_distance=kind == "occupancy")
        s["dist"] = torch.empty(s["grid"].shape, dtype=torch.float32, device="cuda") if kind == "device" else None
        s["occ"] = torch.empty(s["grid"].shape, dtype=torch.uint8, device="cuda")
    elif kind == "host":
        s["v"], s["f"] = _mesh_for(case, seed)
        s["grid"] = _unit_grid(case["nx"], case["ny"], case["nz"])
        s["out"] = (_pinned(s["grid"].shape, torch.float32), _pinned(s["grid"].shape, torch.uint8))
    elif kind == "soup":
        s["p"], s["lo"], s["hi"] = _soup(case, seed)
        s["res"] = case["res"]
        g = sdfb.grid_from_bounds_res(s["lo"], s["hi"], case["res"])
        s["out"] = {np.float32: np.zeros(g.shape, np.float32), np.uint8: np.zeros(g.shape, np.uint8)}
    elif kind == "batch":
        meshes = [(_mesh(m, t, seed * 1000003 + k), n) for k, (m, t, n) in enumerate(_batch_sizes(case))]
        s["mem"] = [(_dev(v), _dev(f)) for (v, f), _ in meshes]
        s["meshes"] = [(v.data_ptr(), len(v), f.data_ptr(), len(f)) for v, f in s["mem"]]
        s["grids"] = [_unit_grid(n, n, n) for _, n in meshes]
        cells = sum(n ** 3 for _, n in meshes)  # one allocation for all the grids, as a program makes it
        s["dist"] = torch.empty(cells, dtype=torch.float32, device="cuda")
        s["occ"] = torch.empty(cells, dtype=torch.uint8, device="cuda")
        at = np.cumsum([0] + [n ** 3 for _, n in meshes])[:-1]
        s["dp"] = [s["dist"].data_ptr() + 4 * int(a) for a in at]
        s["op"] = [s["occ"].data_ptr() + int(a) for a in at]
        s["opts"] = sdfb.make_opts()
    elif kind in ("sparse", "materials"):
        s["p"], s["lo"], s["hi"] = _soup(case, seed)
        s["res"] = case["res"]
        if kind == "sparse":  # the caller's list: room for a surface several times the grid's faces
            s["cells"] = np.zeros((8 * case["res"] ** 2, 3), np.int32)
            s["count"], s["origin"], s["voxel"] = ctypes.c_uint64(), np.zeros(3, np.float32), ctypes.c_float()
        if kind == "materials":
            s["grid"] = sdfb.grid_from_bounds_res(s["lo"], s["hi"], case["res"])
            s["mat"] = mg.random_materials(len(s["p"]) // 3, seed, num_materials=6, tex_sizes=((256, 128), (64, 64)))
    else:
        s["jobs"] = []
        for k, (m, t, n) in enumerate(_batch_sizes(case)):
            v, f = _mesh(m, t, seed * 1000003 + k)
            s["jobs"].append((v, f, _unit_grid(n, n, n), _pinned((n, n, n), torch.float32),
                              _pinned((n, n, n), torch.uint8)))
        _server()
    if kind != "serve":
        _context()
    return s


def run(state):
    s, kind = state, state["kind"]
    if kind in ("device", "occupancy"):
        _context().bake_device(s["v"].data_ptr(), len(s["v"]), s["f"].data_ptr(), len(s["f"]), s["grid"], s["opts"],
                               s["dist"].data_ptr() if s["dist"] is not None else 0, s["occ"].data_ptr())
        return {"dist": s["dist"], "occ": s["occ"]} if s["dist"] is not None else {"occ": s["occ"]}
    if kind == "host":
        dist, occ = _context().bake(s["v"], s["f"], s["grid"], out=s["out"])
        return {"dist": dist, "occ": occ}
    if kind == "soup":
        _, dist, occ = _context().bake_soup(s["p"], s["lo"], s["hi"], s["res"], alloc=lambda _, dt: s["out"][dt])
        return {"dist": dist, "occ": occ}
    if kind == "batch":
        _context().bake_batch_device(s["meshes"], s["grids"], s["opts"], s["dp"], s["op"])
        return {"dist": s["dist"], "occ": s["occ"]}
    if kind == "sparse":
        ctx = _context()
        status = ctx.lib.sdfb_voxelize_sparse(
            ctx.h, s["p"].ctypes.data, len(s["p"]) // 3, s["lo"].ctypes.data, s["hi"].ctypes.data, s["res"],
            s["cells"].ctypes.data, len(s["cells"]), ctypes.byref(s["count"]), s["origin"].ctypes.data,
            ctypes.byref(s["voxel"]))
        if status != sdfb.OK:
            raise sdfb.SdfbError(status, ctx.error())
        return {"cells": s["cells"], "count": s["count"].value, "origin": s["origin"]}
    if kind == "materials":
        color, metal, rough = _context().bake_materials(s["p"], s["grid"], s["mat"])
        return {"color": color, "metal": metal, "rough": rough}
    srv = _server()
    ids = [srv.submit(srv.register(v, f), g, dist, occ) for v, f, g, dist, occ in s["jobs"]]
    for r in ids:
        srv.poll(r)
    return {"dist": [j[3] for j in s["jobs"]], "occ": [j[4] for j in s["jobs"]]}


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without: every vertex, index and texel read once, every cell written once,
# and one point-triangle distance (about 60 flops) a cell, or one triangle-box test (about 120) a
# triangle where only occupancy is asked for.


def _verts_of(mesh, tris):
    return tris // 2 + 2 if mesh != "open" else int(tris * 0.53)


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        sizes = _batch_sizes(case)
        cells = sum(n ** 3 for _, _, n in sizes)
        return {"bytes": sum(t * 12 + _verts_of(m, t) * 12 for m, t, _ in sizes) + 5 * cells, "flops": 60 * cells}
    t = case["tris"]
    if "res" in case:
        # a soup: 36 bytes a triangle; the longest axis of the padded grid has res + 5 cells
        cells = (case["res"] + 5) ** 3
        if kind == "sparse":
            return {"bytes": 36 * t + 12 * 6 * case["res"] ** 2, "flops": 120 * t}
        if kind == "materials":
            return {"bytes": (36 + 24 + 4) * t + 20 * cells, "flops": 120 * t}
        return {"bytes": 36 * t + 5 * cells, "flops": 60 * cells}
    cells = case["nx"] * case["ny"] * case["nz"]
    mesh = 12 * t + 12 * _verts_of(case["mesh"], t)
    if kind == "occupancy":
        return {"bytes": mesh + cells, "flops": 120 * t}
    return {"bytes": mesh + 5 * cells, "flops": 60 * cells}


# ---------------------------------------------------------------------------------------------
# The signed distance in 64 bits, by brute force: every cell against every triangle, the sign from
# the winding number summed over all triangles.

_MOST_PAIRS = 12e9  # about the pairs that brute force does in some seconds


def _signed_distance(v, f, grid, dev):
    h = np.float32(grid.voxel_size)
    axes = [torch.tensor((np.float32(grid.origin[a]) + (np.arange(n, dtype=np.float32) + np.float32(0.5)) * h)
                         .astype(np.float64), device=dev) for a, n in enumerate((grid.nx, grid.ny, grid.nz))]
    Z, Y, X = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    P = torch.stack([X.reshape(-1), Y.reshape(-1), Z.reshape(-1)], 0)
    tri = torch.tensor(v.astype(np.float64)[f.astype(np.int64)], device=dev)  # T, 3, 3
    T = len(tri)
    out = torch.empty(P.shape[1], dtype=torch.float64, device=dev)
    step_t = 2048
    step_p = 8192

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    def edge2(d, e):  # squared distance from the point at offset d from an edge's start
        q = (dot(d, e) / dot(e, e).clamp_min(1e-300)).clamp_(0.0, 1.0)
        r = [d[a] - q * e[a] for a in range(3)]
        return dot(r, r)

    for p0 in range(0, P.shape[1], step_p):
        p = P[:, p0:p0 + step_p, None]
        best = torch.full((p.shape[1],), math.inf, dtype=torch.float64, device=dev)
        wind = torch.zeros(p.shape[1], dtype=torch.float64, device=dev)
        for t0 in range(0, T, step_t):
            q = tri[t0:t0 + step_t].permute(1, 2, 0)[:, :, None, :]  # corner, axis, 1, T
            e = [[q[(k + 1) % 3][a] - q[k][a] for a in range(3)] for k in range(3)]
            n = [e[0][(a + 1) % 3] * e[1][(a + 2) % 3] - e[0][(a + 2) % 3] * e[1][(a + 1) % 3] for a in range(3)]
            n2 = dot(n, n)
            d = [[p[a] - q[k][a] for a in range(3)] for k in range(3)]
            best2 = torch.minimum(torch.minimum(edge2(d[0], e[0]), edge2(d[1], e[1])), edge2(d[2], e[2]))
            inside = n2 > 0
            for k in range(3):  # on the inner side of every edge's plane along the normal
                m = [n[(a + 1) % 3] * e[k][(a + 2) % 3] - n[(a + 2) % 3] * e[k][(a + 1) % 3] for a in range(3)]
                inside = inside & (dot(d[k], m) > 0)
            hgt = dot(d[0], n)
            plane2 = hgt * hgt / n2.clamp_min(1e-300)
            best2 = torch.where(inside, plane2, best2)
            best = torch.minimum(best, best2.amin(dim=1))
            len_ = [dot(x, x).sqrt() for x in d]
            # the corners seen from the point are -d: the triple product changes sign, the dots do not
            den = (len_[0] * len_[1] * len_[2] + dot(d[0], d[1]) * len_[2] + dot(d[1], d[2]) * len_[0]
                   + dot(d[2], d[0]) * len_[1])
            wind += torch.atan2(-hgt, den).sum(dim=1)
        out[p0:p0 + step_p] = torch.where((wind / (2.0 * math.pi)).abs() > 0.5, -best.sqrt(), best.sqrt())
    return out.reshape(grid.shape).cpu().numpy()


def exact(case, seed):
    """Distances in 64 bits where brute force takes seconds. Occupancy and the sparse cells are whole
    numbers; a material mean is over the triangles that a test defined in FP32 selects, so it has no
    value of its own in 64 bits."""
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    most = _MOST_PAIRS if dev == "cuda" else _MOST_PAIRS / 100
    if kind in ("device", "host"):
        if float(case["nx"]) * case["ny"] * case["nz"] * case["tris"] > most:
            return None
        v, f = _mesh_for(case, seed)
        return {"dist": _signed_distance(v, f, _unit_grid(case["nx"], case["ny"], case["nz"]), dev), "occ": None}
    if kind == "soup":
        if float(case["res"] + 5) ** 3 * case["tris"] > most:
            return None
        p, lo, hi = _soup(case, seed)
        g = sdfb.grid_from_bounds_res(lo, hi, case["res"])
        return {"dist": _signed_distance(p, np.arange(len(p)).reshape(-1, 3), g, dev), "occ": None}
    if kind == "serve":
        sizes = _batch_sizes(case)
        if not any(float(n) ** 3 * t <= most / len(sizes) for _, t, n in sizes):
            return None
        dist = []
        for k, (m, t, n) in enumerate(sizes):
            v, f = _mesh(m, t, seed * 1000003 + k)
            small = float(n) ** 3 * len(f) <= most / len(sizes)
            dist.append(_signed_distance(v, f, _unit_grid(n, n, n), dev) if small else None)
        return {"dist": dist, "occ": [None] * len(sizes)}
    return None
