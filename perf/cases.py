"""The work that users of this engine have it do, as cases that can be timed.

A case is one pass through the public entry points of libmat_gb300.rpd on a
seeded workload: the restricted power diagram of a set of weighted sites in a
tet mesh (`rpd`), that of many meshes at once (`batch`), its update after some
spheres moved (`partial`), and the distance of samples to their medial
primitives (`dist2mat`).  Meshes and site distributions are those of
libmat_gb300.workloads; the mesh of a size is the same for every seed (a user
optimises many sphere sets in one mesh), the sites are drawn from the seed.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W

PRED = {"fp64": rpd.PRED_FP64, "fp32_filter": rpd.PRED_FP32_FILTER, "exact": rpd.PRED_EXACT}

# what an engine is created with unless the case says otherwise: the
# defaults of rpd.RPD()
DEFAULTS = {"pred": "fp32_filter", "certify": False, "knn_k": 64, "clip_variant": 0,
            "topology_hash": True, "user_lists": False, "then": "cells"}


def _rpd(name, shape, tets, sites, **options):
    c = {"kind": "rpd", "shape": shape, "tets": tets, "sites": sites}
    c.update(DEFAULTS)
    c.update(options)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small part under interactive edit: the smallest call, all latency
        _rpd("cube_5k_small_part", "slotted", 5_280, 92),
        # the 'plain RPD, small' workload of the benchmark, engine defaults
        _rpd("cube_48k_defaults", "cube", 48_000, 2_000),
        # the same with the caller's own neighbour lists (libmat's site_knn
        # from its triangulation): the drop-in call
        _rpd("cube_48k_user_lists", "cube", 48_000, 2_000, user_lists=True),
        # every predicate in FP64, the reference's arithmetic: what results
        # are checked against
        _rpd("cube_48k_fp64", "cube", 48_000, 2_000, pred="fp64", topology_hash=False),
        # lattice sites with exact ties, exact predicates
        _rpd("lattice_146k_exact", "lattice", 146_334, 3_375, pred="exact"),
        # an ordinary organic model with certified lists; the FP64 vertices
        # are handed on in cell order
        _rpd("ellipsoid_200k_vertices", "ellipsoid", 200_000, 10_000, certify=True, knn_k=96,
             then="vertices"),
        # the loop of the medial-axis optimisation: diagram, topology of every
        # cell, power cells
        _rpd("ellipsoid_200k_power_cells", "ellipsoid", 200_000, 10_000, certify=True, knn_k=96,
             topology_hash=False, then="power_cells"),
        # the Houdini export's polygon soup
        _rpd("ellipsoid_120k_polygons", "ellipsoid", 120_000, 4_001, certify=True, knn_k=64,
             topology_hash=False, then="polygons"),
        # the headline workload with the settings its autotuner keeps
        _rpd("ellipsoid_1M", "ellipsoid", 1_000_000, 50_000, certify=True, knn_k=128,
             clip_variant=2, topology_hash=False),
        # an optimisation step: some spheres moved, their cells redone
        {"name": "partial_200k", "kind": "partial", "tets": 200_000, "sites": 10_000, "moved": 40,
         "knn_k": 64},
        # a dataset of uneven meshes, from few sites in many tets to many
        # sites in few
        {"name": "batch_24", "kind": "batch", "meshes": 24, "most_tets": 100_000,
         "most_sites": 10_000, "knn_k": 64},
        # the geometry-error check of a whole surface
        {"name": "dist2mat_150k", "kind": "dist2mat", "samples": 150_000, "spheres": 20_000,
         "per_sample": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rpd"] * 6 + ["partial", "batch", "dist2mat"])
    if kind == "partial":
        tets = _log(rng, 20_000, 400_000)
        sites = max(200, int(tets * math.exp(rng.uniform(math.log(0.01), math.log(0.08)))))
        return {"kind": "partial", "tets": tets, "sites": sites,
                "moved": _log(rng, 1, max(2, sites // 50)), "knn_k": rng.choice([48, 64, 96])}
    if kind == "batch":
        return {"kind": "batch", "meshes": rng.randint(3, 24),
                "most_tets": _log(rng, 20_000, 100_000), "most_sites": _log(rng, 1_000, 10_000),
                "knn_k": rng.choice([48, 64, 96])}
    if kind == "dist2mat":
        return {"kind": "dist2mat", "samples": _log(rng, 1_000, 200_000),
                "spheres": _log(rng, 100, 40_000), "per_sample": rng.randint(1, 70)}
    shape = rng.choice(["cube", "ellipsoid", "ellipsoid", "ellipsoid", "slotted", "lattice"])
    most = {"cube": 400_000, "ellipsoid": 900_000, "slotted": 60_000, "lattice": 150_000}[shape]
    tets = _log(rng, 3_000, most)
    sites = min(45_000, max(30, int(tets * math.exp(rng.uniform(math.log(0.005),
                                                                 math.log(0.2))))))
    pred = rng.choice(["fp32_filter"] * 8 + ["exact"])
    if shape == "lattice":
        pred = rng.choice(["fp32_filter", "exact"])
    elif tets <= 60_000 and rng.random() < 0.2:
        pred = "fp64"
    certify = pred == "fp32_filter" and shape != "lattice" and rng.random() < 0.6
    return _rpd(None, shape, tets, sites, pred=pred, certify=certify,
                knn_k=rng.choice([48, 64, 64, 96, 127, 128]), clip_variant=rng.choice([0, 1, 2]),
                topology_hash=rng.random() < 0.5,
                user_lists=not certify and rng.random() < 0.25,
                then=rng.choice(["cells", "cells", "vertices", "power_cells", "polygons"]))


# ---- workloads ------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _mesh(shape, tets):
    """Vertices in [0, 1000]^3, tets and their adjacency, and the frame
    (origin, scale) that maps the unit domain's sites into it."""
    if shape == "ellipsoid":
        v, t = W.ellipsoid_mesh(tets, seed=2)
    else:
        n = max(2, int(round((tets / (5.28 if shape == "slotted" else 6.0)) ** (1.0 / 3.0))))
        v, t = W.cube_grid_mesh(n)
        if shape == "slotted":  # config_slotted_cube's slot, for any n
            c = v[t].mean(axis=1)
            t = t[~((c[:, 0] > 0.4) & (c[:, 0] < 0.5) & (c[:, 1] < 0.8))]
            used, t = np.unique(t, return_inverse=True)
            v, t = v[used], t.reshape(-1, 4).astype(np.int32)
    lo = v.min(axis=0)
    scale = W.SCALE / float((v.max(axis=0) - lo).max())
    v = np.ascontiguousarray((v - lo) * scale)
    t = np.ascontiguousarray(t, np.int32)
    return v, t, rpd.mesh_adjacency(v.shape[0], t), lo, scale


def _sites(shape, n, seed, frame):
    """n weighted sites (x, y, z, r^2) of the shape's distribution."""
    rng = np.random.default_rng([seed, n])
    lo, scale = frame
    if shape == "ellipsoid":  # 70 % near the surface, 30 % inside, as config_ellipsoid
        axes = np.array([1.0, 0.6, 0.4])
        n_surf = int(round(0.7 * n))
        u = rng.normal(size=(n_surf, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        nrm = u / axes
        nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
        surf = u * axes - np.abs(rng.normal(0.0, 0.02, size=(n_surf, 1))) * nrm
        ball = rng.normal(size=(n - n_surf, 3))
        ball /= np.linalg.norm(ball, axis=1, keepdims=True)
        inside = ball * rng.uniform(size=(n - n_surf, 1)) ** (1.0 / 3.0) * axes
        xyz = rng.permutation(np.concatenate([surf, inside]))
        r = rng.lognormal(np.log(0.01), 0.5, size=n)
    elif shape == "lattice":  # config_lattice: equal radii, a few sites a hair off their place
        m = max(2, int(math.ceil(n ** (1.0 / 3.0))))
        g = (np.arange(m) + 0.5) / m
        xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
        xyz = xyz[np.sort(rng.choice(m ** 3, min(n, m ** 3), replace=False))]
        move = rng.choice(len(xyz), max(1, len(xyz) // 20), replace=False)
        xyz[move] += rng.normal(0.0, 1e-12, size=(len(move), 3))
        r = np.full(len(xyz), 0.01 * rng.uniform(0.9, 1.1))
    else:  # config_small_cube; in the slotted cube some sites lie in the slot
        xyz = rng.uniform(0.05, 0.95, size=(n, 3))
        if shape == "slotted":
            xyz[: n // 8, 0] = 0.45
        r = rng.uniform(0.01, 0.05, size=n)
    x = (xyz - lo) * scale
    return np.ascontiguousarray(np.concatenate([x, ((r * scale) ** 2)[:, None]], axis=1))


def _engine(mesh, **kw):
    v, t, adj = mesh[:3]
    r = rpd.RPD(**kw)
    r.set_mesh(v, t, adj["v_adjs"], adj["e_adj6"], adj["f_adjs"], adj["f_ids"])
    return r


@functools.lru_cache(maxsize=None)
def _batch_mesh(i, most_tets, most_sites):
    m = W.batch_mesh(i, seed=3, tet_range=(2_000, most_tets), site_range=(100, most_sites))
    return m, rpd.mesh_adjacency(m["vert3d"].shape[0], m["tets"])


def _dist2mat_inputs(case, seed):
    """Spheres along a medial sheet in the unit cube, samples anywhere, and
    for each sample a list of slabs, cones and spheres near one another."""
    g = np.random.default_rng([seed, case["samples"]])
    ns, m, k = case["spheres"], case["samples"], case["per_sample"]
    sph = np.empty((ns, 4), np.float32)
    sph[:, :3] = g.uniform(0.0, 1.0, (ns, 3))
    sph[:, 3] = g.uniform(0.01, 0.06, ns)
    smp = g.uniform(0.0, 1.0, (m, 3)).astype(np.float32)
    cnt = g.integers(max(1, k // 2), k + 1, m).astype(np.uint32)
    off = np.zeros(m, np.uint32)
    off[1:] = np.cumsum(cnt[:-1])
    n = int(cnt.sum())
    prm = g.integers(0, ns, (n, 3)).astype(np.int32)
    prm[:, 1] = (prm[:, 2] + 1 + prm[:, 1] % max(1, ns - 1)) % ns  # no sphere twice
    prm[:, 0] = (prm[:, 2] + prm[:, 1] + 1) % ns
    same = (prm[:, 0] == prm[:, 1]) | (prm[:, 0] == prm[:, 2])
    kind = g.integers(0, 4, n)  # half slabs, a quarter cones, a quarter spheres
    prm[(kind >= 2) | same, 0] = -1
    prm[kind == 3, 1] = -1
    return sph, smp, off, cnt, prm


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "dist2mat":
        s["engine"] = rpd.RPD()
        s["args"] = _dist2mat_inputs(case, seed)
        return s
    s["kept"] = _kept(case)
    if kind == "batch":
        b = rpd.Batch(certify=True, knn_k=case["knn_k"], clip_variant=2, topology_hash=False)
        for i in range(case["meshes"]):
            m, adj = _batch_mesh(i, case["most_tets"], case["most_sites"])
            sites = m["sites"].copy()
            rng = np.random.default_rng([seed, i])
            sites[:, :3] += rng.normal(0.0, 5.0, (len(sites), 3))
            b.add_mesh(m["vert3d"], m["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                       adj["f_ids"], sites)
        s["engine"] = b
    elif kind == "partial":
        mesh = _mesh("ellipsoid", case["tets"])
        n = case["sites"]
        r = _engine(mesh, knn_k=case["knn_k"], certify=True, topology_hash=False)
        before = _sites("ellipsoid", n, seed, mesh[3:])
        rng = np.random.default_rng([seed, 7])
        moved = rng.choice(n, min(n, case["moved"]), replace=False)
        after = before.copy()
        after[moved, :3] += rng.normal(0.0, 0.3 * 1000.0 / n ** (1.0 / 3.0), (len(moved), 3))
        # the sites whose cells can change: the moved ones, the neighbours
        # they had, and the sites that list one
        r.set_sites(before)
        r.compute()
        lists = r.neighbor_lists(n)
        redo = np.zeros(n, bool)
        redo[moved] = True
        redo[lists[moved][lists[moved] >= 0]] = True
        redo |= np.isin(lists, moved).any(axis=1)
        s.update(engine=r, after=after, redo=redo)
    else:
        mesh = _mesh(case["shape"], case["tets"])
        sites = _sites(case["shape"], case["sites"], seed, mesh[3:])
        r = _engine(mesh, predicate_mode=PRED[case["pred"]], certify=case["certify"],
                    knn_k=case["knn_k"], clip_variant=case["clip_variant"],
                    topology_hash=case["topology_hash"],
                    neighbor_source=rpd.NEIGH_USER if case["user_lists"] else rpd.NEIGH_KNN)
        r.set_sites(sites)
        if case["user_lists"]:
            r.set_neighbors(_lists(mesh, sites, case["knn_k"]))
        s.update(engine=r, then=case["then"])
    return s


def _lists(mesh, sites, k):
    """Neighbour lists as a caller has them: the k nearest of each site."""
    with _engine(_mesh("cube", 48), knn_k=k, exact_lists=False) as r:
        r.set_sites(sites)
        r.compute()
        return r.neighbor_lists(len(sites))


# ---- one pass -------------------------------------------------------------

class _DeviceArray:
    """n values of a numpy type in an engine's device memory, for torch."""

    def __init__(self, ptr, n, dtype):
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": np.dtype(dtype).str,
                                         "data": (int(ptr), False), "version": 3, "strides": None}


def _device(ptr, n, dtype):
    if not ptr or n <= 0:
        return torch.empty(0, dtype=getattr(torch, np.dtype(dtype).name), device="cuda")
    return torch.as_tensor(_DeviceArray(ptr, n, dtype), device="cuda")


class _Kept:
    """A caller's own array for one of the results, made once and large enough
    for any of this case's: `rows` of them, zero past the last one written."""

    def __init__(self, rows, width, dtype):
        self.array = torch.zeros((rows, width), dtype=dtype, device="cuda")
        self.used = 0

    def keep(self, values):
        n = values.shape[0]
        self.array[:n].copy_(values)
        if n < self.used:
            self.array[n:self.used].zero_()
        self.used = n
        return self.array


def _kept(case):
    """The arrays a pass of this case fills, by name: (rows, values a row,
    type), sized from the number of cells to be expected."""
    n = int(1.6 * _cells_of(case)) + 4096
    i32, i64, f32, f64 = torch.int32, torch.int64, torch.float32, torch.float64
    a = {"ids": (n, 4, i32), "volume": (n, 1, f64)}
    if case.get("then") == "vertices":
        a["vertices"] = (12 * n, 3, f64)
    if case.get("then") == "power_cells":
        a.update(site_cells=(n, 1, i32), cell_nbr_off=(n + 1, 1, i64),
                 facet_keys=(4 * n, 1, i64), facet_cells=(4 * n, 1, i32), edges=(4 * n, 7, i32),
                 vertex_cell=(5 * n, 1, i32), vertex_ids=(5 * n, 3, i32),
                 vertex_pos=(5 * n, 3, f32), surface_fid=(n, 1, i32), surface_pos=(n, 3, f32),
                 cell_cc=(n, 1, i32), facet_cc=(4 * n, 1, i32), edge_cc=(4 * n, 1, i32))
    if case.get("then") == "polygons":
        a.update(points=(12 * n, 3, f32), offsets=(10 * n + 1, 1, i64), indices=(40 * n, 1, i32),
                 site=(10 * n, 1, i32), adj_site=(10 * n, 1, i32))
    return {k: _Kept(*v) for k, v in a.items()}


def _cells(view):
    """The cells' headers as they lie on the device: (tet, site, status,
    packed counts and flags) and volumes.  (The record offsets between them
    say where a cell's record landed, which differs from pass to pass.)"""
    h = _device(view.headers, 8 * view.n_cells, np.int32).reshape(-1, 8)
    return {"ids": h[:, :4], "volume": h.view(torch.float64)[:, 3:]}


def _vertices(view):
    """The FP64 vertices of every cell, in cell order (rpd_payload_bytes: a
    record's coordinates are its last section)."""
    h = _device(view.headers, 4 * view.n_cells, np.int64).reshape(-1, 4)
    counts = h[:, 1] >> 32
    nv, np_, ne = counts & 255, (counts >> 8) & 255, (counts >> 16) & 255

    def al16(x):
        return (x + 15) & ~15

    first = (h[:, 2] + 16 * np_ + al16(8 * np_) + al16(4 * nv) + al16(4 * ne) + al16(np_)) >> 3
    stop = torch.cumsum(nv, 0)
    rows = torch.arange(int(stop[-1]) if len(stop) else 0, device="cuda")
    at = torch.repeat_interleave(first - 3 * (stop - nv), nv, output_size=len(rows)) + 3 * rows
    xyz = _device(view.payload, view.payload_bytes // 8, np.float64)
    return xyz[at[:, None] + torch.arange(3, device="cuda")]


def _power_cells(r):
    v = rpd.PowerCellsView()
    lib = rpd.load()
    if lib.rpd_get_power_cells(r._h, ctypes.byref(v)):
        raise RuntimeError("no power cells")
    n, i32, i64, f32 = v.n_cells, np.int32, np.int64, np.float32
    return {
        "site_cells": _device(v.site_cells, n, i32),
        "cell_nbr_off": _device(v.cell_nbr_off, n + 1, i64),
        "facet_keys": _device(v.facet_keys, v.n_facets, i64),
        "facet_cells": _device(v.facet_cells, v.n_facets, i32),
        "edges": _device(v.edges, 7 * v.n_edges, i32),
        "vertex_cell": _device(v.vertex_cell, v.n_vertices, i32),
        "vertex_ids": _device(v.vertex_ids, 3 * v.n_vertices, i32),
        "vertex_pos": _device(v.vertex_pos, 3 * v.n_vertices, f32),
        "surface_fid": _device(v.surface_fid, v.n_surface, i32),
        "surface_pos": _device(v.surface_pos, 3 * v.n_surface, f32),
        "cell_cc": _device(v.cell_cc, n, i32),
        "facet_cc": _device(v.facet_cc, v.n_facets, i32),
        "edge_cc": _device(v.edge_cc, v.n_edges, i32),
    }


class _PolygonView(ctypes.Structure):
    """rpd_polygon_view of include/rpd_gb300.h."""
    _fields_ = [("n_points", ctypes.c_int64), ("points", ctypes.c_void_p),
                ("n_polys", ctypes.c_int64), ("poly_offsets", ctypes.c_void_p),
                ("n_indices", ctypes.c_int64), ("indices", ctypes.c_void_p),
                ("poly_site", ctypes.c_void_p), ("poly_adj_site", ctypes.c_void_p)]


def _polygons(r):
    v = _PolygonView()
    if rpd.load().rpd_get_polygons(r._h, ctypes.byref(v)):
        raise RuntimeError("no polygons")
    return {
        "points": _device(v.points, 3 * v.n_points, np.float32),
        "offsets": _device(v.poly_offsets, v.n_polys + 1, np.int64),
        "indices": _device(v.indices, v.n_indices, np.int32),
        "site": _device(v.poly_site, v.n_polys, np.int32),
        "adj_site": _device(v.poly_adj_site, v.n_polys, np.int32),
    }


def run(state):
    r, kind = state["engine"], state["kind"]
    if kind == "dist2mat":
        dist, closest = r.dist2mat(*state["args"])
        return {"dist": dist, "closest": closest}
    if kind == "batch":
        r.compute()
        v = rpd.CellsView()
        lib = rpd.load()
        if lib.rpd_get_cells(lib.rpd_batch_context(r._h), ctypes.byref(v)):
            raise RuntimeError("no cells")
        out = _cells(v)
    elif kind == "partial":
        r.set_sites(state["after"])
        r.compute_partial(state["redo"])
        out = _cells(r.view())
    else:
        r.compute()
        out = _cells(r.view())
        if state["then"] == "vertices":
            out["vertices"] = _vertices(r.view())
        elif state["then"] == "power_cells":
            r.compute_topology()
            r.compute_power_cells()
            out.update(_power_cells(r))
        elif state["then"] == "polygons":
            r.compute_polygons()
            out.update(_polygons(r))
    return {k: a.keep(out[k].reshape(-1, a.array.shape[1])) for k, a in state["kept"].items()}


# ---- the least a pass has to do -------------------------------------------

def _cells_of(case):
    """Cells to be expected.  A tet gives one cell and one more for each face
    between two sites that crosses it: the faces of s cells have an area of
    2.9 s^(1/3) in a unit volume, and t tets of mean width 1.86 t^(-1/3) meet
    1.86 t^(2/3) times the area."""
    return sum(t + 5.4 * t ** (2.0 / 3.0) * s ** (1.0 / 3.0) for t, s in _sizes(case))


def _sizes(case):
    if case["kind"] != "batch":
        return [(case["tets"], case["sites"])]
    return [(len(m["tets"]), len(m["sites"])) for m, _ in
            (_batch_mesh(i, case["most_tets"], case["most_sites"]) for i in range(case["meshes"]))]


def work(case):
    """Inputs read once and cells written once.  A cell's record holds about
    480 bytes (its planes, plane ids, dual triangles, edges and FP64 vertices,
    as the 1M-tet workload's 3.35M cells in 1.66 GB)."""
    if case["kind"] == "dist2mat":
        n = 0.75 * case["samples"] * case["per_sample"]
        # a slab's closed form and its three cones take about 400 operations,
        # a cone 60, a sphere 10
        return {"bytes": 28.0 * case["samples"] + 16.0 * case["spheres"] + 12.0 * n,
                "flops": n * (0.5 * 400 + 0.25 * 60 + 0.25 * 10)}
    cells = _cells_of(case)
    tets, sites = (sum(x[i] for x in _sizes(case)) for i in (0, 1))
    read = 60.0 * tets + 48.0 * sites  # the tets with their adjacency, the sites
    if case["kind"] == "partial":
        # the kept cells are in place; those of the moved sites and of their
        # power neighbours (about 15 each) are made again
        cells *= min(1.0, 16.0 * case["moved"] / case["sites"])
        return {"bytes": 48.0 * sites + cells * 480.0, "flops": cells * 1500.0}
    write = 512.0 * cells
    then = case.get("then", "cells")
    if then == "vertices":
        write += 2 * 24.0 * 7 * cells
    elif then == "power_cells":
        write += 480.0 * cells + 160.0 * cells
    elif then == "polygons":
        write += 480.0 * cells + 230.0 * cells
    # a cell: its planes (12 operations each), the signs of its vertices'
    # tests, about seven vertices solved
    return {"bytes": read + write, "flops": cells * 1500.0}


# ---- 64-bit values --------------------------------------------------------

def _cone64(p, a, b):
    """|p - c(t)| - r(t) at the stationary point of the cone from the larger
    sphere (t = 0) to the smaller (t = 1); where one sphere holds the other
    the point is the smaller sphere, as libmat's formula has it."""
    swap = (a[:, 3] > b[:, 3])[:, None]
    m1, m2 = torch.where(swap, b, a), torch.where(swap, a, b)
    c21, cq2 = m1[:, :3] - m2[:, :3], m2[:, :3] - p
    A, D, F = (c21 * c21).sum(1), 2 * (c21 * cq2).sum(1), (cq2 * cq2).sum(1)
    R1 = m1[:, 3] - m2[:, 3]
    arg = (D * D - 4 * A * F) * (R1 * R1 - A) * R1 * R1
    t = (-(A * D - R1 * R1 * D) - torch.sqrt(arg)) / (2 * (A * A - A * R1 * R1))
    t = torch.where(t.isnan(), torch.ones_like(t), t.clamp(0, 1))
    return _sphere64(p, m2 + t[:, None] * (m1 - m2))


def _sphere64(p, s):
    return (p - s[:, :3]).norm(dim=1) - s[:, 3]


def _slab64(p, m1, m2, m3):
    """The interior stationary point of |p - c| - r over a slab whose radii
    differ, else the nearest of its three cones."""
    c31, c32, cm3 = m1[:, :3] - m3[:, :3], m2[:, :3] - m3[:, :3], m3[:, :3] - p
    R1, R2 = m1[:, 3] - m3[:, 3], m2[:, 3] - m3[:, 3]
    A, B, C = (c31 * c31).sum(1), 2 * (c31 * c32).sum(1), (c32 * c32).sum(1)
    D, E, F = 2 * (c31 * cm3).sum(1), 2 * (c32 * cm3).sum(1), (cm3 * cm3).sum(1)
    L1, L2, L3 = 2 * A * R2 - B * R1, 2 * C * R1 - B * R2, E * R1 - D * R2
    H, K = L2 / L1, L3 / L1
    q = A * H * H + B * H + C
    W1 = (2 * C + B * H) ** 2 - 4 * R2 * R2 * q
    W2 = 2 * (2 * C + B * H) * (B * K + E) - 4 * R2 * R2 * (2 * A * H * K + B * K + D * H + E)
    W3 = (B * K + E) ** 2 - 4 * R2 * R2 * (A * K * K + D * K + F)
    disc = W2 * W2 - 4 * W1 * W3
    root = torch.sqrt(disc.clamp(min=0))
    best = None
    for sign in (-1.0, 1.0):
        t2 = torch.where(disc >= 0, (-W2 + sign * root) / (2 * W1), -torch.ones_like(W1))
        t1 = H * t2 + K
        w = torch.stack([t1, t2, 1 - t1 - t2], 1)
        d = _sphere64(p, w[:, :1] * m1 + w[:, 1:2] * m2 + w[:, 2:] * m3)
        if best is None:
            best, b1, b2 = d, t1, t2
        else:
            better = d < best
            best, b1, b2 = (torch.where(better, x, y) for x, y in ((d, best), (t1, b1), (t2, b2)))
    inside = (b1 + b2 < 1) & (b1 >= 0) & (b1 <= 1) & (b2 >= 0) & (b2 <= 1)
    edge = torch.minimum(torch.minimum(_cone64(p, m1, m3), _cone64(p, m2, m3)), _cone64(p, m1, m2))
    return torch.where(inside, best, edge)


def exact(case, seed):
    """Distances in 64 bits.  The diagram's cells have no such value that is
    quick to make: each is the intersection of a tet with all bisectors of its
    site, in the topology the predicates decide."""
    if case["kind"] != "dist2mat":
        return None
    sph, smp, _, cnt, prm = (torch.from_numpy(a.astype(np.float64 if a.dtype == np.float32
                                                       else np.int64)).cuda()
                             for a in _dist2mat_inputs(case, seed))
    row = torch.repeat_interleave(torch.arange(len(smp), device="cuda"), cnt)
    p = smp[row]
    d = torch.empty(len(row), dtype=torch.float64, device="cuda")
    slab, ball = prm[:, 0] >= 0, prm[:, 1] < 0
    cone = ~slab & ~ball
    d[ball] = _sphere64(p[ball], sph[prm[ball, 2]])
    d[cone] = _cone64(p[cone], sph[prm[cone, 1]], sph[prm[cone, 2]])
    d[slab] = _slab64(p[slab], *(sph[prm[slab, i]] for i in range(3)))
    out = torch.full((len(smp),), math.inf, dtype=torch.float64, device="cuda")
    return {"dist": out.scatter_reduce(0, row, d, "amin"), "closest": None}
