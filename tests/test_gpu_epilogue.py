"""The epilogue (rpd_epilogue.cu) over its layouts -- one cell a warp, sixteen,
cells so large that a warp's share does not fit its store, no geometry --
against FP64: every vertex solved in numpy from planes made of the FP64 mesh
and sites, per-tet sums of the volumes, and the canonical hashes of
tests/helpers.py's mixing."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from tests.helpers import SUCCESS, mix64, tet_volumes

pytestmark = pytest.mark.gpu

NO_INTERSECTION = 6
FACES = np.array([[2, 1, 3], [0, 2, 3], [1, 0, 3], [0, 1, 2]])


def compute(cfg, adj, k, **kw):
    with rpd.RPD(knn_k=k, **kw) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        r.compute()
        return r.pair_headers(), r.cells()[1], r.topology_hashes()


def sections(h, p):
    """(ids, dual triangles, FP64 vertices) of one record."""
    al = lambda x: (x + 15) & ~15  # noqa: E731
    nv, np_, ne = int(h["nb_v"]), int(h["nb_p"]), int(h["nb_e"])
    o = int(h["offset"]) + 16 * np_
    ids = p[o:o + 8 * np_].view(np.int32).reshape(-1, 2)
    o += al(8 * np_)
    ver = p[o:o + 4 * nv].reshape(-1, 4)
    o += al(4 * nv) + al(4 * ne) + al(np_)
    return ids, ver, p[o:o + 24 * nv].view(np.float64).reshape(-1, 3)


def planes64(cfg, tet, sid, ids):
    """The cell's planes n.x + d about the seed, in FP64."""
    S = cfg["sites"][sid]
    v = cfg["vert3d"][cfg["tets"][tet]] - S[:3]
    a, b, c = (v[FACES[:, i]] for i in range(3))
    n = np.cross(b - a, c - a)
    out = [np.concatenate([n, -(a * n).sum(1, keepdims=True)], 1)]
    B = cfg["sites"][np.where(ids[4:, 0] == sid, ids[4:, 1], ids[4:, 0])]
    n = S[:3] - B[:, :3]
    d = ((n * n).sum(1) + S[3] - B[:, 3]) / 2
    out.append(np.concatenate([n, d[:, None]], 1))
    return np.concatenate(out)


@pytest.mark.parametrize("n,sites,k", [(2, 5, 4), (10, 400, 30), (3, 600, 100)])
def test_vertices_volumes_and_hashes(n, sites, k):
    cfg = W.config_small_cube(n=n, n_site=sites, seed=9)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    h, p, hashes = compute(cfg, adj, k)
    ok = np.flatnonzero(h["status"] == SUCCESS)
    if sites > 500:  # sixteen of these do not fit a warp's store
        assert h["nb_p"][ok].astype(int).max() > 16 and h["nb_v"][ok].astype(int).max() > 16
    for q in np.random.default_rng(1).permutation(ok)[:400]:
        ids, ver, xyz = sections(h[q], p)
        pl = planes64(cfg, h["tet_id"][q], h["site_id"][q], ids)
        tri = pl[ver[:, :3].astype(int)]
        N = tri[:, :, :3]
        det = np.linalg.det(N)
        well = np.abs(det) > 1e-4 * np.prod(np.linalg.norm(N, axis=2), axis=1)
        x = np.linalg.solve(N[well], -tri[well][:, :, 3:])[..., 0] + cfg["sites"][h["site_id"][q], :3]
        # double-float Cramer: about 2^-44 of the 1000-unit frame over det's 1e-4
        assert np.abs(xyz[well] - x).max(initial=0.0) < 1e-6
        key = (ids[:, 0].astype(np.uint32).astype(object) << 32) | ids[:, 1].astype(np.uint32).astype(object)
        want = 0
        for t in ver:
            z = 0
            for f in sorted(int(key[i]) for i in t[:3]):
                z = mix64(z ^ f)
            want += mix64(z ^ int(t[3]))
        assert int(hashes[q]) == want & ((1 << 64) - 1)
    # (the reference's capacities drop a cell of too many edges: its tet is
    # then not covered)
    whole = np.ones(len(cfg["tets"]), bool)
    whole[h["tet_id"][(h["status"] != SUCCESS) & (h["status"] != NO_INTERSECTION)]] = False
    assert whole.mean() > 0.5
    vol = np.bincount(h["tet_id"][ok], weights=h["volume"][ok], minlength=len(cfg["tets"]))
    tv = tet_volumes(cfg["vert3d"], cfg["tets"])
    assert np.all(np.abs(vol - tv)[whole] <= 1e-4 * tv[whole])


def test_without_geometry():
    cfg = W.config_small_cube(n=10, n_site=400, seed=9)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    h, p, hashes = compute(cfg, adj, 30, compute_geometry=False)
    h1, _, hashes1 = compute(cfg, adj, 30)
    assert np.array_equal(hashes, hashes1) and np.all(h["volume"] == 0.0)
    for q in np.flatnonzero(h["status"] == SUCCESS)[:100]:
        assert np.all(sections(h[q], p)[2] == 0.0)
