"""Candidate pairs on meshes with two classes of tets, whose larger class takes
its search regions from the smaller's (site_box_kernel): graded meshes with a
few tets many times larger than the rest, single tets, sites hidden in heavy
ones (empty regions), outside the mesh and on top of one another, GPU and
user lists, single meshes and batches -- against the reference's rule over all
tets and sites."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def graded(n, power, n_site, seed, heavy=0, outside=0, spikes=0):
    vert, tets = W.cube_grid_mesh(n)
    vert = 1000.0 * vert ** power
    # spikes: tets from faces of the x = 0 side to far apexes, many times the
    # radius of the others
    faces = np.concatenate([np.delete(tets, i, 1) for i in range(4)])
    faces = faces[(vert[faces][:, :, 0] == 0.0).all(1)]
    apex = np.array([[-3000.0, 300.0 + 200.0 * i, 500.0] for i in range(spikes)]).reshape(-1, 3)
    ids = len(vert) + np.arange(spikes)
    tets = np.concatenate([tets, np.concatenate([faces[:spikes], ids[:, None]], 1)])
    vert = np.concatenate([vert, apex])
    tets, _ = W._orient_positive(vert, tets)
    rng = np.random.default_rng(seed)
    xyz = 1000.0 * rng.uniform(0.0, 1.0, (n_site, 3)) ** power
    r = rng.uniform(5.0, 40.0, n_site)
    r[:heavy] = rng.uniform(200.0, 500.0, heavy)  # hide their neighbours
    xyz[n_site - outside:] += rng.uniform(200.0, 900.0, (outside, 3))
    xyz[heavy] = xyz[heavy + 1]
    return dict(vert3d=vert, tets=tets.astype(np.int32), flags=np.ones(n_site, np.uint32),
                sites=np.concatenate([xyz, (r * r)[:, None]], 1))


CASES = [(1, 1.0, 3, {}), (9, 3.0, 40, {"spikes": 1}), (9, 3.0, 300, {"heavy": 6, "spikes": 3}),
         (12, 4.0, 500, {"heavy": 3, "outside": 30, "spikes": 4}),
         (10, 1.0, 200, {"heavy": 20, "spikes": 2})]


def compare(cfg, nbr, offs, ps):
    ro, rp = O.candidate_pairs(cfg["vert3d"].astype(np.float32), cfg["tets"],
                               cfg["sites"].astype(np.float32), cfg["flags"], nbr)
    assert np.array_equal(offs, ro) and np.array_equal(ps, rp)


@pytest.mark.parametrize("user", [False, True])
@pytest.mark.parametrize("n,power,sites,kw", CASES)
def test_pairs_match_the_rule(n, power, sites, kw, user):
    cfg = graded(n, power, sites, 7, **kw)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    nbr = None
    for source in [rpd.NEIGH_KNN] + ([rpd.NEIGH_USER] if user else []):
        with rpd.RPD(neighbor_source=source, knn_k=20, exact_lists=False) as r:
            r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                       adj["f_ids"])
            r.set_sites(cfg["sites"], cfg["flags"])
            if source == rpd.NEIGH_USER:
                r.set_neighbors(nbr)
            r.compute()
            info = r.mesh_info()
            nbr = r.neighbor_lists(sites) if nbr is None else nbr
            offs, ps = r.pairs(len(cfg["tets"]))
        if "spikes" in kw:
            assert info["class_count"][1] > 0
            assert info["class_radius"][1] > 3.0 * info["class_radius"][0]
        compare(cfg, nbr, offs, ps)


def test_batch_cells_match_single_meshes():
    cfgs = [graded(n, power, sites, 3 + i, **kw) for i, (n, power, sites, kw) in enumerate(CASES)]
    adjs = [rpd.mesh_adjacency(c["vert3d"].shape[0], c["tets"]) for c in cfgs]
    kw = dict(knn_k=20, exact_lists=False)
    with rpd.Batch(**kw) as b:
        for c, a in zip(cfgs, adjs):
            b.add_mesh(c["vert3d"], c["tets"], a["v_adjs"], a["e_adj6"], a["f_adjs"], a["f_ids"],
                       c["sites"], c["flags"])
        b.compute()
        got = [b.mesh_cells(i)[0] for i in range(len(cfgs))]
    for c, a, h in zip(cfgs, adjs, got):
        with rpd.RPD(**kw) as r:
            r.set_mesh(c["vert3d"], c["tets"], a["v_adjs"], a["e_adj6"], a["f_adjs"], a["f_ids"])
            r.set_sites(c["sites"], c["flags"])
            r.compute()
            want, _ = r.cells()
        for f in ("tet_id", "site_id", "status", "nb_v", "nb_p", "nb_e"):
            assert np.array_equal(h[f], want[f])
