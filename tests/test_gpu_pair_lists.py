"""The candidate pairs' lists by tet (pairs_to_csr): lists of a few sites to
more than a warp's stage holds, warps whose tets do not fit it together, ragged
last warps -- against the reference's rule, and the cells' tets against the
lists."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_site,longest", [(1, 25, 1), (1, 400, 40), (1, 9000, 1025),
                                              (2, 4000, 60), (3, 2000, 10), (7, 500, 2)])
def test_lists_are_the_rules_in_site_order(n, n_site, longest):
    cfg = W.config_small_cube(n=n, n_site=n_site, seed=n + n_site)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    with rpd.RPD(knn_k=20, exact_lists=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        st = r.compute()
        nbr = r.neighbor_lists(n_site)
        offs, ps = r.pairs(len(cfg["tets"]))
        h, _ = r.cells()
    ro, rp = O.candidate_pairs(cfg["vert3d"].astype(np.float32), cfg["tets"],
                               cfg["sites"].astype(np.float32), cfg["flags"], nbr)
    assert np.array_equal(offs, ro) and np.array_equal(ps, rp)
    assert np.diff(offs).max() == st.tet_k >= longest
    # the emitted cells: a subsequence of the pairs, in their order
    pairs = np.repeat(np.arange(len(cfg["tets"])), np.diff(offs)).astype(np.int64) << 32 | ps
    cells = h["tet_id"].astype(np.int64) << 32 | h["site_id"]
    assert np.all(np.diff(cells) > 0) and np.isin(cells, pairs).all()
