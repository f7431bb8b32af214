"""The incremental update's merge (rpd_partial.cu): recomputing some sites of an
unchanged diagram gives the same cells, record for record, one behind the
other."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# from a handful of records (one a warp) to hundreds of thousands (many a warp,
# ragged last ones); all kept, some or all replaced
@pytest.mark.parametrize("n,n_site", [(1, 9), (2, 20), (6, 40), (14, 300), (24, 700)])
@pytest.mark.parametrize("share", [0.0, 0.1, 1.0])
def test_merge_of_unchanged_sites_keeps_every_record(n, n_site, share):
    cfg = W.config_small_cube(n=n, n_site=n_site, seed=n)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    rng = np.random.default_rng(n)
    flags = rng.random(n_site) < share
    with rpd.RPD(knn_k=8 if n_site < 65 else 64, certify=True, topology_hash=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        r.compute()
        h0, p0 = r.cells()
        r.compute_partial(flags)
        h1, p1 = r.cells()
    assert len(h0) == len(h1)
    for f in ("tet_id", "site_id", "status", "nb_v", "nb_p", "nb_e", "volume"):
        assert np.array_equal(h0[f], h1[f]), f
    assert int(h1["offset"][0]) == 0
    for q in rng.choice(len(h0), min(len(h0), 5000), replace=False):
        size = rpd.payload_bytes(h0["nb_v"][q], h0["nb_p"][q], h0["nb_e"][q])
        a, b = int(h0["offset"][q]), int(h1["offset"][q])
        assert np.array_equal(p0[a:a + size], p1[b:b + size])
        if q + 1 < len(h1):
            assert int(h1["offset"][q + 1]) == b + size
