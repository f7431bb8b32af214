"""The scans and compactions (rpd_scan.cuh) at the edges of their tiles and
launch shapes, through the calls that use them: cells compacted from pair
headers (kept in pair order), and record offsets of the topology and polygon
passes scanned over the cells."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from tests.helpers import SUCCESS

pytestmark = pytest.mark.gpu


# pairs (and cells) below one tile of 1,024, one scan block of 16,384, and
# many tiles, whose compaction tile has grown past its least
@pytest.mark.parametrize("n,sites", [(1, 1), (2, 5), (5, 40), (12, 30), (20, 2_000), (60, 4_000)])
def test_compaction_and_offsets(n, sites):
    cfg = W.config_small_cube(n=n, n_site=sites, seed=3)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    with rpd.RPD(knn_k=24, topology_hash=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        st = r.compute()
        ph = r.pair_headers()
        h, _ = r.cells()
        r.compute_topology()
        th, _ = r.topology()
        r.compute_polygons()
        poly = r.polygons()
    ok = ph["status"] == SUCCESS
    assert len(ph) == st.n_pairs and np.array_equal(h, ph[ok])
    counts = st.as_dict()["status_counts"]
    assert [counts[s] for s in rpd.STATUS_NAMES[:9]] == \
        [int((ph["status"] == i).sum()) for i in range(9)]
    assert np.array_equal(np.lexsort((h["site_id"], h["tet_id"])), np.arange(len(h)))
    # topology records (12 B a plane's 4 + 1 + 1, an edge's 1, a vertex's 3,
    # to 16) lie one after the other
    size = 6 * h["nb_p"].astype(np.int64) + h["nb_e"] + 3 * h["nb_v"].astype(np.int64)
    size = (size + 15) // 16 * 16
    assert np.array_equal(th["offset"].astype(np.int64), np.cumsum(size) - size)
    assert np.all(np.diff(poly["poly_offsets"]) >= 3)
    assert poly["poly_offsets"][0] == 0 and poly["poly_offsets"][-1] == len(poly["indices"])


@pytest.mark.parametrize("n,sites", [(2, 3), (7, 90), (20, 700), (30, 4_000)])
def test_power_cell_records_are_sorted(n, sites):
    """The radix sort's tiles: one, a few, many; site ids of one and two digits."""
    cfg = W.config_small_cube(n=n, n_site=sites, seed=6)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    with rpd.RPD(knn_k=24, topology_hash=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        r.compute()
        h, _ = r.cells()
        r.compute_topology()
        r.compute_power_cells()
        d = r.power_cells()
    # cells by site, in cell order within one
    want = np.argsort(h["site_id"], kind="stable")
    assert np.array_equal(d["site_cells"].astype(np.int64), want)
    # facets by (site, neighbour), then cell; each names its cell's site
    key, cell = d["facet_keys"], d["facet_cells"].astype(np.int64)
    assert np.array_equal(np.lexsort((cell, key)), np.arange(len(key)))
    assert np.array_equal(key >> np.uint64(32), h["site_id"][cell].astype(np.uint64))
    # edges (site, neighbour pair, cell, ...) by site, pair and cell
    e = d["edges"].astype(np.int64)
    assert np.array_equal(np.lexsort((e[:, 3], e[:, 2], e[:, 1], e[:, 0])), np.arange(len(e)))
    assert np.array_equal(h["site_id"][e[:, 3]], e[:, 0])
