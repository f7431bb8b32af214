"""The thread-per-cell clipper (rpd_clip_thread.cu) against the FP64 path,
which a warp per cell clips (and which the parity tests pin to the oracle):
the same records byte for byte in site-id order, the same cells by canonical
topology with certified lists, over list lengths that are and are not
multiples of a group of four, few and many pairs per tet (cells that outgrow a
lane go back to the warps), fewer pairs than lanes, ties, duplicated and
unflagged sites, and lists with holes."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from tests.helpers import SUCCESS

pytestmark = pytest.mark.gpu

MIN_PAIRS = 20000  # kThreadsPairs of rpd_clip_thread.cu


def run(cfg, adj, pred, nbr=None, **kw):
    with rpd.RPD(predicate_mode=pred, neighbor_source=rpd.NEIGH_KNN if nbr is None
                 else rpd.NEIGH_USER, **kw) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        if nbr is not None:
            r.set_neighbors(nbr)
        st = r.compute()
        return st, r.pair_headers(), r.cells(), r.topology_hashes()


def records(h, p):
    """The topology and plane bytes of every emitted cell, in pair order, and
    the statuses and counts."""
    ok = h["status"] == SUCCESS
    nv, np_, ne = (h[f][ok].astype(np.int64) for f in ("nb_v", "nb_p", "nb_e"))
    al = lambda x: (x + 15) // 16  # noqa: E731
    chunks = np_ + al(8 * np_) + al(4 * nv) + al(4 * ne) + al(np_)
    start = h["offset"][ok].astype(np.int64) // 16 - (np.cumsum(chunks) - chunks)
    at = np.repeat(start, chunks) + np.arange(chunks.sum())
    counts = np.stack([h[f] for f in ("tet_id", "site_id", "status", "nb_v", "nb_p", "nb_e")], 1)
    return counts, p[:p.size // 16 * 16].reshape(-1, 16)[at]


def same_records(ha, pa, hb, pb):
    return all(np.array_equal(x, y) for x, y in zip(records(ha, pa), records(hb, pb)))


def case(kind):
    if kind == "lattice":
        return W.config_lattice(n=16, m=8)
    if kind == "ellipsoid":
        return W.config_ellipsoid(target_tets=40_000, n_site=2_000, seed=11)
    n, sites = {"cube": (20, 2_000), "few_pairs": (10, 400), "dense": (9, 3_000)}[kind]
    return W.config_small_cube(n=n, n_site=sites, seed=5)


@pytest.mark.parametrize("kind,k", [("cube", 64), ("cube", 63), ("cube", 5), ("few_pairs", 1),
                                    ("few_pairs", 30), ("dense", 48), ("dense", 127),
                                    ("lattice", 64), ("ellipsoid", 96)])
def test_equals_fp64_path(kind, k):
    cfg = case(kind)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    a, ha, (_, pa), _ = run(cfg, adj, rpd.PRED_FP64, knn_k=k, exact_lists=False)
    b, hb, (_, pb), _ = run(cfg, adj, rpd.PRED_FP32_FILTER, knn_k=k, exact_lists=False)
    assert b.n_pairs == a.n_pairs >= MIN_PAIRS
    assert np.array_equal(ha["flags"], hb["flags"])
    assert np.array_equal(ha["volume"], hb["volume"], equal_nan=True)
    assert same_records(ha, pa, hb, pb)


@pytest.mark.parametrize("kind,k", [("cube", 64), ("dense", 33), ("ellipsoid", 128)])
def test_certified_cells_equal_fp64_path(kind, k):
    cfg = case(kind)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    a, ha, _, ta = run(cfg, adj, rpd.PRED_FP64, knn_k=k, certify=True)
    b, hb, _, tb = run(cfg, adj, rpd.PRED_FP32_FILTER, knn_k=k, certify=True)
    assert b.n_pairs == a.n_pairs >= MIN_PAIRS
    assert a.n_uncertified == b.n_uncertified == 0
    assert np.array_equal(ha["status"], hb["status"])
    assert np.array_equal(ta, tb)


def test_user_lists_with_holes_duplicates_and_unflagged_sites():
    cfg = case("cube")
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    rng = np.random.default_rng(3)
    cfg["sites"][100:140] = cfg["sites"][200:240]  # the same sphere twice
    cfg["flags"][rng.choice(2_000, 300, replace=False)] = 0
    with rpd.RPD(knn_k=50, exact_lists=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        r.compute()
        nbr = r.neighbor_lists(2_000)
    nbr[rng.integers(0, 2_000, 400), rng.integers(0, 50, 400)] = -1  # a list ends at its hole
    a, ha, (_, pa), _ = run(cfg, adj, rpd.PRED_FP64, nbr=nbr)
    b, hb, (_, pb), _ = run(cfg, adj, rpd.PRED_FP32_FILTER, nbr=nbr)
    assert b.n_pairs == a.n_pairs >= MIN_PAIRS
    assert same_records(ha, pa, hb, pb)


@pytest.mark.parametrize("n,m", [(14, 7), (16, 8)])
def test_exact_signs_equal_the_oracle(n, m):
    """Lattices whose coordinates are (m = 8) and are not (m = 7) short binary
    fractions: determinants that vanish exactly, and ones that only nearly do."""
    from oracle import oracle as O

    cfg = W.config_lattice(n=n, m=m)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    with rpd.RPD(predicate_mode=rpd.PRED_EXACT, knn_k=40, exact_lists=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        st = r.compute()
        nbr = r.neighbor_lists(len(cfg["sites"]))
        offs, ps = r.pairs(len(cfg["tets"]))
        ph, p = r.pair_headers(), r.cells()[1]
    assert st.n_pairs >= MIN_PAIRS and st.n_fp64_uncertain > 0
    mesh = dict(vert3d=cfg["vert3d"], tets=cfg["tets"],
                **{k: adj[k] for k in ("v_adjs", "e_adj6", "f_adjs", "f_ids")})
    oh, op, _ = O.clip_cells(mesh, cfg["sites"], nbr, offs, ps, pred_mode=2)
    assert same_records(ph, p, oh, op)


@pytest.mark.parametrize("certify", [False, True])
def test_extended_rows_equal_fp64_path(certify):
    """Short base lists: the exact-lists rounds clip enough cells again for the
    lanes, with rows of up to 512 entries at odd places."""
    cfg = W.config_small_cube(n=20, n_site=2_000, seed=5)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    a, ha, (_, pa), ta = run(cfg, adj, rpd.PRED_FP64, knn_k=14, certify=certify)
    b, hb, (_, pb), tb = run(cfg, adj, rpd.PRED_FP32_FILTER, knn_k=14, certify=certify)
    assert b.n_cert_reclipped >= MIN_PAIRS and a.n_uncertified == b.n_uncertified == 0
    assert np.array_equal(ha["status"], hb["status"]) and np.array_equal(ta, tb)
    if not certify:
        assert same_records(ha, pa, hb, pb)
