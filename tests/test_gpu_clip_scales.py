"""The clippers on scenes scaled by powers of two.  The planes' minors then fall
through the range of the single precision's subnormals, where an error is not
in proportion to the terms any more; every sign has to stay the sign of the
reference's FP64 determinant (which no such scale touches), with a lane and
with a warp per cell.  Scaling changes no plane's float mantissa as long as
nothing underflows, so the FP64 path, the oracle and the unscaled scene are all
references."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from oracle import oracle as O
from tests.helpers import SUCCESS
from tests.test_gpu_clip_threads import MIN_PAIRS, run, same_records

pytestmark = pytest.mark.gpu


def scaled(cfg, k):
    """The scene in a frame of 1000 x 2^-k units."""
    s = np.ldexp(1.0, -k)
    return dict(cfg, vert3d=cfg["vert3d"] * s, sites=cfg["sites"] * np.array([s, s, s, s * s]))


SIZES = {"lanes": (20, 2_000), "warps": (8, 250)}  # pairs above and below MIN_PAIRS


def scene(size):
    n, sites = SIZES[size]
    cfg = W.config_small_cube(n=n, n_site=sites, seed=5)
    return cfg, rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])


@pytest.mark.parametrize("size", ["lanes", "warps"])
@pytest.mark.parametrize("k", [10, 20, 24, 25, 26, 27, 29, 30])
def test_filtered_signs_equal_fp64_path(size, k):
    cfg, adj = scene(size)
    cfg = scaled(cfg, k)
    a, ha, (_, pa), _ = run(cfg, adj, rpd.PRED_FP64, knn_k=64, exact_lists=False)
    b, hb, (_, pb), _ = run(cfg, adj, rpd.PRED_FP32_FILTER, knn_k=64, exact_lists=False)
    assert (b.n_pairs >= MIN_PAIRS) == (size == "lanes") and b.n_pairs == a.n_pairs
    assert (ha["status"] == SUCCESS).mean() > 0.5
    assert same_records(ha, pa, hb, pb)


@pytest.mark.parametrize("n,m", [(14, 7), (8, 4)])  # pairs above and below MIN_PAIRS
@pytest.mark.parametrize("k", [10, 24, 25, 26, 27, 28, 29])
def test_exact_signs_equal_the_oracle(n, m, k):
    """Ties of lattice sites, which FP64 leaves undecided at every scale."""
    cfg = W.config_lattice(n=n, m=m)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    cfg = scaled(cfg, k)
    with rpd.RPD(predicate_mode=rpd.PRED_EXACT, knn_k=40, exact_lists=False) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        st = r.compute()
        nbr = r.neighbor_lists(len(cfg["sites"]))
        offs, ps = r.pairs(len(cfg["tets"]))
        ph, p = r.pair_headers(), r.cells()[1]
    assert (st.n_pairs >= MIN_PAIRS) == (n == 14) and st.n_fp64_uncertain > 0
    mesh = dict(vert3d=cfg["vert3d"], tets=cfg["tets"],
                **{q: adj[q] for q in ("v_adjs", "e_adj6", "f_adjs", "f_ids")})
    oh, op, _ = O.clip_cells(mesh, cfg["sites"], nbr, offs, ps, pred_mode=2)
    assert same_records(ph, p, oh, op)


@pytest.mark.parametrize("size", ["lanes", "warps"])
@pytest.mark.parametrize("pred", ["fp64", "fp32_filter", "exact"])
@pytest.mark.parametrize("certify", [False, True])
def test_certified_topology_as_unscaled(size, pred, certify):
    """The radius bounds behind the certificate and the uncertified flags: short
    lists, so that the exact-lists rounds have cells to complete.  A topology
    hash is made of ids, which no scale changes."""
    cfg, adj = scene(size)
    mode = {"fp64": rpd.PRED_FP64, "fp32_filter": rpd.PRED_FP32_FILTER, "exact": rpd.PRED_EXACT}[pred]
    a, ha, _, ta = run(cfg, adj, rpd.PRED_FP64, knn_k=24, certify=certify)
    assert a.n_extended_sites > 0 and a.n_uncertified == 0
    for k in (10, 15, 17, 20, 23, 25, 27, 29):
        b, hb, _, tb = run(scaled(cfg, k), adj, mode, knn_k=24, certify=certify)
        assert b.n_uncertified == 0, k
        assert np.array_equal(ha["status"], hb["status"]), k
        assert np.array_equal(ta, tb), k
