"""The GPU's neighbour lists (knn_kernel) at the sizes where its sorts change:
list lengths around the powers of two, more and fewer sites than entries, ties
in the key (lattice sites, sites on one another) and long lists of the
exact-lists rounds -- against the oracle's lists, key by key and id by id."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu

_mesh = W.cube_grid_mesh(2)


def lists(sites, k, order):
    vert, tets = _mesh[0] * 1000.0, _mesh[1]
    adj = rpd.mesh_adjacency(vert.shape[0], tets)
    with rpd.RPD(knn_k=k, clip_order=order, exact_lists=False) as r:
        r.set_mesh(vert, tets, adj["v_adjs"], adj["e_adj6"], adj["f_adjs"], adj["f_ids"])
        r.set_sites(sites)
        r.compute()
        return r.neighbor_lists(len(sites))


def sites_of(kind, n):
    rng = np.random.default_rng(n)
    if kind == "lattice":
        m = int(round(n ** (1 / 3)))
        g = (np.arange(m) + 0.5) * (1000.0 / m)
        xyz = np.stack(np.meshgrid(g, g, g), -1).reshape(-1, 3)
        return np.concatenate([xyz, np.full((len(xyz), 1), 100.0)], 1)
    xyz = rng.uniform(0.0, 1000.0, (n, 3))
    if kind == "clustered":  # a third of the sites in 1 % of the volume
        xyz[: n // 3] = 500.0 + rng.normal(0.0, 30.0, (n // 3, 3))
    if kind == "stacked":
        xyz[: n // 4] = xyz[n // 4: 2 * (n // 4)]
    r = rng.uniform(5.0, 60.0, n)
    return np.concatenate([xyz, (r * r)[:, None]], 1)


@pytest.mark.parametrize("kind,n", [("uniform", 1), ("uniform", 40), ("uniform", 900),
                                    ("clustered", 3_000), ("stacked", 700), ("lattice", 1_000)])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64, 65, 127, 128])
def test_lists_match_the_oracle(kind, n, k):
    s = sites_of(kind, n)
    want, _ = O.knn(s.astype(np.float32), k)
    got = lists(s, k, rpd.ORDER_SITE_ID)
    by_id = np.where(want < 0, np.iinfo(np.int32).max, want)
    by_id.sort(axis=1)
    assert np.array_equal(np.where(got < 0, np.iinfo(np.int32).max, got), by_id)
    assert np.array_equal(lists(s, k, rpd.ORDER_DISTANCE), want)
