"""The predicate counts of a compute are those of its cells: a cell that a lane
gives up and a warp takes up again counts once.  A lane evaluates some of the
signs that clipping the cell plane by plane takes, a warp all of them (and some
for planes that an earlier one of the same step makes void), so the counts of a
compute by lanes are at most those by warps -- which the same sites give a part
at a time, with too few pairs for the lanes."""
import numpy as np
import pytest

from libmat_gb300 import rpd
from libmat_gb300 import workloads as W
from tests.test_gpu_clip_threads import MIN_PAIRS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pred", ["fp32_filter", "exact"])
@pytest.mark.parametrize("n,n_site,k", [(4, 3_000, 127), (5, 2_000, 64)])  # half of the cells outgrow a lane
def test_cells_given_up_count_once(n, n_site, k, pred):
    cfg = W.config_small_cube(n=n, n_site=n_site, seed=5)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    mode = {"fp32_filter": rpd.PRED_FP32_FILTER, "exact": rpd.PRED_EXACT}[pred]

    def counts(flags):
        with rpd.RPD(predicate_mode=mode, knn_k=k, exact_lists=False) as r:
            r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                       adj["f_ids"])
            r.set_sites(cfg["sites"], flags)
            s = r.compute()
        return np.array([s.n_pairs, s.n_predicates, s.n_escalated, s.n_fp64_uncertain,
                         s.n_exact_flips], np.int64)

    lanes = counts(np.ones(n_site, np.uint32))
    parts = [counts((np.arange(n_site) % 4 == i).astype(np.uint32)) for i in range(4)]
    assert lanes[0] >= MIN_PAIRS and all(p[0] < MIN_PAIRS for p in parts)
    warps = np.sum(parts, axis=0)
    assert lanes[0] == warps[0] and lanes[2] > 0
    assert np.all(lanes[1:] <= warps[1:])
