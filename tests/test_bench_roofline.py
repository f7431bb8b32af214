"""The roofline entry of the bench line names the kernels that the first
clipping pass ran, and gives captured counters only for those they are of."""
import re

import pytest

import bench
from tests.conftest import ROOT


def test_lane_pairs_are_the_dispatch_rules():
    src = open(ROOT + "/libmat_gb300/csrc/rpd_clip_thread.cu").read()
    assert bench.CLIP_LANE_PAIRS == int(re.search(r"kThreadsPairs = (\d+);", src).group(1))


@pytest.mark.parametrize("n_pairs,shortened,lanes", [(20_000, False, True), (19_999, False, False),
                                                   (4_000_000, True, False), (0, False, False)])
def test_kernels_and_counters(n_pairs, shortened, lanes):
    r = bench.clip_pass(n_pairs, shortened)
    assert ("clip_threads_kernel" in r["kernel"]) == lanes and "clip_cells_kernel" in r["kernel"]
    assert all((r[k] is not None) == lanes for k in ("traffic", "issue_active_frac",
                                                     "threads_per_inst"))
    if lanes:
        assert r["traffic"] == pytest.approx(n_pairs * bench.CLIP_DRAM_BYTES_PER_PAIR)
