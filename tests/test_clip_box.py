"""The box by which the thread-per-cell clipper passes over list entries
(rpd_clip_box.cuh), run on the host: as long as no clip reports a vertex
outside, every vertex lies in the box that the group of entries met, however
often the cell grew by less than the slack."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from libmat_gb300 import build as libbuild
from tests.conftest import ROOT

CPP = os.path.join(ROOT, "tests", "cpp", "cull_box.cpp")


@pytest.fixture(scope="module")
def fit(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("cull_box") / "cull_box.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(libbuild.cuda_home(), "include"), CPP, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    f32 = np.ctypeslib.ndpointer(np.float32, flags="C")
    lib.fit_boxes.argtypes = [f32, ctypes.c_int, ctypes.c_float,
                              np.ctypeslib.ndpointer(np.uint8, flags="C"), f32]

    def run(v, slack):
        v = np.ascontiguousarray(v, np.float32)
        outside, out = np.empty(len(v), np.uint8), np.empty_like(v)
        lib.fit_boxes(v, len(v), slack, outside, out)
        return outside.astype(bool), out

    return run


# steps outwards a clip, in slacks: below, around and above one
@pytest.mark.parametrize("step", [0.0, 0.3, 0.9, 1.1])
@pytest.mark.parametrize("seed", range(5))
def test_vertices_stay_in_the_box_the_group_met(fit, step, seed):
    rng = np.random.default_rng(seed)
    span, slack = 1.0, 1.0 / 1024.0
    n = 8
    lo, hi = -rng.uniform(0.3, 1.0, 3), rng.uniform(0.3, 1.0, 3)
    grow = step * slack * np.arange(n)[:, None]
    v = np.concatenate([lo - grow, np.repeat(hi[None], n, 0), 1.0 + grow], 1).astype(np.float32)
    outside, box = fit(v, slack)
    assert not outside[0]
    ulps = 8 * 2.0 ** -24 * span  # of mid and half, a few clips
    first = 0  # the clip whose box the group met
    for i in range(1, n):
        inside = np.all(v[i, :3] >= box[first, :3] - i * ulps) and \
            np.all(v[i, 3:] <= box[first, 3:] + i * ulps)
        assert outside[i] or inside
        if outside[i]:  # looked over again, by a box around these vertices
            assert np.all(box[i, :3] <= v[i, :3]) and np.all(box[i, 3:] >= v[i, 3:])
            first = i
    assert outside.any() == (step > 0.0)


def test_a_shrinking_cell_keeps_its_slack(fit):
    v = np.array([[-1, -1, -1, 1, 1, 1, 2], [-1, -0.5, -1, 1, 1, 0.5, 1.5]], np.float32)
    outside, box = fit(v, 0.001)
    assert not outside.any()
    assert np.allclose(box[1], [-1.001, -0.501, -1.001, 1.001, 1.001, 0.501, 1.501], atol=1e-6)
