"""Cones and slabs (rpd_dist2mat) whose larger sphere holds the others: the
radicand of a cone is negative and its parameter no number, which the device
takes for the larger sphere -- the least distance over the primitive, as the
oracle's convex minimisation has it.  (The oracle's restatement of the
reference's clamp on the CPU takes it for the smaller sphere.)"""
import numpy as np
import pytest

from libmat_gb300 import rpd
from oracle import dist2mat_oracle as D

pytestmark = pytest.mark.gpu


def scene(seed, n=120):
    """n samples, each with a large sphere and two inside it, in a random order."""
    rng = np.random.default_rng(seed)
    big = np.c_[rng.uniform(0, 1, (n, 3)), rng.uniform(0.2, 0.4, n)]
    sph = np.repeat(big[:, None], 3, 1)
    sph[:, 1:, 3] = rng.uniform(0.02, 0.08, (n, 2))
    sph[:, 1:, :3] += rng.uniform(-0.06, 0.06, (n, 2, 3))  # |c - c'| + r' < 0.104 + 0.08 < r
    sph = np.take_along_axis(sph, rng.permuted(np.tile(np.arange(3), (n, 1)), axis=1)[:, :, None], 1)
    return sph.reshape(-1, 4).astype(np.float32), rng.uniform(-1, 2, (n, 3)).astype(np.float32)


def device(sph, smp, prims):
    n = len(smp)
    with rpd.RPD() as r:
        return r.dist2mat(sph, smp, np.arange(n, dtype=np.uint32), np.ones(n, np.uint32),
                          np.ascontiguousarray(prims, np.int32))[0]


@pytest.mark.parametrize("seed", [0, 1])
def test_contained_spheres(seed):
    sph, smp = scene(seed)
    n = len(smp)
    ids = np.arange(3 * n).reshape(n, 3)
    largest = ids[np.arange(n), np.argmax(sph[:, 3].reshape(n, 3), axis=1)]
    none = np.full(n, -1)
    ball = device(sph, smp, np.stack([none, none, largest], 1))
    others = np.array([np.setdiff1d(ids[i], largest[i]) for i in range(n)])
    # a cone of the large sphere with one inside it, either way round
    for pair in ((largest, others[:, 0]), (others[:, 1], largest)):
        cone = device(sph, smp, np.stack([none, *pair], 1))
        assert np.array_equal(cone, ball)
        for i in range(n):
            m1, m2 = (sph[q[i]].astype(np.float64) for q in pair)
            assert abs(cone[i] - D.numeric_cone_d(smp[i].astype(np.float64), m1, m2)) < 1e-6
    # a slab whose closed form has no point inside: its cones, two with the
    # large sphere and one of the two in it, which is farther
    slab = device(sph, smp, ids)
    seen = 0
    for i in range(n):
        m = [sph[q] for q in ids[i]]
        with np.errstate(all="ignore"):
            edges = min(D.cone_d(smp[i], m[a], m[b]) for a, b in ((0, 2), (1, 2), (0, 1)))
            if D.slab_d(smp[i], *m) == edges:
                assert slab[i] == ball[i]
                seen += 1
    assert seen > n // 2
