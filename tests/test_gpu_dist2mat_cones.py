"""Cone distances (rpd_dist2mat) where the radicand of the closest sphere is
hard to round or out of the float pairs' range: samples on a cone's axis, nearly
tangent and equal spheres, coordinates of few bits, tiny and huge scenes --
bit for bit the closed form with the radicand in float64."""
import numpy as np
import pytest

from libmat_gb300 import rpd
pytestmark = pytest.mark.gpu


def scene(kind, scale, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0.0, 1.0, (60, 3))
    r = rng.uniform(0.01, 0.05, 60)
    a, b = rng.integers(0, 30, 1500), rng.integers(30, 60, 1500)
    t = rng.uniform(-0.5, 1.5, 1500)
    smp = rng.uniform(0.0, 1.0, (1500, 3))
    if kind == "axis":
        smp = c[a] + t[:, None] * (c[b] - c[a])
    elif kind == "tangent":
        r[30:] = r[:30].mean() + np.linalg.norm(c[30:] - c[:30], axis=1) * (1.0 - 1e-6)
        b = a + 30
    elif kind == "equal":
        r[:] = 0.03
    elif kind == "grid":  # sums and products of few bits
        c, r, smp = np.round(c * 16) / 16, np.round(r * 64) / 64, np.round(smp * 16) / 16
    sph = np.c_[c * scale, r * scale].astype(np.float32)
    prims = np.stack([np.full(1500, -1), a, b], 1).astype(np.int32)
    same = np.all(sph[a] == sph[b], axis=1) | np.all(sph[a, :3] == sph[b, :3], axis=1)
    prims[same, 1] = -1  # one centre: a sphere
    return sph, (smp * scale).astype(np.float32), prims


def closed_form(sph, smp, prims):
    """cone_d of oracle/dist2mat_oracle.py over arrays, but for a parameter that
    is no number (a negative radicand, 0 / 0), which the device's clamp takes to 0."""
    f, d = np.float32, np.float64
    cone = prims[:, 1] >= 0
    m1, m2 = sph[prims[:, 1]].copy(), sph[prims[:, 2]].copy()
    swap = m1[:, 3] > m2[:, 3]
    m1[swap], m2[swap] = m2[swap].copy(), m1[swap].copy()

    def dot(a, b):
        return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]

    c21, cq2 = m1[:, :3] - m2[:, :3], m2[:, :3] - smp
    A, B, F = dot(c21, c21), f(2) * dot(c21, cq2), dot(cq2, cq2)
    R = m1[:, 3] - m2[:, 3]
    with np.errstate(all="ignore"):
        arg = (d(B * B) - 4.0 * d(A) * d(F)) * d(R * R - A) * d(R) * d(R)
        t = (-(A * B - R * R * B) - np.sqrt(arg.astype(f))) / (f(2) * (A * A - A * R * R))
    t = np.where(np.isnan(t), f(0), np.fmax(f(0), np.fmin(t, f(1))))
    s = np.where(cone[:, None], m2 + t[:, None] * (m1 - m2), sph[prims[:, 2]])
    e = smp - s[:, :3]
    return np.sqrt(dot(e, e)) - s[:, 3]


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e9])
@pytest.mark.parametrize("kind", ["free", "axis", "tangent", "equal", "grid"])
def test_cones_equal_the_closed_form(kind, scale):
    sph, smp, prims = scene(kind, scale, 5)
    offs, cnts = np.arange(1500, dtype=np.uint32), np.ones(1500, np.uint32)
    with rpd.RPD() as r:
        dist, closest = r.dist2mat(sph, smp, offs, cnts, prims)
    assert np.array_equal(dist, closed_form(sph, smp, prims))
    assert np.all(closest == 0)
