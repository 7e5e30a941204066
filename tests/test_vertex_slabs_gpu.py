"""The 13-DOP leaf slabs, formed from slabs per vertex, against the oracle's
candidates where the two ways of forming them could part: NaN positions,
vertices that few faces or none use."""
import os
import sys
import time

import numpy as np
import pytest

import collisiondetection_gb300 as C
from collisiondetection_gb300 import workloads as W

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def orc():
    from collisiondetection_gb300 import build as B

    B.build_library()
    O.build()
    return O.Oracle()


@pytest.mark.parametrize("kind", [C.BROADPHASE_KDOP13, C.BROADPHASE_AABB])
@pytest.mark.parametrize("share", [0.02, 0.3])
def test_nan_start_positions(orc, kind, share):
    # NaN at the start, ordinary at the end: every face's bounds are ordinary
    # numbers again after its last entry, without what came before the NaN.
    rng = np.random.default_rng(6)
    q0, q1, f = W.two_spheres(3, level=2)
    q0 = q0.reshape(-1, 3).copy()
    bad = rng.random(len(q0)) < share
    q0[bad, rng.integers(0, 3, int(bad.sum()))] = np.nan
    q0 = q0.ravel()
    with C.Context(0) as ctx, C.Mesh(ctx, f, q0, q1) as m:
        vf, ee = m.broadphase(kind, 1e-6)
        again = m.broadphase(kind, 1e-6)  # the kept tree, refitted
    ovf, oee = orc.broadphase(kind, q0, q1, f, 1e-6)
    for a, b in ((vf, ovf), (ee, oee), (again[0], ovf), (again[1], oee)):
        np.testing.assert_array_equal(a, b)


def _soup(rng, n):
    """n triangles that share no vertex."""
    q0 = rng.random((n, 1, 3)) + 0.1 * rng.normal(size=(n, 3, 3))
    q1 = q0 + 0.05 * rng.normal(size=(n, 1, 3))
    return q0.ravel(), q1.ravel(), np.arange(3 * n, dtype=np.int32).reshape(n, 3)


@pytest.mark.parametrize("kind", [C.BROADPHASE_KDOP13, C.BROADPHASE_AABB])
@pytest.mark.parametrize("mesh", ["bare", "bare_first", "soup", "pair"])
def test_vertices_that_few_or_no_faces_use(orc, kind, mesh):
    rng = np.random.default_rng(8)
    if mesh == "soup":  # more than two vertices a face
        q0, q1, f = _soup(rng, 600)
    elif mesh == "pair":  # the smallest mesh with a tree
        q0, q1, f = _soup(rng, 2)
        q1 = q0.copy()
        q1[9:] = q0[:9]
    else:  # vertices that no face uses, after and between the others
        q0, q1, f = W.two_spheres(3, level=2)
        n = q0.size // 3
        at = np.arange(n) if mesh == "bare" else np.sort(rng.permutation(3 * n)[:n])
        a, b = rng.random((3 * n, 3)), rng.random((3 * n, 3))
        a[at], b[at] = q0.reshape(-1, 3), q1.reshape(-1, 3)
        q0, q1, f = a.ravel(), b.ravel(), at[f].astype(np.int32)
    ovf, oee = orc.broadphase(kind, q0, q1, f, 1e-6)
    with C.Context(0) as ctx, C.Mesh(ctx, f, q0, q1) as m:
        for _ in range(2):  # a new tree, then the kept one
            vf, ee = m.broadphase(kind, 1e-6)
            np.testing.assert_array_equal(vf, ovf)
            np.testing.assert_array_equal(ee, oee)


def test_bare_vertices_cost_nothing():
    # Two million vertices that no face uses beside 20,480 faces' own (1.6
    # times the broad phase when every vertex had slabs).
    q0, q1, f = W.two_spheres(1, level=5)
    extra = np.random.default_rng(0).random(6_000_000) * 0.5

    def median(a, b):
        with C.Context(0) as ctx, C.Mesh(ctx, f, a, b) as m:
            times = []
            for _ in range(20):
                t0 = time.perf_counter()
                m.broadphase(C.BROADPHASE_KDOP13, 1e-6)
                times.append(time.perf_counter() - t0)
        return float(np.median(times[5:]))

    q0, q1 = q0.ravel(), q1.ravel()
    assert median(np.concatenate([q0, extra]), np.concatenate([q1, extra])) < 1.25 * median(q0, q1)
