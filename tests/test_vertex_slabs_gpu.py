"""The 13-DOP leaf slabs, formed from slabs per vertex, against the oracle's
candidates where the two ways of forming them could part: NaN positions."""
import os
import sys

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
