"""The broad phase's key sorts at the sizes where their two forms and their
blocks change: candidate lists (sorted, duplicates removed) against the
oracle's."""
import os
import sys

import numpy as np
import pytest

import collisiondetection_gb300 as C
from collisiondetection_gb300 import workloads as W

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _sheets(n, seed):
    """Two n x n sheets a tenth of a cell apart that pass through each other."""
    rng = np.random.default_rng(seed)
    v, f = W.grid_sheet(n, n)
    h = 1.0 / (n - 1)
    q0 = np.concatenate([v, v + [0.3 * h, 0.2 * h, 0.1 * h]])
    q1 = q0 + 0.05 * h * rng.normal(size=q0.shape)
    q1[len(v):, 2] -= 0.2 * h
    return q0.ravel(), q1.ravel(), np.concatenate([f, f + len(v)]).astype(np.int32)


# Six keys per face pair for the vertex-face list, nine for the edge-edge one:
# from a handful through one block's 2,048 keys, a few blocks, every SM, to more
# than 2^22 edge-edge keys (a launch per pass).
@pytest.mark.parametrize("n", [2, 3, 5, 8, 12, 40, 210])
@pytest.mark.parametrize("kind", [C.BROADPHASE_KDOP13, C.BROADPHASE_AABB])
def test_candidates_across_sort_sizes(kind, n):
    O.build()
    q0, q1, f = _sheets(n, n)
    with C.Context(0) as ctx, C.Mesh(ctx, f, q0, q1) as m:
        vf, ee = m.broadphase(kind, 1e-6)
        pairs = m.stats()["face_pairs"]
    ovf, oee = O.Oracle().broadphase(kind, q0, q1, f, 1e-6)
    np.testing.assert_array_equal(vf, ovf)
    np.testing.assert_array_equal(ee, oee)
    if n == 210:
        assert 9 * pairs > 1 << 22
