"""Single queries against the FP64 kernel on the same rows: the same flag and,
bit for bit, the same contact time (both form the same polynomials and solve
those that matter with the same root finder)."""
import numpy as np
import pytest

import collisiondetection_gb300 as C
from collisiondetection_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from collisiondetection_gb300 import build as B

    B.build_library()
    c = C.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE, C.VERTEX_EDGE, C.VERTEX_VERTEX])
@pytest.mark.parametrize("scale,eta", [(1.0, 1e-6), (1.0, 1e-2), (1e-3, 1e-6), (1e6, 1e-3)])
def test_single_query_equals_fp64_kernel(ctx, kind, scale, eta):
    # a few hits, misses and near-degenerate rows, and rows that cannot be bounded in FP32
    rows = W.primitive_batch(kind, 4096, seed=9) * scale
    h, t = ctx.prim_batch(kind, rows, eta, path=C.PATH_FP64)
    pick = np.r_[np.flatnonzero(h)[:24], np.flatnonzero(h == 0)[:24]]
    for i in pick:
        hit, time = ctx.single(kind, rows[i], eta)
        assert hit == h[i]
        if hit:
            assert np.float64(time).view(np.uint64) == t[i].view(np.uint64)
    odd = rows[:4].copy()
    odd[0] *= 1e-250
    odd[1] *= 1e150
    odd[2, 0] = np.inf
    odd[3, 1] = np.nan
    h, t = ctx.prim_batch(kind, odd, eta, path=C.PATH_FP64)
    assert [bool(ctx.single(kind, r, eta)[0]) for r in odd] == [bool(v) for v in h]
