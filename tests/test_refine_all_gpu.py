"""CCD_PATH_REFINE_ALL solves every polynomial of every row, also those whose
list the other rows of CCD_PATH_CULL_REFINE can do without."""
import numpy as np
import pytest

import collisiondetection_gb300 as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
@pytest.mark.parametrize("n", [1, 1000])
def test_every_polynomial_is_solved_in_one_round(kind, n):
    from collisiondetection_gb300 import build as B

    B.build_library()
    # corners of a flat sheet in rigid motion: sextics with roots at t = 0
    rng = np.random.default_rng(5)
    s = 0.25 * rng.integers(0, 4, (n, 4, 3))
    s[:, :, 2] = 0.0
    rows = np.concatenate([s.reshape(n, 12), (s + 0.25 * rng.normal(size=(n, 1, 3))).reshape(n, 12)], 1)
    with C.Context(0) as ctx:
        h64, t64 = ctx.prim_batch(kind, rows, 1e-6, path=C.PATH_FP64)
        ctx.set_profiling(True)
        h, t = ctx.prim_batch(kind, rows, 1e-6, path=C.PATH_REFINE_ALL)
        launches = ctx.timings()["launches"]
    np.testing.assert_array_equal(h, h64)
    np.testing.assert_array_equal(t[h64 == 1].view(np.uint64), t64[h64 == 1].view(np.uint64))
    assert launches == 4  # the row list, build, pool, combine: nothing is left for a second round
