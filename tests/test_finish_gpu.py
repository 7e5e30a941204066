"""The one-solve-per-warp finish of a wavefront batch with work to do: a short
split leaves it solves of every length, and each of its modes gives the bits of
the default split."""
import numpy as np
import pytest

import collisiondetection_gb300 as C
from collisiondetection_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
def test_every_finish_gives_the_bits_of_the_default_split(kind):
    from collisiondetection_gb300 import build as B

    B.build_library()
    rows = W.primitive_batch(kind, 600_000, seed=508)
    with C.Context(0) as ctx:
        h0, t0 = ctx.prim_batch(kind, rows, 1e-6)
    m = h0 == 1
    assert m.any()
    for mode, after in ((None, None), (0, None), (1, None), (2, None), (2, 0), (2, 7)):
        with C.Context(0) as ctx:  # its own defaults for what is not set
            ctx.set_option("wave_steps", 40)
            ctx.set_option("pool_budget", 16)
            if mode is not None:
                ctx.set_option("warp_finish", mode)
            if after is not None:
                ctx.set_option("shift_after", after)
            h, t = ctx.prim_batch(kind, rows, 1e-6)
        np.testing.assert_array_equal(h, h0)
        np.testing.assert_array_equal(t[m].view(np.uint64), t0[m].view(np.uint64))
