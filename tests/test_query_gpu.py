"""One vertex-face or edge-edge row in FP64 (a cluster of blocks, one list
each) against the one-lane kernel that larger FP64 batches take: the same flag,
the same contact time bit for bit and the same status, whichever list settles
the row."""
import time

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


def _flat(n):
    rng = np.random.default_rng(7)
    h = 1.0 / rng.integers(3, 9, (n, 1, 1))
    s = rng.integers(0, 4, (n, 4, 3)) * h
    s[:, :, 2] = np.where(rng.random((n, 4)) < 0.125, 2.0, 0.0) * h[:, :, 0]
    e = s + rng.normal(size=(n, 1, 3)) * h + rng.choice([0.0, 1e-9, 0.1], (n, 1, 1)) * h * rng.normal(size=s.shape)
    return np.concatenate([s.reshape(n, 12), e.reshape(n, 12)], 1)


def _rows(name, kind):
    if name == "flat":  # solves that fail shift after shift, parallel edges, exact zeros
        return _flat(96)
    if name == "whole":
        rng = np.random.default_rng(3)
        s = rng.integers(-2, 3, (96, 12)).astype(float)
        return np.concatenate([s, s + rng.integers(-2, 3, (96, 12))], 1)
    rows = W.primitive_batch(kind, 96, seed=41)
    if name == "odd":  # not finite, and beyond what a product of coordinates holds
        rng = np.random.default_rng(4)
        rows[np.arange(96), rng.integers(0, 24, 96)] = rng.choice([np.nan, np.inf, -np.inf, 1e160, 1e-300, 3e30], 96)
    return rows


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
@pytest.mark.parametrize("name", ["ordinary", "flat", "whole", "odd"])
def test_one_row_equals_the_one_lane_kernel(ctx, kind, name):
    for row in _rows(name, kind):
        h2, t2 = ctx.prim_batch(kind, np.stack([row, row]), 1e-4, path=C.PATH_FP64)
        st2 = ctx.stats()
        h, t = ctx.prim_batch(kind, row[None], 1e-4, path=C.PATH_FP64)
        st = ctx.stats()
        hit, time_ = ctx.single(kind, row, 1e-4)
        assert h[0] == h2[0] == h2[1] == hit
        assert t[0].view(np.uint64) == t2[0].view(np.uint64)
        if hit:
            assert np.float64(time_).view(np.uint64) == t2[0].view(np.uint64)
        assert [st[k] * 2 for k in ("rows", "survivors", "hits", "status_flags")] == \
            [st2[k] for k in ("rows", "survivors", "hits", "status_flags")]


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
def test_a_query_ends_with_the_list_that_settles_it(ctx, kind):
    # Each row alone against the one-lane kernel on two copies of it: never
    # much slower (the FP32 stage and the pool in its place took up to 6 times
    # as long on rows that one list settles early).
    def least(f):
        f()
        times = []
        for _ in range(5):
            t0 = time.perf_counter()
            f()
            times.append(time.perf_counter() - t0)
        return min(times)

    worst = 0.0
    for row in np.concatenate([_rows("ordinary", kind), _rows("flat", kind)[:48]]):
        two = np.stack([row, row])
        lane = least(lambda: ctx.prim_batch(kind, two, 1e-6, path=C.PATH_FP64))
        worst = max(worst, least(lambda: ctx.single(kind, row, 1e-6)) / lane)
    assert worst < 1.5
