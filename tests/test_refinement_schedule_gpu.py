"""How the refinement's kernels are scheduled, by times of one process that lie
well apart when a kernel waits for another without need.  Both sides of every
comparison are medians on the same GPU; the results are those of the other
tests."""
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


def _median(f, reps=15):
    for _ in range(3):
        f()
    times = []
    for _ in range(reps):
        t0 = time.perf_counter()
        f()
        times.append(time.perf_counter() - t0)
    return float(np.median(times))


def _still(n):
    """One point of each row moves, the other feature and the point's own edge's far end are still."""
    rng = np.random.default_rng(5)
    s = rng.random((n, 4, 3)) * 0.3
    e = s.copy()
    e[:, :1] += 0.2 * rng.normal(size=(n, 1, 3))
    return np.concatenate([s.reshape(n, 12), e.reshape(n, 12)], 1)


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
def test_kernels_do_not_wait_on_the_sms(ctx, kind):
    # Rows without a solve: the GPU is nearly empty at either size, so they
    # take the same time (4.1 and 4.4 times when the blocks of the next
    # kernels held the SMs' shared memory while the first one still ran).
    torch = pytest.importorskip("torch")

    def batch(n):
        rows = torch.from_numpy(_still(n)).cuda()
        eta = torch.full((1,), 1e-6, dtype=torch.float64, device="cuda")
        hit = torch.zeros(n, dtype=torch.uint8, device="cuda")
        t = torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()

        def run():
            ctx.prim_batch_device(kind, n, rows.data_ptr(), eta.data_ptr(), 1, hit.data_ptr(), t.data_ptr())
            ctx.synchronize()

        return run

    assert _median(batch(17_576)) <= 2.0 * _median(batch(1000))


def _flat(rng, n):
    """Corners of a grid sheet in rigid motion, with and without jitter, some a layer apart."""
    h = 1.0 / rng.integers(3, 9, (n, 1, 1))
    s = rng.integers(0, 4, (n, 4, 3)) * h
    s[:, :, 2] = np.where(rng.random((n, 4)) < 0.125, 2.0, 0.0) * h[:, :, 0]
    e = s + rng.normal(size=(n, 1, 3)) * h + rng.choice([0.0, 1e-9, 0.1], (n, 1, 1)) * h * rng.normal(size=s.shape)
    return np.concatenate([s.reshape(n, 12), e.reshape(n, 12)], 1)


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
def test_small_flat_batch_finishes_its_last_solves_together(kind):
    # Sextics of a flat sheet fail shift after shift; a warp that holds one as
    # its last solve tries the shifts at once, also when it fills one slot
    # only (the default), which is no slower than filling four (by 5.6 when it
    # did not notice that its solve was the last: 27 ms instead of 4.8).
    rows = _flat(np.random.default_rng(7), 64)
    with C.Context(0) as ctx:
        one = _median(lambda: ctx.prim_batch(kind, rows, 1e-6), 7)
        h1, t1 = ctx.prim_batch(kind, rows, 1e-6)
        ctx.set_option("pool_slots_min", 4)
        four = _median(lambda: ctx.prim_batch(kind, rows, 1e-6), 7)
        h4, t4 = ctx.prim_batch(kind, rows, 1e-6)
        h64, t64 = ctx.prim_batch(kind, rows, 1e-6, path=C.PATH_FP64)
    for h, t in ((h1, t1), (h4, t4)):
        np.testing.assert_array_equal(h, h64)
        np.testing.assert_array_equal(t[h64 == 1].view(np.uint64), t64[h64 == 1].view(np.uint64))
    assert one <= 2.0 * four


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
@pytest.mark.parametrize("n", [1, 33, 5000])
def test_still_rows_equal_fp64_kernel(ctx, kind, n):
    # Sextics whose leading coefficient vanishes beside ordinary ones in the
    # same warp: the sextic formed once serves the bounds and the queue.
    rows = _still(n)
    rows[::3] = W.primitive_batch(kind, n, seed=13)[::3]
    h64, t64 = ctx.prim_batch(kind, rows, 1e-3, path=C.PATH_FP64)
    for path in (C.PATH_CULL_REFINE, C.PATH_REFINE_ALL):
        h, t = ctx.prim_batch(kind, rows, 1e-3, path=path)
        np.testing.assert_array_equal(h, h64)
        np.testing.assert_array_equal(t[h64 == 1].view(np.uint64), t64[h64 == 1].view(np.uint64))


@pytest.mark.parametrize("seed", [1, 354])
def test_solves_that_fail_few_shifts_are_not_tried_all_at_once(seed):
    # Batches whose slowest solve ends in the third or fourth shift of a stage:
    # about as fast as with the shifts one by one (1.6 times as long and more
    # when the rest were tried at once after two).
    rows = W.primitive_batch(C.EDGE_EDGE, 20_001, seed=seed)
    with C.Context(0) as ctx:
        default = _median(lambda: ctx.prim_batch(C.EDGE_EDGE, rows, 1e-6), 7)
        h0, t0 = ctx.prim_batch(C.EDGE_EDGE, rows, 1e-6)
        ctx.set_option("warp_finish", 1)
        one_by_one = _median(lambda: ctx.prim_batch(C.EDGE_EDGE, rows, 1e-6), 7)
        h1, t1 = ctx.prim_batch(C.EDGE_EDGE, rows, 1e-6)
    np.testing.assert_array_equal(h0, h1)
    np.testing.assert_array_equal(t0[h0 == 1].view(np.uint64), t1[h0 == 1].view(np.uint64))
    assert default <= 1.3 * one_by_one
