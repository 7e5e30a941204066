"""How the refinement's kernels are scheduled, by times of one process that lie
well apart when a kernel waits for another without need.  Both sides of every
comparison are medians on the same GPU; the results are those of the other
tests."""
import time

import numpy as np
import pytest

import collisiondetection_gb300 as C

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
