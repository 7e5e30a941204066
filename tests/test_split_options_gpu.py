"""The split of the root solves as a caller sets it: a value that is set is
taken, whatever it is, and the autotuner reports the split that runs."""
import numpy as np
import pytest

import collisiondetection_gb300 as C
from collisiondetection_gb300 import workloads as W

pytestmark = pytest.mark.gpu

N = 300_000
# besides the lock-step steps: the FP32 stage, build, wave start, gather, pool, finish, combine and the second
# round's pool and combine
OTHERS = 9


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    from collisiondetection_gb300 import build as B

    B.build_library()
    return torch


def _batch(torch, kind):
    rows = torch.from_numpy(W.primitive_batch(kind, N, seed=23)).cuda()
    eta = torch.full((1,), 1e-6, dtype=torch.float64, device="cuda")
    hit = torch.zeros(N, dtype=torch.uint8, device="cuda")
    t = torch.full((N,), -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return kind, rows, eta, hit, t


def _run(ctx, batch):
    """Kernels launched by one batch, and its results."""
    kind, rows, eta, hit, t = batch
    ctx.set_profiling(True)
    ctx.prim_batch_device(kind, N, rows.data_ptr(), eta.data_ptr(), 1, hit.data_ptr(), t.data_ptr())
    ctx.synchronize()
    n = ctx.timings()["launches"]
    ctx.set_profiling(False)
    return n, hit.cpu().numpy(), t.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
@pytest.mark.parametrize("set_, steps", [({}, 4), ({"wave_steps": 64, "pool_budget": 64}, 64), ({"wave_steps": 64}, 64),
                                         ({"pool_budget": 64}, 64), ({"wave_steps": 5}, 5),
                                         ({"wave_steps": 7, "pool_budget": 0}, 7)])
def test_a_split_that_is_set_is_taken(torch, kind, set_, steps):
    batch = _batch(torch, kind)
    with C.Context(0) as ctx:
        _, h0, t0 = _run(ctx, batch)
        for name, value in set_.items():
            ctx.set_option(name, value)
        launches, h, t = _run(ctx, batch)
    assert launches == steps + OTHERS
    assert np.array_equal(h, h0) and np.array_equal(t, t0)


@pytest.mark.parametrize("set_", [{}, {"wave_steps": 64, "pool_budget": 64}])
def test_autotuner_reports_what_runs(torch, set_):
    batch = _batch(torch, C.VERTEX_FACE)
    kind, rows, eta, _, _ = batch
    with C.Context(0) as ctx:
        for name, value in set_.items():
            ctx.set_option(name, value)
        before, _, _ = _run(ctx, batch)
        res = ctx.autotune_prim_batch(kind, N, rows.data_ptr(), eta.data_ptr(), 1, reps=1)
        launches, _, _ = _run(ctx, batch)
    if res["wave_min_rows"] <= N:
        assert launches == res["wave_steps"] + OTHERS
    else:
        assert launches == 6  # the pool alone
    if res["chosen"] == 0:
        assert launches == before
