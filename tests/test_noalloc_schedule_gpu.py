"""The allocation-free batch solves on the schedule of the context's batches."""
import ctypes
import time

import numpy as np
import pytest

import collisiondetection_gb300 as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
@pytest.mark.parametrize("n", [64, 1000])
def test_flat_rows_take_no_longer_than_in_a_context(kind, n):
    # Corners of a flat sheet, whose sextics fail shift after shift: the same
    # results and about the same time (7 to 9 times as long, 1,000 rows, when
    # this call alone kept the schedule of before).
    torch = pytest.importorskip("torch")
    from collisiondetection_gb300 import build as B

    B.build_library()
    rng = np.random.default_rng(7)
    h = 1.0 / rng.integers(3, 9, (n, 1, 1))
    s = rng.integers(0, 4, (n, 4, 3)) * h
    s[:, :, 2] = np.where(rng.random((n, 4)) < 0.125, 2.0, 0.0) * h[:, :, 0]
    e = s + rng.normal(size=(n, 1, 3)) * h + rng.choice([0.0, 1e-9, 0.1], (n, 1, 1)) * h * rng.normal(size=s.shape)
    rows = torch.from_numpy(np.concatenate([s.reshape(n, 12), e.reshape(n, 12)], 1)).cuda()
    eta = torch.full((1,), 1e-6, dtype=torch.float64, device="cuda")
    hit = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2)]
    t = [torch.full((n,), -1.0, dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    with C.Context(0) as ctx:
        fn = ctx.lib.ccd_prim_batch_device_noalloc
        fn.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p,
                       ctypes.c_void_p, ctypes.c_void_p]
        fn.restype = ctypes.c_int

        def in_context():
            ctx.prim_batch_device(kind, n, rows.data_ptr(), eta.data_ptr(), 1, hit[0].data_ptr(), t[0].data_ptr())
            ctx.synchronize()

        def noalloc():
            assert fn(kind, n, rows.data_ptr(), eta.data_ptr(), 1, hit[1].data_ptr(), t[1].data_ptr(), None) == 0
            torch.cuda.synchronize()

        def median(f):
            f()
            times = []
            for _ in range(7):
                t0 = time.perf_counter()
                f()
                times.append(time.perf_counter() - t0)
            return float(np.median(times))

        a, b = median(in_context), median(noalloc)
    assert torch.equal(hit[0], hit[1]) and torch.equal(t[0].view(torch.int64), t[1].view(torch.int64))
    assert b <= 2.5 * a
