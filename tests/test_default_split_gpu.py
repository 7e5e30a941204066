"""The default split of the root solves (lock-step steps, then the pool) depends
on the batch size; a split only reschedules the solves, so flags and contact
times equal those of an explicit long split bit for bit."""
import numpy as np
import pytest

import collisiondetection_gb300 as C
from collisiondetection_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [C.VERTEX_FACE, C.EDGE_EDGE])
@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, (1 << 21) + 1, 1 << 22])
def test_default_split_equals_explicit_split(kind, n):
    torch = pytest.importorskip("torch")
    from collisiondetection_gb300 import build as B

    B.build_library()
    ctx = C.Context(0)
    dev = torch.device("cuda", 0)
    base = torch.from_numpy(W.primitive_batch(kind, 1 << 18, seed=17)).to(dev)
    rows = base.repeat((n + (1 << 18) - 1) >> 18, 1)[:n].contiguous()
    rows[:, :12] += torch.linspace(0.0, 0.01, n, dtype=torch.float64, device=dev)[:, None] * base.std()
    eta = torch.tensor([1e-6], dtype=torch.float64, device=dev)
    out = []
    for split in (None, (63, 63)):
        if split:
            ctx.set_option("wave_steps", split[0])
            ctx.set_option("pool_budget", split[1])
        hit = torch.zeros(n, dtype=torch.uint8, device=dev)
        t = torch.full((n,), -1.0, dtype=torch.float64, device=dev)
        torch.cuda.synchronize()
        ctx.prim_batch_device(kind, n, rows.data_ptr(), eta.data_ptr(), 1, hit.data_ptr(), t.data_ptr())
        ctx.synchronize()
        out.append((hit, t.view(torch.int64)))
    ctx.close()
    assert out[0][0].any()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
