"""The classification of rows (csrc/ccd_classify.h) against the full decision,
on the host: over random and structured rows, every row decided without the
root finder is decided as by all its interval lists, and the rows whose lists
partly stand in give the same flag and the same contact time, bit for bit."""
import ctypes

import numpy as np
import pytest

from collisiondetection_gb300 import workloads as W
from hostcheck import build as hb

P = ctypes.c_void_p
N = 60_000


def _classify(kind, rows, eta):
    lib = ctypes.CDLL(hb._build("hc_classify", "hostcheck_classify.cpp"))
    n = len(rows)
    rows = np.ascontiguousarray(rows)
    eta = np.ascontiguousarray(np.broadcast_to(eta, (n,)), dtype=np.float64)
    out, differs = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
    jobs, solved = np.zeros(n, np.int32), np.zeros(n, np.int32)
    lib.hc_classify(kind, ctypes.c_int64(n), *(a.ctypes.data_as(P) for a in (rows, eta, out, differs, jobs, solved)))
    return out, differs, jobs, solved


def _flat(rng):
    """Corners of a grid sheet in rigid motion, with and without jitter, some a layer apart."""
    h = 1.0 / rng.integers(3, 9, (N, 1, 1))
    s = rng.integers(0, 4, (N, 4, 3)) * h
    s[:, :, 2] = np.where(rng.random((N, 4)) < 0.125, 2.0, 0.0) * h[:, :, 0]
    e = s + rng.normal(size=(N, 1, 3)) * h + rng.choice([0.0, 1e-9, 0.1], (N, 1, 1)) * h * rng.normal(size=(N, 4, 3))
    return s, e


def _family(name, rng):
    if name == "random":
        s = rng.random((N, 4, 3))
        return s, s + rng.normal(0.0, 0.1, s.shape)
    if name == "lattice":
        size = rng.integers(1, 10, (N, 1, 1))
        s = np.rint(rng.uniform(-1, 1, (N, 4, 3)) * size)
        return s, s + np.rint(rng.uniform(-1, 1, (N, 4, 3)) * size)
    if name == "flat":
        return _flat(rng)
    if name == "scaled":
        s = rng.random((N, 4, 3)) * 10.0 ** rng.uniform(-6, 4, (N, 1, 1))
        return s, s + s * rng.normal(size=s.shape) * 10.0 ** rng.uniform(-6, 2, (N, 1, 1))
    if name == "static":  # some points still, some motions along one axis
        s = rng.random((N, 4, 3))
        return s, s + 0.3 * rng.normal(size=s.shape) * (rng.random((N, 4, 1)) < 0.5) * np.where(
            rng.random((N, 1, 1)) < 0.5, 1.0, np.eye(3)[rng.integers(0, 3, N)][:, None])
    if name == "small":  # short edges far from the origin, one feature moving rigidly
        s = rng.random((N, 1, 3)) + 0.01 * rng.normal(size=(N, 4, 3))
        e = s + 0.01 * rng.normal(size=(N, 1, 3)) * np.array([1.0, 1.0, 0.0, 0.0])[:, None]
        return s, e + 0.001 * rng.normal(size=s.shape) * (rng.random((N, 1, 1)) < 0.25)
    # opposite double roots of the sextic, their moduli a few percent apart or less
    s = rng.random((N, 4, 3))
    e = s + rng.normal(0.0, 0.1, s.shape)
    t = rng.random((N, 1)) * 0.9 + 0.05
    back = -t * (1.0 + 0.03 * rng.normal(size=t.shape))
    for _ in range(4):
        for at in (t, back):
            x = s + at[:, :, None] * (e - s)
            n = np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
            d = (np.einsum("ij,ij->i", x[:, 3] - x[:, 0], n) / np.einsum("ij,ij->i", n, n))[:, None] * n
            other = np.where(at is t, back, t)
            s[:, 3] -= d * (-other) / (at - other)
            e[:, 3] -= d * (1.0 - other) / (at - other)
    return s, e


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("family", ["random", "lattice", "flat", "scaled", "static", "small", "mirrored"])
def test_decides_as_all_lists_do(family, kind):
    rng = np.random.default_rng([11, kind, len(family)])
    s, e = _family(family, rng)
    rows = np.concatenate([s.reshape(N, 12), e.reshape(N, 12)], 1)
    eta = np.where(rng.random(N) < 0.5, 1e-6, 10.0 ** rng.uniform(-8, -2, N))
    out, differs, _, _ = _classify(kind, rows, eta)
    assert (out > 0).any()
    assert differs.sum() == 0


@pytest.mark.parametrize("kind", [0, 1])
def test_leaves_little_of_the_benchmark_rows(kind):
    # 20% near-degenerate rows: coplanar, parallel and tangential ones included
    rows = W.primitive_batch(kind, 200_000, seed=21)
    out, differs, jobs, solved = _classify(kind, rows, 1e-6)
    assert differs.sum() == 0
    assert solved.sum() < (0.30 if kind == 0 else 0.16) * jobs.sum()


@pytest.mark.parametrize("kind", [0, 1])
def test_takes_no_row_that_it_cannot_bound(kind):
    # vanishing, infinite and NaN coefficients, and leading coefficients that
    # are exactly zero, are left to the full solve
    rng = np.random.default_rng(3)
    rows = rng.random((4000, 24))
    rows[:, 12:] = rows[:, :12] + 0.1 * rng.normal(size=(4000, 12))
    rows[0::4, 12:] = rows[0::4, :12]
    rows[1::4, rng.integers(0, 24)] = np.nan
    rows[2::4, rng.integers(0, 24)] = np.inf
    rows[3::4] *= 1e-60
    out, differs, _, _ = _classify(kind, rows[np.r_[0:4000:4, 3:4000:4]], 1e-6)
    assert set(np.unique(out)) <= {0, 4}
    assert differs.sum() == 0


def test_leaves_rows_of_far_apart_coefficients_to_the_solver():
    # coordinates 70 orders of magnitude apart: the solver loses a root of the
    # second side and reports it positive up to t = 1, which decides the row
    row = [
        1.3412941393225036e-09, 7.680402678565238e-30, 1.1797703088715006e-29, 1.6909395566468181e-40,
        28123401653.643394, 6.661879818881568e-09, 1.2909404345665422e+24, 1.758315190363229e+32,
        6.990541081300586e-27, 1.0676368764076317e+18, 6.840042438680488e-28, 1.6032392515276564e-06,
        532036290.6228999, 1.9107187881559787e-34, 7526.8785214051695, 1.132284335397677e-37, 0.42749773874772373,
        1.6464199379580506e-06, 1.1066387145431088e+26, 0.001784983565492135, 4.324384243362487e+23,
        1.9697658226502924e-29, 3.344853031520508e-11, 0.001334615982166079,
    ]
    out, differs, _, _ = _classify(0, np.array([row]), 1e-6)
    assert out[0] == 4 and not differs[0]
