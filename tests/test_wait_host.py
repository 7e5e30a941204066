"""The distance sextics that wait for a row's other lists
(csrc/ccd_classify.h), on the host: a row settled without its sextic misses in
the full decision too, over features that start in contact."""
import ctypes

import numpy as np
import pytest

from hostcheck import build as hb

P = ctypes.c_void_p
N = 40_000


def _lib():
    return ctypes.CDLL(hb._build("hc_wait", "hostcheck_wait.cpp"))


def _decide(kind, rows, eta):
    n = len(rows)
    rows = np.ascontiguousarray(rows)
    eta = np.ascontiguousarray(np.broadcast_to(eta, (n,)), dtype=np.float64)
    out, hit = np.zeros(n, np.uint8), np.zeros(n, np.uint8)
    _lib().hc_wait(kind, ctypes.c_int64(n), *(a.ctypes.data_as(P) for a in (rows, eta, out, hit)))
    return out, hit


def _moved(rng, s, h):
    """Rigid motion of all points, of the second half alone, or of each point, with and without jitter."""
    e = s + rng.normal(size=(N, 1, 3)) * h * rng.choice([0.0, 1.0], (N, 1, 1))
    e[:, 2:] += rng.normal(size=(N, 1, 3)) * h * rng.choice([0.0, 0.3], (N, 1, 1))
    return e + rng.choice([0.0, 1e-9, 0.1], (N, 1, 1)) * h * rng.normal(size=s.shape)


def _family(name, rng, kind):
    h = 1.0 / rng.integers(3, 9, (N, 1, 1))
    if name == "sheet":  # corners of a grid sheet, some a layer apart
        s = rng.integers(0, 4, (N, 4, 3)) * h
        s[:, :, 2] = np.where(rng.random((N, 4)) < 0.125, 2.0, 0.0) * h[:, :, 0]
    elif name == "coplanar":  # in a plane at the start
        s = rng.random((N, 4, 3))
        s[:, :, 2] = 0.5
    elif name == "shared":  # features that share a point at the start
        s = rng.random((N, 4, 3))
        s[:, 2 if kind else 0] = s[:, 1]
    elif name == "parallel":  # edges parallel, or a point in the face's plane and moving along it
        s = rng.random((N, 4, 3))
        s[:, 3] = s[:, 2] + (s[:, 1] - s[:, 0]) * rng.choice([1.0, -0.5, 2.0], (N, 1))
        s[:, 2:] += rng.choice([0.0, 1e-7, 1e-3], (N, 1, 1)) * rng.normal(size=(N, 1, 3))
    else:  # whole numbers: exact zeros among the coefficients
        s = rng.integers(-2, 3, (N, 4, 3)).astype(float)
        return s, s + rng.integers(-2, 3, (N, 4, 3)) * (rng.random((N, 4, 1)) < 0.7)
    return s, _moved(rng, s, h)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("family", ["sheet", "coplanar", "shared", "parallel", "whole"])
def test_settled_rows_miss(family, kind):
    rng = np.random.default_rng([17, kind, len(family)])
    s, e = _family(family, rng, kind)
    rows = np.concatenate([s.reshape(N, 12), e.reshape(N, 12)], 1)
    eta = np.where(rng.random(N) < 0.5, 1e-6, 10.0 ** rng.uniform(-8, -2, N))
    out, hit = _decide(kind, rows, eta)
    assert (out > 0).any()
    assert not hit[out == 1].any()


def test_which_sextics_wait():
    ops = np.array([
        [1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 7.0],      # an ordinary one
        [1.0, 2.0, 3.0, 4.0, 5.0, 1e-9, 1e-9],    # roots near t = 0
        [1.0, 2.0, 3.0, 4.0, 5.0, 0.0, 0.0],      # and exactly there
        [1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0],      # nothing but the leading term
        [0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0],
    ])
    out = np.zeros(len(ops), np.uint8)
    _lib().hc_waits(ctypes.c_int64(len(ops)), ops.ctypes.data_as(P), out.ctypes.data_as(P))
    assert out.tolist() == [0, 1, 3, 1, 1]


@pytest.mark.parametrize("at", range(7))
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_sextics_that_are_not_finite_do_not_wait(at, bad):
    # the solver reports them in the row's status
    op = np.array([[1.0, 2.0, 3.0, 4.0, 5.0, 0.0, 0.0]])
    op[0, at] = bad
    out = np.zeros(1, np.uint8)
    _lib().hc_waits(ctypes.c_int64(1), op.ctypes.data_as(P), out.ctypes.data_as(P))
    assert out[0] == 0
