"""The classification of rows (csrc/ccd_classify.h) against the full decision
where it is most exposed: contacts in the first cells of the step, whose mirror
images are not looked at, and rows whose coefficients are not finite."""
import numpy as np
import pytest

from test_classify_host import N, _classify, _family


def _mirrored_early(rng):
    """Double roots of the sextic at t and near -t, the whole motion then made up to 1000 times as fast, which
    brings them to t from 5e-5 of the step on."""
    s, e = _family("mirrored", rng)
    return s, s + (e - s) * 10.0 ** rng.uniform(0.0, 3.0, (N, 1, 1))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("seed", range(4))
def test_contacts_in_the_first_cells(seed, kind):
    rng = np.random.default_rng([29, kind, seed])
    s, e = _mirrored_early(rng)
    rows = np.concatenate([s.reshape(N, 12), e.reshape(N, 12)], 1)
    eta = np.where(rng.random(N) < 0.5, 1e-6, 10.0 ** rng.uniform(-8, -2, N))
    out, differs, _, _ = _classify(kind, rows, eta)
    assert ((out == 1) | (out == 2)).any()
    assert differs.sum() == 0


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e160, -1e200])
def test_rows_that_are_not_finite_are_left_to_the_solver(bad, kind):
    rng = np.random.default_rng(3)
    n = 2000
    rows = rng.random((n, 24))
    rows[:, 12:] = rows[:, :12] + 0.1 * rng.normal(size=(n, 12))
    rows[np.arange(n), rng.integers(0, 24, n)] = bad
    out, differs, _, _ = _classify(kind, rows, 1e-6)
    assert set(np.unique(out)) <= {0, 4}
    assert differs.sum() == 0
