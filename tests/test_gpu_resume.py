"""Solves that one launch does not finish: more iterations than a launch of the grid does, and a recurrence that goes on
after the true residual disagreed.  Beside them the general form (the product pinned), three launches an iteration.

K = tridiag(-1, 2 + e, -1) has its eigenvalues in [e, 4 + e]; CG needs about sqrt(4 / e) ln(2 / 1e-10) / 2 iterations
for 1e-10.
"""
import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import gefel

pytestmark = pytest.mark.gpu


def chain(n, e):
    rowptr = np.concatenate([[0], np.cumsum(np.full(n, 3))])
    rowptr[1:] -= 1
    rowptr[-1] -= 1
    i = np.repeat(np.arange(n), 3) + np.tile([-1, 0, 1], n)
    keep = (i >= 0) & (i < n)
    return rowptr, i[keep], np.tile([-1.0, 2.0 + e, -1.0], n)[keep]


def both(n, e, **kw):
    """(solution, report, launches) of the grid, (solution, report) of the general form"""
    rowptr, col, val = chain(n, e)
    f = np.random.default_rng(1).standard_normal(n)
    with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
        K.pcg(f, ni=1)  # whatever is allocated once
        before = L.lib().sgpu_kernel_launches()
        grid = K.pcg(f, **kw) + (L.lib().sgpu_kernel_launches() - before,)
        K.set_spmv(64, 0, 4)
        general = K.pcg(f, **kw)
    return f, grid, general


@pytest.mark.parametrize("n", [30001, 200003])  # resident; in tiles
def test_more_iterations_than_one_launch(gpu_lib, n):
    f, (x, r, _), (_, general) = both(n, 1.6e-5, res=1e-20)
    assert r.status == general.status == L.OK and r.ani > 4096
    assert r.info["spmv_variant"] in (0, 2)
    assert abs(r.ani - general.ani) <= 0.02 * general.ani
    # the recurrence met 1e-10; the true residual adds the iteration's rounding, a few times eps ||K|| ||x|| / ||f||
    assert r.info["true_relres"] <= 1e-10 + 64 * 2.3e-16 * 4.0 * np.linalg.norm(x) / np.linalg.norm(f)


@pytest.mark.parametrize("n", [30001, 200003])
def test_going_on_after_the_true_residual_disagreed(gpu_lib, n):
    """A threshold close to the floor of f - K x itself (eps ||K|| ||x|| / ||f||, here about 1e-12): the recurrence meets
    it before the iterate does, is corrected and goes on."""
    f, (x, r, launches), (y, general) = both(n, 1e-4, res=1e-12, crit="true", ni=40000)
    assert r.status in (L.OK, L.NOT_CONVERGED) and general.status in (L.OK, L.NOT_CONVERGED)
    assert launches >= 10  # one confirmation takes six launches, each further one four
    floor = 64 * 2.3e-16 * 4.0 * np.linalg.norm(x) / np.linalg.norm(f)
    for q in (r, general):
        assert q.info["true_relres"] <= max(1e-12, floor)
        assert (q.status == L.OK) == (q.info["true_relres"] < 1e-12)
    # two residuals of that size, and the smallest eigenvalue
    assert np.linalg.norm(x - y) <= 2 * max(1e-12, floor) / 1e-4 * np.linalg.norm(f)
