"""Which form iterates where rows are short or uneven: on both sides of each line of the rule.

A grid needs one launch for thousands of iterations, the general form three
launches for each.  The systems are diagonally dominant with eigenvalues in
[1, 3]: a residual of 1e-10 bounds the error by 3e-10; 1e-9 is asserted.
"""
import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import gefel
from test_gpu_resident import banded, blocked, product

pytestmark = pytest.mark.gpu


def one_long(n, offsets, spokes, seed):
    """A band, and entries of its last row and column with the `spokes` rows in front of those it has already; the
    off-diagonal part halved, so that both together keep the eigenvalues in [1, 3]."""
    rowptr, col, val = banded(n, offsets, seed)
    rows = np.repeat(np.arange(n), np.diff(rowptr))
    val = np.where(rows == col, val, 0.5 * val)
    k = np.arange(n - 1 - max(offsets) - spokes, n - 1 - max(offsets))
    v = np.full(spokes, -0.5 / np.sqrt(spokes))
    last = np.full(spokes, n - 1)
    r, c, v = np.concatenate([rows, k, last]), np.concatenate([col, last, k]), np.concatenate([val, v, v])
    order = np.lexsort((c, r))
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), c[order], v[order]


SYSTEMS = {
    # name: (matrix, one grid)
    "short_few": (lambda: banded(500003, [1], 1), True),  # 9 n - nnz = 3.0M of 3.5M
    "short_many": (lambda: banded(700001, [1], 1), False),  # 4.2M
    "short_many_of_seven": (lambda: banded(1000003, [1, 2, 50], 1), True),  # 2.0M
    "one_stage_many": (lambda: one_long(2000003, [1, 2, 3, 5], 50, 8), False),  # 24 n - nnz = 30M of 25M
    "one_stage_fewer": (lambda: one_long(1000003, [1, 2, 3, 5], 50, 8), True),  # 15M
    "resident_lane_of_160": (lambda: one_long(140001, [1, 2], 160 - 3, 2), True),
    "resident_lane_of_161": (lambda: one_long(140001, [1, 2], 161 - 3, 2), False),  # 8 lanes: 7.0M of 5M
    "resident_32_lanes_of_160": (lambda: one_long(9001, [1], 32 * 64 - 2, 3), True),  # 16 lanes, 2048 entries
    "eight_lanes_few": (lambda: one_long(120001, range(1, 9), 100, 4), True),  # 4.6M of 5M
    "eight_lanes_many": (lambda: one_long(160001, range(1, 9), 100, 4), False),  # 6.1M
    "thirty_two_lanes_few": (lambda: one_long(25001, range(1, 26), 300, 5), True),  # resident
    "thirty_two_lanes_many": (lambda: one_long(160001, range(1, 31), 300, 5), False),
    "blocks_few": (lambda: blocked(150001, [1, 2, 50], 6), True),  # 0.45M of 1M
    "blocks_many_short": (lambda: blocked(350003, [1], 6), False),  # 2.5M
    "blocks_uneven": (lambda: blocked_long(150001, [1, 2, 50], 50, 7), False),  # 16 lanes: 1.7M of 0.7M
    "blocks_uneven_few": (lambda: blocked_long(40001, [1, 2, 50], 50, 7), True),  # 0.44M
}


def blocked_long(nb, offsets, spokes, seed):
    """`blocked` of a scalar pattern with one long row (eigenvalues in [1, 3] times [1.29, 2.71])."""
    import test_gpu_resident as R
    kept = R.banded
    try:
        R.banded = lambda n, o, s: one_long(n, o, spokes, s)
        return blocked(nb, offsets, seed)
    finally:
        R.banded = kept


@pytest.mark.parametrize("name", SYSTEMS)
def test_form_and_solution(gpu_lib, name):
    make, grid = SYSTEMS[name]
    rowptr, col, val = make()
    n = len(rowptr) - 1
    x = np.random.default_rng(11).standard_normal(n)
    f = product(np.asarray(rowptr), col, val, x)
    with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
        K.pcg(f, ni=1)  # whatever is tuned or allocated once
        before = gpu_lib.sgpu_kernel_launches()
        got, r = K.pcg(f, res=1e-20)
        launches = gpu_lib.sgpu_kernel_launches() - before
    assert r.status == L.OK and r.info["iterations"] > 8
    assert (launches < 8) == grid, (launches, r.info)
    assert np.linalg.norm(got - x) <= (1e-9 if not name.startswith("blocks") else 2e-9) * np.linalg.norm(x)
