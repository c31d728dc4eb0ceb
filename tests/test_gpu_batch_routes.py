"""Which form an uneven batch takes: clusters (two launches: the gathers' places, then the solve) or a CTA per system
(one launch), on both sides of each line; and what a system reports at the iteration limit.

Systems have condition below 4 (`banded`): a residual of 1e-10 bounds the error by 4e-10; 1e-9 is asserted.
"""
import ctypes as C

import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200.gefel import DeviceMatrix
from test_gpu_batch_forms import solve, stack
from test_gpu_resident import banded, product

pytestmark = pytest.mark.gpu


def batch(rows, offsets):
    """Every system of a size is the same one, so that thousands of them are quickly made."""
    made = {n: banded(n, [o for o in offsets if o < n], n) for n in set(rows)}
    return stack([made[n] for n in rows])


BATCHES = {
    # name: (rows, offsets, clusters)
    "many_small": ([60] * 1500, (1, 2, 3, 5), False),
    "many_of_1000": ([1000] * 500, (1, 2, 3, 5), False),
    "few_of_2048": ([2048] * 40, range(1, 9), True),
    "two_per_sm": ([2048] * 256, range(1, 9), True),
    "one_large_among_small": ([12000] + [100] * 100, (1, 2, 3, 5), True),
    "largest_of_a_cluster": ([32768, 500], range(1, 9), True),
    "beyond_a_cluster": ([32769, 500], range(1, 9), False),
}


@pytest.mark.parametrize("name", BATCHES)
def test_form_and_solutions(gpu_lib, name):
    rows, offsets, clusters = BATCHES[name]
    rp, col, val = batch(rows, offsets)
    x = np.random.default_rng(3).standard_normal(sum(rows))
    f = product(rp, col, val, x)
    with DeviceMatrix(rp, col, val, 0) as K:
        solve(K, rows, f, ni=1)
        before = gpu_lib.sgpu_kernel_launches()
        rc, got, ani, st, its = solve(K, rows, f)
        assert gpu_lib.sgpu_kernel_launches() - before == (2 if clusters else 1)
    assert rc == L.OK and not st.any() and np.array_equal(its, ani + 1)
    at = np.concatenate([[0], np.cumsum(rows)])
    for a, b in zip(at, at[1:]):
        assert np.linalg.norm(got[a:b] - x[a:b]) <= 1e-9 * np.linalg.norm(x[a:b])


@pytest.mark.parametrize("rows", [[9001, 1, 2049, 40, 700], [60] * 300 + [2]])
def test_iteration_limit(gpu_lib, rows):
    rp, col, val = batch(rows, (1, 7, 50))
    f = product(rp, col, val, np.random.default_rng(3).standard_normal(sum(rows)))
    with DeviceMatrix(rp, col, val, 0) as K:
        rc, _, ani, st, its = solve(K, rows, f, ni=2)
    assert rc == L.NOT_CONVERGED
    for k, n in enumerate(rows):
        if n <= 2:  # as many iterations as equations are enough
            assert st[k] == L.OK and its[k] == ani[k] + 1 <= 2
        else:
            assert st[k] == L.NOT_CONVERGED and its[k] == 2 and ani[k] == -1


@pytest.mark.parametrize("name", ["many_small", "few_of_2048", "beyond_a_cluster"])
def test_report_names_the_lanes_that_ran(gpu_lib, name):
    rows, offsets, clusters = BATCHES[name]
    rp, col, val = batch(rows, offsets)
    f, info = np.ones(sum(rows)), L.SolveInfo()
    mean = val.size / f.size
    with DeviceMatrix(rp, col, val, 0) as K:
        rc = gpu_lib.sgpu_matrix_pcg_batch(K.h, len(rows), np.array(rows, dtype=np.int64), np.empty_like(f), f, 2, 1e-20,
                                           1e-30, 0, None, None, None, None, C.byref(info))
    assert rc == L.NOT_CONVERGED and info.spmv_format == 0
    assert info.spmv_variant == (2 if clusters else 8 if mean > 12 else 4)
