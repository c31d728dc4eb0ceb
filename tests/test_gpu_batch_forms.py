"""The uneven batch where its layout changes: systems that one CTA or a whole
cluster takes (2048 rows), of one row, at the largest a cluster holds, rows of
one and of several chunks of a lane, neighbours several ranges away; systems
too large, and a matrix that couples its systems, take the other form.

Systems have condition below 4 (`banded` of the resident tests), so a
recurrence residual of 1e-10 bounds the error by 4e-10; 1e-9 is asserted.
"""
import ctypes as C

import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200.gefel import DeviceMatrix
from test_gpu_resident import banded, product

pytestmark = pytest.mark.gpu


def stack(parts):
    rp, cols, vals, base, nnz = [np.zeros(1, dtype=np.int64)], [], [], 0, 0
    for rowptr, col, val in parts:
        rp.append(rowptr[1:].astype(np.int64) + nnz)
        cols.append(col.astype(np.int64) + base)
        vals.append(val)
        base += len(rowptr) - 1
        nnz += len(col)
    return np.concatenate(rp), np.concatenate(cols), np.concatenate(vals)


def solve(K, rows, f, ni=2000, res=1e-20):
    n = len(rows)
    x, ani, ares = np.empty(f.size), np.full(n, -1, dtype=np.int64), np.zeros(n)
    st, its = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int64)
    rc = L.lib().sgpu_matrix_pcg_batch(K.h, n, np.array(rows, dtype=np.int64), x, f, ni, res, 1e-30, 0, ani.ctypes.data,
                                       ares.ctypes.data, st.ctypes.data, its.ctypes.data, None)
    return rc, x, ani, st, its


BATCHES = {
    "small": ([1, 2, 15, 16, 17, 33, 511, 513, 2047, 2048], (1, 3)),
    "at_the_line": ([2048, 2049, 2050, 4095, 4096, 4097], (1, 7, 300)),
    "mixed": ([9001, 1, 2049, 40, 16384, 700, 3000], (1, 50)),
    "largest": ([31000, 17, 30999], (1, 60)),
    "far_neighbours": ([8001, 2100], (1, 1500)),
    "long_rows": ([2500, 900, 64], tuple(range(1, 30))),
    "too_large": ([60000, 100], (1, 50)),
}


@pytest.mark.parametrize("name", BATCHES)
@pytest.mark.parametrize("uneven", [False, True])
def test_uneven_systems(gpu_lib, name, uneven):
    rows, offsets = BATCHES[name]
    parts = [banded(n, [o for o in offsets if o < n], n + k, uneven) for k, n in enumerate(rows)]
    x = np.random.default_rng(3).standard_normal(sum(rows))
    rp, col, val = stack(parts)
    f = product(rp, col, val, x)
    with DeviceMatrix(rp, col, val, 0) as K:
        rc, got, ani, st, its = solve(K, rows, f)
        again = solve(K, rows, f)
        assert rc == L.OK and not st.any() and np.array_equal(its, ani + 1)
        assert np.array_equal(again[1], got) and np.array_equal(again[4], its)
        at = np.cumsum([0] + rows)
        for k in range(len(rows)):
            a, b = at[k], at[k + 1]
            assert np.linalg.norm(got[a:b] - x[a:b]) <= 1e-9 * np.linalg.norm(x[a:b])
        # limits and a zero right-hand side, per system
        rc, _, ani, st, its = solve(K, rows, f, ni=2)
        assert all(s == (L.OK if n <= 2 else L.NOT_CONVERGED) or its[k] <= 2 for k, (s, n) in enumerate(zip(st, rows)))
        f[at[0]:at[1]] = 0.0
        rc, got, ani, st, its = solve(K, rows, f)
        assert rc == st[0] == L.ZERO_RHS and ani[0] == 0 and not got[:at[1]].any() and not st[1:].any()


def test_coupled_systems_keep_the_other_form(gpu_lib):
    """sys_rows that cut through one banded matrix: every sum of the iteration is per system, the product is not --
    what the call always did with such input, unchanged."""
    rp, col, val = banded(6000, [1, 7], 5)
    f = np.random.default_rng(1).standard_normal(6000)
    with DeviceMatrix(rp, col, val, 0) as K:
        rc, x, _, st, its = solve(K, [3000, 3000], f, ni=3)
        assert rc in (L.OK, L.NOT_CONVERGED) and np.isfinite(x).all() and (its <= 3).all()
