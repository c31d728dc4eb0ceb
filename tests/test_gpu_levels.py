"""Level products of the aggregation cycle where the lanes of a row change: a
plane level 1 large enough for 8 lanes a block row (about 9 blocks each), a
batch whose FP64 product takes 4 or 8 lanes a row.

The matrix is `banded` (condition below 4), whose start of the recurrence and
cycle are well inside FP32; a recurrence residual of 1e-10 bounds the error by
4e-10, and 1e-9 is asserted.
"""
import ctypes as C

import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import decks, mefel
from ssf_b200.gefel import DeviceMatrix
from test_gpu_batch_forms import stack
from test_gpu_resident import banded, product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offsets", [(1, 2, 3), tuple(range(1, 10)), tuple(range(1, 11)), tuple(range(1, 14))])
def test_batch_rows(gpu_lib, offsets):  # 7, 19, 21 and 27 entries a row
    rows = [3001, 17, 2048, 4097]
    rp, col, val = stack([banded(n, [o for o in offsets if o < n], n) for n in rows])
    x = np.random.default_rng(3).standard_normal(sum(rows))
    f, got = product(rp, col, val, x), np.empty(sum(rows))
    n = len(rows)
    ani, ares = np.full(n, -1, dtype=np.int64), np.zeros(n)
    st, its = np.zeros(n, dtype=np.int32), np.zeros(n, dtype=np.int64)
    with DeviceMatrix(rp, col, val, 0) as K:
        rc = L.lib().sgpu_matrix_pcg_batch_agg(K.h, n, np.array(rows, dtype=np.int64), got, f, 500, 1e-20, 1e-30, L.MIXED,
                                               ani.ctypes.data, ares.ctypes.data, st.ctypes.data, its.ctypes.data,
                                               None)
    assert rc == L.OK and not st.any()
    assert np.linalg.norm(got - x) <= 1e-9 * np.linalg.norm(x)


def test_large_plane_level(gpu_lib):
    # 1.5M equations: level 1 is beyond a program's 20 MB, its rows have 9 blocks.  A wrong product there is a wrong
    # preconditioner: the count (41 on 2.7M equations of plates) would multiply.
    m = decks.plate_quad(1100, 700, E=3e10, nu=0.22)
    with mefel.stiffness_matrix(m) as K:
        K.set_nullspace(mefel.rigid_body_modes(m))
        f = np.random.default_rng(5).standard_normal(K.n)
        x, r = K.pcg(f, res=1e-10, crit="true", prec="agg", mode="mixed")
        assert r.status == L.OK and r.info["iterations"] <= 100
        assert np.linalg.norm(f - K.mxv(x)) <= 1.01e-10 * np.linalg.norm(f)
