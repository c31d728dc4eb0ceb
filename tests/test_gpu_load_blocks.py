"""Load cases with the aggregation cycle where the block kernels change: one
and several columns a lane, rows of more than 32 blocks (taken in pieces), a
last piece of one block, levels of few and of many block rows, the largest
number of columns.

Matrices are a `banded` one (condition below 4) times a 3 x 3 block of
condition 2, so a recurrence residual of 1e-10 bounds the error by 8e-10; 1e-9
is asserted.
"""
import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200.gefel import DeviceMatrix, pcg_multi_blocks
from test_gpu_resident import banded, product

pytestmark = pytest.mark.gpu

BLOCK = np.array([[1.5, 0.5, 0.0], [0.5, 1.5, 0.0], [0.0, 0.0, 2.0]])  # eigenvalues 1, 2, 2


def in_blocks(rowptr, col, val):
    nb = len(rowptr) - 1
    rp, cs, vs = [0], [], []
    for i in range(nb):
        k = slice(rowptr[i], rowptr[i + 1])
        for q in range(3):
            cs.append((3 * np.asarray(col[k])[:, None] + np.arange(3)).ravel())
            vs.append((np.asarray(val[k])[:, None] * BLOCK[q]).ravel())
            rp.append(rp[-1] + cs[-1].size)
    return np.array(rp, dtype=np.int64), np.concatenate(cs).astype(np.int64), np.concatenate(vs)


MATRICES = {
    "few_rows": (40, (1, 2)),
    "pieces": (700, tuple(range(1, 41))),    # 81 blocks a row
    "one_over": (900, tuple(range(1, 17))),  # 33 blocks a row
    "many_rows": (20011, (1, 30, 900)),
}


@pytest.mark.parametrize("nrhs", [1, 32, 33, 64, 100, 128])
@pytest.mark.parametrize("mode", ["mixed", "fp64"])
@pytest.mark.parametrize("name", MATRICES)
def test_columns(gpu_lib, name, mode, nrhs):
    n, offsets = MATRICES[name]
    rp, col, val = in_blocks(*banded(n, offsets, n, False))
    X = np.random.default_rng(nrhs).standard_normal((nrhs, 3 * n))
    F = np.stack([product(rp, col, val, x) for x in X])
    with DeviceMatrix(rp, col, val, 0) as K:
        got, out = pcg_multi_blocks(K, F, res=1e-20, prec="agg", mode=mode)
    assert all(r.status == L.OK for r in out)
    assert np.max(np.linalg.norm(got - X, axis=1) / np.linalg.norm(X, axis=1)) <= 1e-9
