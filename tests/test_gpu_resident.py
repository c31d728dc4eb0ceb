"""The resident Jacobi-PCG grid at the sizes where its layout changes.

Rows are spread over 32, 16, ... 1 lanes as the system grows (148 CTAs of
1024 threads: the split changes at multiples of 148 x 32 rows), and warps
whose entries do not fit the SM's memory read them from the caller's arrays.
The matrices are diagonally dominant with condition below 4, so a residual of
1e-10 bounds the relative solution error by 4e-10; 1e-9 is asserted.
"""
import ctypes as C

import numpy as np
import pytest

from ssf_b200 import _lib as L

pytestmark = pytest.mark.gpu


def banded(n, offsets, seed, uneven=False):
    """CSR of a symmetric matrix with entries in (-1, 0) / (2 * len(offsets)) at the given offsets and a diagonal of
    2: eigenvalues in [1, 3].  uneven: the offsets beyond the first only in every third row and column."""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.full(n, 2.0)]
    for q, o in enumerate(offsets):
        i = np.arange(n - o)
        if uneven and q:
            i = i[(i % 3 == 0)]
        v = -rng.random(i.size) / (2.0 * len(offsets))
        rows += [i, i + o]
        cols += [i + o, i]
        vals += [v, v]
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order], v[order]
    rowptr = np.zeros(n + 1, dtype=np.int32)
    rowptr[1:] = np.cumsum(np.bincount(r, minlength=n))
    return rowptr, c.astype(np.int32), v


def product(rowptr, col, val, x):
    return np.add.reduceat(val * x[col], rowptr[:-1])


def solve(rowptr, col, val, f, x, ni=20000, iv=0):
    import torch
    d = [torch.from_numpy(v).cuda() for v in (rowptr, col, val, f, x)]
    ani, ares, its = C.c_int64(-1), C.c_double(-1.0), C.c_int64(0)
    st = L.lib().sgpu_csr_pcg_noalloc_d(f.size, *[v.data_ptr() for v in d], ni, 1e-20, 1e-30, iv, None, C.byref(ani),
                                        C.byref(ares), C.byref(its))
    return st, d[4].cpu().numpy(), ani.value, its.value


@pytest.mark.parametrize("n", [1, 2, 31, 33, 148, 149, 4736, 4737, 9473, 18945, 37889, 75776, 75777, L.NOALLOC_MAX_N])
@pytest.mark.parametrize("uneven", [False, True])
def test_row_splits(gpu_lib, n, uneven):
    offsets = [o for o in (1, 7, 300) if o < n]
    rowptr, col, val = banded(n, offsets, n, uneven)
    x = np.random.default_rng(n + 1).standard_normal(n)
    f = product(rowptr, col, val, x)
    st, got, ani, its = solve(rowptr, col, val, f, np.full(n, 7.0))
    assert st == L.OK and its == ani + 1
    assert np.linalg.norm(got - x) <= 1e-9 * np.linalg.norm(x)


@pytest.mark.parametrize("n,width", [(L.NOALLOC_MAX_N, 24), (60000, 60), (20000, 90)])
def test_rows_beyond_shared_memory(gpu_lib, n, width):
    rowptr, col, val = banded(n, list(range(1, width + 1)), n)
    x = np.random.default_rng(5).standard_normal(n)
    f = product(rowptr, col, val, x)
    x0 = np.random.default_rng(6).standard_normal(n)
    for iv, start in ((0, np.zeros(n)), (1, x0)):
        st, got, _, _ = solve(rowptr, col, val, f, start, iv=iv)
        assert st == L.OK
        # the start residual of x0 is below 10 |f|: the same bound times 10
        assert np.linalg.norm(got - x) <= 1e-9 * np.linalg.norm(x)


def test_more_iterations_than_one_launch(gpu_lib, oracle):
    """A 1D Laplacian takes about as many iterations as it has equations: more than the 2048 of one launch."""
    n = 2600
    rowptr, col, val = banded(n, [1], 0)
    val = np.where(val == 2.0, 2.0, -1.0)
    f = np.random.default_rng(1).standard_normal(n)
    st, x, ani, its = solve(rowptr, col, val, f, np.zeros(n))
    assert st == L.OK and its > 2048
    # the recurrence residual met 1e-10; the true one adds the iteration's rounding, a few times
    # eps ||K|| ||x|| / ||f||
    r = f - product(rowptr, col, val, x)
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(f) + 64 * 2.3e-16 * 4.0 * np.linalg.norm(x)


def test_iteration_limit_and_zero_right_hand_side(gpu_lib):
    rowptr, col, val = banded(500, [1], 3)
    st, _, ani, its = solve(rowptr, col, val, np.ones(500), np.zeros(500), ni=2)
    assert st == L.NOT_CONVERGED and ani == -1 and its == 2
    st, x, ani, _ = solve(rowptr, col, val, np.zeros(500), np.zeros(500))
    assert st == L.ZERO_RHS and ani == 0 and not x.any()


# ---------------------------------------------------------------------------
# the same iteration on a handle: resident, streamed in tiles, or the general
# graph of kernels (rows too long for the tiles' stages, or a pinned product)
# ---------------------------------------------------------------------------
def blocked(nb, offsets, seed):
    """3x3 block rows: the scalar band of `banded` times [[2, .5, 0], [.5, 2, .5], [0, .5, 2]] (eigenvalues in
    [1.29, 2.71]), entry for entry; condition below 6.3."""
    rowptr, col, val = banded(nb, offsets, seed)
    B = np.array([[2.0, 0.5, 0.0], [0.5, 2.0, 0.5], [0.0, 0.5, 2.0]])
    lens = np.diff(rowptr)
    rp = np.concatenate([[0], np.cumsum(np.repeat(3 * lens, 3))])
    row_of = np.repeat(np.arange(nb), lens)
    out_c = np.empty(rp[-1], dtype=np.int64)
    out_v = np.empty(rp[-1])
    within = np.arange(col.size) - rowptr[row_of]
    for i in range(3):
        for j in range(3):
            pos = rp[3 * row_of + i] + 3 * within + j
            out_c[pos] = 3 * col + j
            out_v[pos] = val * B[i, j]
    return rp, out_c, out_v


def arrow(n, spokes, seed):
    """A diagonal of 2 and couplings of row 0 with `spokes` others, weak enough for eigenvalues in [1, 3]."""
    c = -1.0 / np.sqrt(spokes) * np.random.default_rng(seed).random(spokes)
    k = np.arange(1, spokes + 1)
    r = np.concatenate([np.arange(n), np.zeros(spokes, dtype=np.int64), k])
    q = np.concatenate([np.arange(n), k, np.zeros(spokes, dtype=np.int64)])
    v = np.concatenate([np.full(n, 2.0), c, c])
    order = np.lexsort((q, r))
    r, q, v = r[order], q[order], v[order]
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]), q, v


SYSTEMS = {
    # name: (matrix, expected (format, lanes) of the iteration; lanes None: the general form)
    "resident": (lambda: banded(3001, [1, 50], 1), (0, 0)),
    "resident_one": (lambda: banded(1, [], 1), (0, 0)),
    "csr_2": (lambda: banded(200003, [1, 7, 300], 2), (0, 2)),
    "csr_2_uneven": (lambda: banded(160001, [1, 7, 300, 9000], 2, True), (0, 2)),
    "csr_8": (lambda: banded(40000, range(1, 41), 3), (0, 8)),
    "csr_32": (lambda: banded(15001, range(1, 101), 4), (0, 8)),  # 201 entries a row: 8 lanes take up to 265
    "csr_32_long": (lambda: banded(15001, range(1, 151), 4), (0, 32)),
    "csr_2_long": (lambda: banded(90001, range(1, 33), 5), (0, 2)),  # 65 entries, one below the line
    "general": (lambda: arrow(200003, 5000, 5), (0, None)),
    "bsr_8": (lambda: blocked(60001, [1, 7, 300], 6), (3, 8)),
    "bsr_16": (lambda: blocked(6001, range(1, 26), 7), (3, 16)),
    "bsr_32": (lambda: blocked(3501, range(1, 46), 8), (3, 32)),
}


@pytest.mark.parametrize("name", SYSTEMS)
@pytest.mark.parametrize("crit,prec", [("scr", 1), ("cr", 0), ("true", 1)])
def test_forms_on_a_handle(gpu_lib, name, crit, prec):
    from ssf_b200 import gefel
    make, (fmt, lanes) = SYSTEMS[name]
    rowptr, col, val = make()
    n = len(rowptr) - 1
    x = np.random.default_rng(11).standard_normal(n)
    f = product(np.asarray(rowptr), col, val, x)
    res = 1e-20 if crit == "scr" else 1e-10
    with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
        got, r = K.pcg(f, res=res, crit=crit, prec=prec)
        start, r2 = K.pcg(f, x=np.full(n, 0.5), res=res, crit=crit, prec=prec)
        # the general form: the product pinned to CSR with 8 lanes a row
        K.set_spmv(64, 0, 8)
        other, r3 = K.pcg(f, res=res, crit=crit, prec=prec)
    assert r.status == r2.status == r3.status == L.OK
    assert r.info["spmv_format"] == fmt and (lanes is None or r.info["spmv_variant"] == lanes)
    # other orders of summation: rounding moves the count by one at most here (10 to 40 iterations)
    assert abs(r.ani - r3.ani) <= 1
    # residual 1e-10 of f (of at most 2 |f| more for the start vector) and condition below 6.3
    for y in (got, start, other):
        assert np.linalg.norm(y - x) <= 2e-9 * np.linalg.norm(x)
    assert r.info["true_relres"] <= 1.1e-10


@pytest.mark.parametrize("name", ["resident", "csr_2", "bsr_8"])
def test_forms_stop_at_the_limit(gpu_lib, name):
    from ssf_b200 import gefel
    rowptr, col, val = SYSTEMS[name][0]()
    n = len(rowptr) - 1
    with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
        _, r = K.pcg(np.ones(n), ni=3, res=1e-20)
        assert r.status == L.NOT_CONVERGED and r.ani is None and r.info["iterations"] == 3
        x, r = K.pcg(np.zeros(n), res=1e-20)
        assert r.status == L.ZERO_RHS and r.ani == 0 and not x.any()
        _, r = K.pcg(np.ones(n), res=1e-20, zero=1e300)
        assert r.status == L.ZERO_RHS or r.status == L.BREAKDOWN
