"""Solves where the process has only a share of the device's SMs.

SGPU_SMS states the share.  More than the device has makes the runtime refuse
the grids of a CTA per SM, which is what a solve meets when it is given fewer
SMs than the device reports; the general forms then take over.  Systems have
condition below 6.3, so a residual of 1e-10 bounds the relative error by 2e-9
(1e-9 below 4).
"""
import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import decks, gefel, mefel
from test_gpu_batch_forms import solve as solve_batch
from test_gpu_batch_forms import stack
from test_gpu_resident import SYSTEMS, banded, product
from test_gpu_resident import solve as solve_noalloc

pytestmark = pytest.mark.gpu

SHARES = ["0", "3", "20", "100", "250"]


@pytest.mark.parametrize("sms", SHARES)
@pytest.mark.parametrize("name", ["resident", "csr_2", "bsr_8"])
@pytest.mark.parametrize("start", [False, True])
def test_solves_on_a_handle(gpu_lib, monkeypatch, sms, name, start):
    monkeypatch.setenv("SGPU_SMS", sms)
    rowptr, col, val = SYSTEMS[name][0]()
    n = len(rowptr) - 1
    x = np.random.default_rng(2).standard_normal(n)
    f = product(np.asarray(rowptr), col, val, x)
    with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
        got, r = K.pcg(f, x=np.full(n, 0.5) if start else None, res=1e-10, crit="true")
        assert r.status == L.OK and r.info["iterations"] == r.ani + 1
        assert np.linalg.norm(got - x) <= 2e-9 * np.linalg.norm(x)
        if sms in ("0", "250"):  # a product's kernel, not the grids (resident: 0, two lanes: 2)
            assert r.info["spmv_variant"] >= 4
        _, r = K.pcg(f, ni=3, res=1e-20)
        assert r.status == L.NOT_CONVERGED and r.info["iterations"] == 3
        y, r = K.pcg(np.zeros(n), res=1e-20)
        assert r.status == L.ZERO_RHS and not y.any()


@pytest.mark.parametrize("sms", SHARES)
@pytest.mark.parametrize("n", [1, 3000, L.NOALLOC_MAX_N])
def test_the_solver_without_allocation(gpu_lib, monkeypatch, sms, n):
    monkeypatch.setenv("SGPU_SMS", sms)
    rowptr, col, val = banded(n, [o for o in (1, 7, 300) if o < n], n)
    x = np.random.default_rng(n + 1).standard_normal(n)
    f = product(rowptr, col, val, x)
    for iv, x0 in ((0, np.full(n, 7.0)), (1, x + 1e-3)):
        st, got, ani, its = solve_noalloc(rowptr, col, val, f, x0, iv=iv)
        assert st == L.OK and its == ani + 1
        assert np.linalg.norm(got - x) <= 1e-9 * np.linalg.norm(x)
    st, _, ani, its = solve_noalloc(rowptr, col, val, np.zeros(n), np.zeros(n))
    assert st == L.ZERO_RHS and ani == 0
    bad = col.copy()
    bad[0] = n
    x0 = np.full(n, 3.0)
    st, got, ani, _ = solve_noalloc(rowptr, bad, val, f, x0)
    assert st == L.BAD_INPUT and ani == -1 and np.array_equal(got, x0)


@pytest.mark.parametrize("sms", ["0", "4", "250"])
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_aggregation(gpu_lib, monkeypatch, sms, mode):
    """The coarse levels' kernels instead of their program: the same sums in the same order."""
    mesh = decks.cantilever_hex(30, 9, 8)
    f = np.random.default_rng(1).standard_normal(mesh.ndof)
    with mefel.stiffness_matrix(mesh) as K:
        K.set_rigid_body_modes(mesh.coords, mesh.code_numbers())
        want, r0 = K.pcg(f, prec="agg", mode=mode, crit="true", res=1e-10)
        monkeypatch.setenv("SGPU_SMS", sms)
        got, r = K.pcg(f, prec="agg", mode=mode, crit="true", res=1e-10)
        assert r0.status == r.status == L.OK and r.info["iterations"] == r0.info["iterations"]
        # a program of four CTAs sums the same rows in the same order, too
        assert np.array_equal(got, want)


@pytest.mark.parametrize("sms", ["0", "7", "250"])
def test_batches(gpu_lib, monkeypatch, sms):
    monkeypatch.setenv("SGPU_SMS", sms)
    rows = [9001, 1, 2049, 40, 700]
    parts = [banded(n, [o for o in (1, 50) if o < n], n) for n in rows]
    rp, col, val = stack(parts)
    x = np.random.default_rng(3).standard_normal(sum(rows))
    f = product(rp, col, val, x)
    with gefel.DeviceMatrix(rp, col, val, 0) as K:
        rc, got, _, st, _ = solve_batch(K, rows, f)
    at = np.cumsum([0] + rows)
    assert rc == L.OK and not st.any()
    for a, b in zip(at, at[1:]):
        assert np.linalg.norm(got[a:b] - x[a:b]) <= 1e-9 * np.linalg.norm(x[a:b])
