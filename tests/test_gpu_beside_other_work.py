"""Solves while other work holds SMs, and several solves at once.

A kernel that ends by itself keeps the shared memory of some SMs, once for
longer than the waits inside a grid last.  A grid of a CTA per SM starts when
it can be complete.  Systems have condition below 6.3: a residual of 1e-10
bounds the error by 2e-9.
"""
import ctypes as C
import os
import subprocess
import threading

import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import build, decks, gefel, mefel
from test_gpu_batch_forms import solve as solve_batch
from test_gpu_batch_forms import stack
from test_gpu_resident import SYSTEMS, banded, product
from test_gpu_resident import solve as solve_noalloc

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
BRIEF, LONG = 100_000_000, 4_500_000_000  # ns


@pytest.fixture(scope="module")
def other(gpu_lib, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hold") / "libhold.so")
    subprocess.run([build.NVCC, *build.ARCH, "-O2", "-shared", "-Xcompiler", "-fPIC", os.path.join(HERE, "hold_sms.cu"),
                    "-o", out], check=True)
    lib = C.CDLL(out)
    lib.hold_sms.argtypes = [C.c_int, C.c_longlong]
    yield lib


def held(other, ns, fn):
    assert other.hold_sms(20, ns) == 0
    try:
        return fn()
    finally:
        assert other.release() == 0


@pytest.mark.parametrize("name,ns", [("resident", LONG), ("csr_2", BRIEF), ("bsr_8", BRIEF)])
def test_solves_on_a_handle(other, ns, name):
    rowptr, col, val = SYSTEMS[name][0]()
    n = len(rowptr) - 1
    x = np.random.default_rng(2).standard_normal(n)
    f = product(np.asarray(rowptr), col, val, x)
    with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
        K.pcg(f)  # the handle's arrays are there
        got, r = held(other, ns, lambda: K.pcg(f))
    assert r.status == L.OK and r.info["iterations"] == r.ani + 1
    assert np.linalg.norm(got - x) <= 2e-9 * np.linalg.norm(x)


def test_the_solver_without_allocation(other):
    for n in (3000, L.NOALLOC_MAX_N):
        rowptr, col, val = banded(n, [1, 7, 300], n)
        x = np.random.default_rng(n + 1).standard_normal(n)
        f = product(rowptr, col, val, x)
        st, got, ani, its = held(other, BRIEF, lambda: solve_noalloc(rowptr, col, val, f, np.full(n, 7.0)))
        assert st == L.OK and its == ani + 1
        assert np.linalg.norm(got - x) <= 1e-9 * np.linalg.norm(x)


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_aggregation(other, mode):
    mesh = decks.cantilever_hex(30, 9, 8)
    f = np.random.default_rng(1).standard_normal(mesh.ndof)
    with mefel.stiffness_matrix(mesh) as K:
        K.set_rigid_body_modes(mesh.coords, mesh.code_numbers())
        want, r0 = K.pcg(f, prec="agg", mode=mode, crit="true", res=1e-10)
        got, r = held(other, BRIEF, lambda: K.pcg(f, prec="agg", mode=mode, crit="true", res=1e-10))
    assert r0.status == r.status == L.OK and np.array_equal(got, want)


def test_batches(other):
    rows = [9001, 1, 2049, 40, 700]
    parts = [banded(n, [o for o in (1, 50) if o < n], n) for n in rows]
    rp, col, val = stack(parts)
    x = np.random.default_rng(3).standard_normal(sum(rows))
    f = product(rp, col, val, x)
    with gefel.DeviceMatrix(rp, col, val, 0) as K:
        solve_batch(K, rows, f)
        rc, got, _, st, _ = held(other, BRIEF, lambda: solve_batch(K, rows, f))
    at = np.cumsum([0] + rows)
    assert rc == L.OK and not st.any()
    for a, b in zip(at, at[1:]):
        assert np.linalg.norm(got[a:b] - x[a:b]) <= 1e-9 * np.linalg.norm(x[a:b])


def test_solves_in_several_threads(gpu_lib):
    """Handles of their own in threads of their own, all forms at once."""
    wrong = []

    def work(name, seed):
        try:
            rowptr, col, val = SYSTEMS[name][0]()
            n = len(rowptr) - 1
            rng = np.random.default_rng(seed)
            with gefel.DeviceMatrix(rowptr, col, val, 0) as K:
                for _ in range(5):
                    x = rng.standard_normal(n)
                    got, r = K.pcg(product(np.asarray(rowptr), col, val, x), res=1e-20)
                    if r.status != L.OK or np.linalg.norm(got - x) > 2e-9 * np.linalg.norm(x):
                        wrong.append((name, r.status))
        except Exception as e:  # noqa: BLE001
            wrong.append((name, repr(e)))

    names = ["resident", "csr_2", "bsr_8", "resident", "bsr_16", "csr_8"]
    threads = [threading.Thread(target=work, args=(n, k)) for k, n in enumerate(names)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
