"""Patterns built from the node adjacency, against the oracle's storage.

Nodes of up to 64 candidates (elements times their nodes) are sorted in
registers, more in shared memory; nodes may be fixed in some components only,
and node numbers may run in any order.  Values given in the storage's order
reach a handle that was assembled (or combined) without one.
"""
import numpy as np
import pytest

from ssf_b200 import decks, mefel
from ssf_b200 import _lib as L

pytestmark = pytest.mark.gpu


def shuffled(mesh, seed):
    """The mesh with its nodes renumbered at random."""
    p = np.random.default_rng(seed).permutation(mesh.nn)
    new = decks.Mesh(**{**mesh.__dict__})
    new.coords, new.dofflag, new.loads = (np.empty_like(v) for v in (mesh.coords, mesh.dofflag, mesh.loads))
    new.coords[p], new.dofflag[p], new.loads[:, p] = mesh.coords, mesh.dofflag, mesh.loads
    new.elems = p[mesh.elems]
    return new


def rollers(mesh, seed):
    """Single components of some nodes fixed beside the clamped ones."""
    new = decks.Mesh(**{**mesh.__dict__})
    new.dofflag = mesh.dofflag.copy()
    rng = np.random.default_rng(seed)
    pick = rng.choice(mesh.nn, size=max(1, mesh.nn // 5), replace=False)
    new.dofflag[pick, rng.integers(0, mesh.ndofn, size=pick.size)] = 0
    return new


MESHES = {
    "hex8_one": lambda: decks.cantilever_hex(1, 1, 1),
    "hex8": lambda: decks.cantilever_hex(7, 4, 3),
    "hex8_shuffled": lambda: shuffled(decks.cantilever_hex(6, 5, 4), 1),
    "hex8_rollers": lambda: rollers(decks.cantilever_hex(6, 3, 3), 2),
    "hex20": lambda: decks.cantilever_hex20(4, 3, 2),
    "hex20_shuffled_rollers": lambda: rollers(shuffled(decks.cantilever_hex20(3, 2, 2), 3), 4),
    "tet4": lambda: shuffled(decks.cantilever_tet(4, 3, 3), 5),
    "quad4": lambda: rollers(decks.plate_quad(9, 7), 6),
    "quad8": lambda: shuffled(decks.plate_quad8(6, 5), 7),
    "tri3": lambda: decks.plate_tri(8, 6),
}


@pytest.mark.parametrize("name", MESHES)
def test_pattern_and_values(gpu_lib, oracle, name):
    mesh = MESHES[name]()
    adr, ci, a = oracle.assemble(mesh, sym=True)
    with mefel.stiffness_matrix(mesh) as K:
        g_adr, g_ci, g_a = K.download(1)
        assert np.array_equal(g_adr, adr) and np.array_equal(g_ci, ci)
        assert K.assembly["negm_scr"] == ci.size
        assert np.abs(g_a - a).max() <= 1e-12 * np.abs(a).max()
        # values in the storage's order: every entry and its mirror image land where the pattern has them
        new = np.random.default_rng(9).standard_normal(ci.size)
        K.update_values(new)
        assert np.array_equal(K.download(1)[2], new)
        n = adr.size - 1
        rows = np.repeat(np.arange(n), np.diff(adr))
        x = np.random.default_rng(10).standard_normal(n)
        y = np.zeros(n)
        np.add.at(y, rows, new * x[ci])
        off = rows != ci
        np.add.at(y, ci[off], new[off] * x[rows[off]])
        # FP64 sums of at most 300 terms in another order
        assert np.abs(K.mxv(x) - y).max() <= 300 * 2.3e-16 * np.abs(new).max() * np.abs(x).max() * 300


def test_values_on_a_copy_and_a_combination(gpu_lib, oracle):
    import ctypes as C
    mesh = decks.heat_cube(4, seed=3)
    adr, ci, _ = oracle.assemble(mesh, sym=True, kind="hex8t_k")
    new = np.random.default_rng(1).standard_normal(ci.size)
    with mefel.conductivity_matrix(mesh) as K, mefel.assemble_copy(K, "hex8t_c") as M:
        h = C.c_void_p()
        L.check(L.lib().sgpu_matrix_combine(K.h, M.h, 2.0, 1.0, C.byref(h)))
        from ssf_b200.gefel import DeviceMatrix
        with DeviceMatrix.from_handle(h, K.n, 1) as A:
            for m in (M, A):
                m.update_values(new)
                assert np.array_equal(m.download(1)[2], new)
