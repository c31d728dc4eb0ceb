"""Meshes whose nodes share equations (code numbers given to several nodes, as gtopology::gencodnum does for tied
degrees of freedom, GEFEL/gtopology.cpp:1619-1680): K = T^T K_free T, with T from the free numbering to the shared one.

The ties: opposite faces several elements apart, neighbouring nodes (elements of one colour that share no node but an
equation), both faces of a layer one element thick (nodes of one element share an equation), single components.
"""
import ctypes as C

import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import decks, mefel
from ssf_b200.gefel import DeviceMatrix

pytestmark = pytest.mark.gpu

KINDS = {
    "hex8": (L.ELEM_HEX8, lambda: decks.cantilever_hex(6, 3, 1)),
    "hex20": (L.ELEM_HEX20, lambda: decks.cantilever_hex20(3, 2, 1)),
    "tet4": (L.ELEM_TET4, lambda: decks.cantilever_tet(5, 3, 1)),
    "quad4": (L.ELEM_QUAD4, lambda: decks.plate_quad(9, 1)),
    "quad8": (L.ELEM_QUAD8, lambda: decks.plate_quad8(7, 1)),
    "tri3": (L.ELEM_TRI3, lambda: decks.plate_tri(8, 1)),
}


def tie(mesh, pairs):
    """Code numbers in which the given (slave, master, component) share the master's equation, renumbered without
    gaps; and the shared equation of every free one."""
    cn = mesh.code_numbers().copy()
    free = cn.copy()
    for s, m, c in pairs:
        if cn[s, c] > 0 and cn[m, c] > 0:
            cn[cn == cn[s, c]] = cn[m, c]
    used = np.unique(cn[cn > 0])
    new = np.zeros(cn.max() + 1, dtype=np.int64)
    new[used] = np.arange(1, used.size + 1)
    tied = np.where(cn > 0, new[np.maximum(cn, 0)], cn)
    to = np.empty(free.max(), dtype=np.int64)
    to[free[free > 0] - 1] = tied[free > 0] - 1
    return tied, to


def assemble(mesh, kind, cn):
    keep = [np.ascontiguousarray(v) for v in (mesh.coords, mesh.elems, cn, mesh.mats[mesh.emat])]
    thick = None if mesh.thick is None else np.ascontiguousarray(mesh.thick)
    m = L.Mesh(kind, cn.shape[1], mesh.nn, keep[0].ctypes.data, keep[1].shape[0], keep[1].ctypes.data,
               keep[2].ctypes.data, keep[3].ctypes.data, None if thick is None else thick.ctypes.data, None, None)
    h, info = C.c_void_p(), L.AssemblyInfo()
    L.check(L.lib().sgpu_assemble(C.byref(m), C.byref(h), C.byref(info)))
    return DeviceMatrix.from_handle(h, info.n, 1)


def dense(K):
    adr, ci, a = K.download(0)
    out = np.zeros((K.n, K.n))
    out[np.repeat(np.arange(K.n), np.diff(adr)), ci] = a
    return out


def ends(mesh):
    """(node of the far face, the node it faces across the length); x runs along the mesh."""
    x = mesh.coords[:, 0]
    far, near = np.flatnonzero(x > x.max() - 1e-9), np.flatnonzero(np.abs(x - np.unique(x.round(9))[2]) < 1e-6)
    return [(a, b) for a in far for b in near if np.allclose(mesh.coords[a, 1:], mesh.coords[b, 1:])]


def faces(mesh):
    """(node of one side of the layer, the node across its thickness)"""
    c = np.flatnonzero(np.ptp(mesh.coords, axis=0) > 0)[-1]
    x = mesh.coords[:, c]
    other = [d for d in range(3) if d != c]
    hi, lo = np.flatnonzero(x > x.max() - 1e-9), np.flatnonzero(x < x.min() + 1e-9)
    return [(a, b) for a in hi for b in lo if np.allclose(mesh.coords[a][other], mesh.coords[b][other])]


def chain(mesh):
    """pairs of nodes two apart all through the mesh"""
    return [(k, k + 2) for k in range(0, mesh.nn - 2, 4)]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("ties", [ends, faces, chain])
def test_the_largest_code_number_is_the_number_of_equations(gpu_lib, kind, ties):
    kid, make = KINDS[kind]
    mesh = make()
    cn, to = tie(mesh, [(s, m, c) for s, m in ties(mesh) for c in range(mesh.ndofn)])
    with mefel.stiffness_matrix(mesh) as F:
        adr, ci, _ = F.download(0)
    rows = np.repeat(np.arange(F.n), np.diff(adr))
    want = np.unique(to[rows] * (to.max() + 1) + to[ci])
    with assemble(mesh, kid, cn) as A:
        assert A.n == cn.max() < F.n
        adr, ci, _ = A.download(0)
        assert np.array_equal(np.repeat(np.arange(A.n), np.diff(adr)) * A.n + ci, want)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("ties", [ends, faces, chain])
@pytest.mark.parametrize("whole", [True, False])
def test_shared_equations(gpu_lib, kind, ties, whole):
    kid, make = KINDS[kind]
    mesh = make()
    comps = range(mesh.ndofn) if whole else range(1)
    pairs = [(s, m, c) for s, m in ties(mesh) for c in comps]
    assert pairs
    cn, to = tie(mesh, pairs)
    with mefel.stiffness_matrix(mesh) as F:
        K = dense(F)
    T = np.zeros((K.shape[0], to.max() + 1))
    T[np.arange(K.shape[0]), to] = 1.0
    want = T.T @ K @ T
    with assemble(mesh, kid, cn) as A:
        assert A.n == to.max() + 1 < K.shape[0]
        got = dense(A)
    # sums of the same element terms in another order; an entry has at most (tied nodes x elements)^2 terms
    terms = int(np.bincount(to).max()) ** 2 * 64
    assert np.abs(got - want).max() <= terms * 2.3e-16 * np.abs(K).max() * terms


@pytest.mark.parametrize("kind", ["hex8", "quad4"])
@pytest.mark.parametrize("ties", [ends, faces, chain])
def test_lifting_onto_shared_equations(gpu_lib, kind, ties):
    kid, make = KINDS[kind]
    mesh = make()
    cn, to = tie(mesh, [(s, m, c) for s, m in ties(mesh) for c in range(mesh.ndofn)])
    r = np.random.default_rng(4).standard_normal((mesh.nn, mesh.ndofn))
    with mefel.stiffness_matrix(mesh) as F, assemble(mesh, kid, cn) as A:
        f, g = np.zeros(F.n), np.zeros(A.n)
        L.check(gpu_lib.sgpu_assembly_lift(F.h, r, f))
        L.check(gpu_lib.sgpu_assembly_lift(A.h, r, g))
        entry = np.abs(F.download(0)[2]).max()
    want = np.zeros(A.n)
    np.add.at(want, to, f)
    # sums of at most 24 x 8 products for each of the tied nodes
    terms = 192 * int(np.bincount(to).max())
    assert np.abs(g - want).max() <= terms * 2.3e-16 * terms * entry * np.abs(r).max()
