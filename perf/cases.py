"""The workloads this framework is measured on.

Each case is one call a user's program makes through the public entry points
(the C ABI of include/sifelgpu.h or its Python mirror): the reference's CG
call on host arrays, solves on a device-resident matrix with both
preconditioners and both cycle precisions, a block of load cases, a batch of
independent plates, time steps of transient conduction, assembly, and the
solver that allocates nothing.  Sizes run from the smallest example problem
(1500 equations) to the 1.01M-equation cantilever.

Meshes are structured grids in SIFEL's node order with seeded materials and
loads; ``distort`` moves interior nodes by that share of a cell, ``scatter``
spreads the elements' moduli lognormally.  Solutions are returned whole;
iteration counts are not, since a last iteration more or less is within the
stopping test.

``exact`` recomputes every result in FP64 torch from element matrices formed
here (no assembled matrix): Jacobi-PCG to the rounding floor.
"""
import ctypes as C

import numpy as np
import torch

from ssf_b200 import _lib as L
from ssf_b200 import decks, gefel

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest example problem, one call of the reference's solver from host arrays: latency
        dict(name="dropin_small", kind="dropin", elem="hex8", nx=20, ny=4, nz=4, storage="scr", distort=0.0,
             scatter=0.0),
        # the same call at the size of an ordinary model: upload, formats, ~600 iterations
        dict(name="dropin_medium", kind="dropin", elem="hex8", nx=100, ny=20, nz=20, storage="scr", distort=0.0,
             scatter=0.0),
        # the plain FP64 Jacobi-PCG on a resident matrix, the largest model
        dict(name="jacobi_1m", kind="jacobi", elem="hex8", nx=200, ny=40, nz=40, distort=0.0, scatter=0.0),
        # the fastest form on the largest model: FP64 flexible CG, FP32 cycle, hierarchy set up in the call
        dict(name="agg_mixed_1m", kind="agg", elem="hex8", nx=200, ny=40, nz=40, mode="mixed", distort=0.0,
             scatter=0.0),
        # the all-FP64 cycle on an ordinary model with odd sides, distorted cells and scattered moduli
        dict(name="agg_fp64_medium", kind="agg", elem="hex8", nx=83, ny=25, nz=19, mode="fp64", distort=0.15,
             scatter=0.3),
        # 64 load cases at once from pinned host memory, the hierarchy set up in the call
        dict(name="load_cases_64", kind="loads", elem="hex8", nx=100, ny=20, nz=20, nrhs=64, mode="mixed", distort=0.0,
             scatter=0.0),
        # many independent plates of uneven size, each its own Jacobi-PCG
        dict(name="plates_jacobi_256", kind="plates", count=256, lo=16, hi=128, prec="jacobi", mode="fp64"),
        # the same batch with the shared hierarchy, FP32 cycle
        dict(name="plates_agg_256", kind="plates", count=256, lo=16, hi=128, prec="agg", mode="mixed"),
        # implicit Euler steps of heterogeneous conduction, the largest grid
        dict(name="heat_128_steps", kind="heat", n=128, steps=10, dt=10.0, sigma=1.0),
        # stiffness matrix of the largest model and one product with it
        dict(name="assemble_hex8_1m", kind="assemble", elem="hex8", nx=200, ny=40, nz=40, distort=0.0, scatter=0.0),
        # stiffness matrix of a quadratic model and one product with it
        dict(name="assemble_hex20", kind="assemble", elem="hex20", nx=48, ny=16, nz=15, distort=0.1, scatter=0.3),
        # the solver that allocates nothing, a plate's matrix near its largest size
        dict(name="noalloc_plate", kind="noalloc", elem="quad4", nx=251, ny=201, distort=0.0, scatter=0.0),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def _beam(rng, lo, hi):
    """Sides of a bar 1 to 6 times as long as it is wide, of about lo..hi hexahedra (log-uniform)."""
    cells, ratio = _log_int(rng, lo, hi), rng.uniform(1.0, 6.0)
    ny = max(2, int(round((cells / ratio) ** (1.0 / 3.0))))
    nz = max(2, ny + rng.randint(-(ny // 4), ny // 4))
    return dict(nx=max(2, cells // (ny * nz)), ny=ny, nz=nz)


def _shape(rng):
    return dict(distort=rng.choice([0.0, 0.0, 0.1, 0.2]), scatter=rng.choice([0.0, 0.0, 0.3, 0.6]))


def draw(rng):
    kind = rng.choice(["dropin", "jacobi", "agg", "loads", "plates", "heat", "assemble", "noalloc"])
    if kind == "dropin":
        if rng.random() < 0.3:
            return dict(kind=kind, elem="quad4", nx=_log_int(rng, 8, 160), ny=_log_int(rng, 8, 160),
                        storage=rng.choice(["scr", "cr"]), **_shape(rng))
        return dict(kind=kind, elem="hex8", **_beam(rng, 60, 40000), storage=rng.choice(["scr", "scr", "cr"]),
                    **_shape(rng))
    if kind == "jacobi":
        return dict(kind=kind, elem="hex8", **_beam(rng, 2000, 200000), **_shape(rng))
    if kind == "agg":
        return dict(kind=kind, elem="hex8", **_beam(rng, 4000, 300000), mode=rng.choice(["mixed", "mixed", "fp64"]),
                    **_shape(rng))
    if kind == "loads":
        return dict(kind=kind, elem="hex8", **_beam(rng, 1000, 40000), nrhs=_log_int(rng, 2, 64), mode="mixed",
                    **_shape(rng))
    if kind == "plates":
        lo = _log_int(rng, 6, 40)
        return dict(kind=kind, count=_log_int(rng, 12, 250), lo=lo, hi=rng.randint(lo + 1, 128),
                    prec=rng.choice(["jacobi", "agg"]), mode=rng.choice(["mixed", "fp64"]))
    if kind == "heat":
        return dict(kind=kind, n=_log_int(rng, 12, 120), steps=rng.randint(3, 10), dt=rng.choice([10.0, 100.0]),
                    sigma=rng.choice([0.5, 1.0]))
    if kind == "assemble":
        elem = rng.choice(["hex8", "hex8", "hex20", "quad4", "quad8"])
        if elem in ("quad4", "quad8"):
            return dict(kind=kind, elem=elem, nx=_log_int(rng, 20, 400), ny=_log_int(rng, 20, 400), **_shape(rng))
        return dict(kind=kind, elem=elem, **_beam(rng, 500, 250000 if elem == "hex8" else 11000), **_shape(rng))
    if rng.random() < 0.5:
        return dict(kind=kind, elem="quad4", nx=_log_int(rng, 16, 250), ny=_log_int(rng, 16, 250), **_shape(rng))
    return dict(kind=kind, elem="hex8", **_beam(rng, 60, 30000), **_shape(rng))


# ---------------------------------------------------------------------------
# structured meshes (both prepare and exact start from these)
# ---------------------------------------------------------------------------

# natural coordinates of the nodes in SIFEL's order; the linear elements are the first nodes of the quadratic ones
HEX20 = np.array([[1, 1, 1], [-1, 1, 1], [-1, -1, 1], [1, -1, 1], [1, 1, -1], [-1, 1, -1], [-1, -1, -1], [1, -1, -1],
                  [0, 1, 1], [-1, 0, 1], [0, -1, 1], [1, 0, 1], [1, 1, 0], [-1, 1, 0], [-1, -1, 0], [1, -1, 0],
                  [0, 1, -1], [-1, 0, -1], [0, -1, -1], [1, 0, -1]])
QUAD8 = np.array([[1, 1], [-1, 1], [-1, -1], [1, -1], [0, 1], [-1, 0], [0, -1], [1, 0]])
NODES = {"hex8": HEX20[:8], "hex20": HEX20, "hex8t": HEX20[:8], "quad4": QUAD8[:4], "quad8": QUAD8}


def _grid(elem, cells, lengths, distort, rng):
    """Nodes (x fastest) and elements of a box of cells; interior corner nodes moved by up to `distort` of half a
    cell, mid-side nodes kept in the middle of their edges."""
    dim, quadratic = len(cells), elem in ("hex20", "quad8")
    half = [np.arange(2 * c + 1) for c in cells[::-1]]  # slowest axis first
    pos = np.stack([g.ravel() for g in np.meshgrid(*half, indexing="ij")][::-1], axis=1)
    odd = (pos % 2).sum(axis=1)
    keep = odd <= (1 if quadratic else 0)
    ids = np.full(keep.size, -1, dtype=np.int64)
    ids[keep] = np.arange(int(keep.sum()))
    pos = pos[keep]
    step = np.array([length / (2.0 * c) for length, c in zip(lengths, cells)])
    xyz = pos * step
    stride = np.cumprod([1] + [2 * c + 1 for c in cells[:-1]])
    if distort:
        inner = ((pos > 0) & (pos < 2 * np.array(cells)) & (pos % 2 == 0).all(axis=1)[:, None]).all(axis=1)
        move = rng.uniform(-distort, distort, xyz.shape) * step * inner[:, None]
        moved = move.copy()
        for a in range(dim):  # an edge's middle moves by the mean of its ends
            mid = pos[:, a] % 2 == 1
            code = pos[mid] @ stride
            moved[mid] = 0.5 * (move[ids[code - stride[a]]] + move[ids[code + stride[a]]])
        xyz = xyz + moved
    centre = np.stack([g.ravel() for g in np.meshgrid(*[2 * np.arange(c) + 1 for c in cells[::-1]], indexing="ij")][::-1],
                      axis=1)
    elems = ids[((centre[:, None, :] + NODES[elem][None]) @ stride)]
    coords = np.zeros((xyz.shape[0], 3))
    coords[:, :dim] = xyz
    return coords, elems


def _body(case, seed):
    """A clamped elastic bar or plate (x = 0 fixed) with a noisy traction on its far end."""
    rng = np.random.default_rng([int(seed), 7])
    elem, solid = case["elem"], case["elem"].startswith("hex")
    cells = (case["nx"], case["ny"], case["nz"]) if solid else (case["nx"], case["ny"])
    lengths = [0.05 * c for c in cells] if solid else [float(c) for c in cells]
    coords, elems = _grid(elem, cells, lengths, case["distort"], rng)
    nn, ne, nd = coords.shape[0], elems.shape[0], 3 if solid else 2
    free = np.ones((nn, nd), dtype=bool)
    free[coords[:, 0] < 1e-9] = False
    E = (210e9 if solid else 10 ** rng.uniform(9.0, 11.0)) * np.exp(case["scatter"] * rng.standard_normal(ne))
    E *= rng.uniform(0.9, 1.1)
    nu = np.full(ne, rng.uniform(0.2, 0.35))
    loads = np.zeros((nn, nd))
    end = coords[:, 0] > lengths[0] - 1e-9
    pull = rng.standard_normal(nd)
    loads[end] = 1.0e3 * (pull / np.linalg.norm(pull) + 0.1 * rng.standard_normal((int(end.sum()), nd)))
    return dict(elem=elem, coords=coords, elems=elems, free=free, mats=np.stack([E, nu], axis=1),
                thick=None if solid else np.full(ne, 0.01), f=loads[free])


def _plates(case, seed):
    """Plates of uneven size (unit cells, left edge clamped, 1 MPa traction on the right), one after the other; the
    sizes belong to the case, materials to the seed."""
    rng = np.random.default_rng([int(seed), 11])
    sides = np.random.default_rng([case["count"], case["lo"], case["hi"]]).integers(case["lo"], case["hi"] + 1,
                                                                                  size=(case["count"], 2))
    parts, rows, base = [], [], 0
    for nx, ny in sides.tolist():
        coords, elems = _grid("quad4", (nx, ny), (float(nx), float(ny)), 0.0, rng)
        free = np.ones((coords.shape[0], 2), dtype=bool)
        free[coords[:, 0] < 1e-9] = False
        mats = np.tile([10 ** rng.uniform(9.0, 11.0), rng.uniform(0.2, 0.35)], (elems.shape[0], 1))
        loads = np.zeros(free.shape)
        end = coords[:, 0] > nx - 1e-9
        loads[end, 0] = 1.0e4 * np.where((coords[end, 1] < 1e-9) | (coords[end, 1] > ny - 1e-9), 0.5, 1.0)
        parts.append((coords, elems + base, free, mats, loads))
        rows.append(int(free.sum()))
        base += coords.shape[0]
    coords, elems, free, mats, loads = (np.concatenate([p[k] for p in parts]) for k in range(5))
    return dict(elem="quad4", coords=coords, elems=elems, free=free, mats=mats, thick=np.full(elems.shape[0], 0.01),
                f=loads[free], rows=np.array(rows, dtype=np.int64))


def _cube(case, seed):
    """A unit cube with lognormal conductivities, heated on its x = 0 face."""
    rng = np.random.default_rng([int(seed), 13])
    n = case["n"]
    coords, elems = _grid("hex8t", (n, n, n), (1.0, 1.0, 1.0), 0.0, rng)
    hot = coords[:, 0] < 1e-9
    k = np.exp(rng.normal(0.0, case["sigma"], size=elems.shape[0]))
    return dict(elem="hex8t", coords=coords, elems=elems, free=~hot[:, None],
                mats=np.stack([k, np.full_like(k, 2.0e6)], axis=1), thick=None, hot=np.where(hot, 1.0, 0.0),
                d0=0.1 * rng.random(int((~hot).sum())))


def _load_block(case, p, seed):
    """nrhs load cases of N(0,1) kN z-forces on the free nodes of the top face, one row each."""
    rng = np.random.default_rng([int(seed), 17])
    top = p["coords"][:, 2] > p["coords"][:, 2].max() - 1e-9
    out = np.zeros((case["nrhs"],) + p["free"].shape)
    out[:, top, 2] = 1.0e3 * rng.standard_normal((case["nrhs"], int(top.sum())))
    return np.ascontiguousarray(out[:, p["free"]])


def _problem(case, seed):
    return {"plates": _plates, "heat": _cube}.get(case["kind"], _body)(case, seed)


# ---------------------------------------------------------------------------
# what a user's program holds before the call
# ---------------------------------------------------------------------------


class _Input:
    """The mesh as sgpu_assemble takes it (the arrays are kept alive beside the struct)."""

    def __init__(self, p, kind):
        mesh = decks.Mesh(kind=p["elem"], coords=p["coords"], elems=p["elems"], dofflag=p["free"].astype(np.int64),
                          emat=np.arange(p["elems"].shape[0]), mats=p["mats"], loads=None, thick=p["thick"])
        self.cn = np.ascontiguousarray(mesh.code_numbers())
        self.coords, self.elems = np.ascontiguousarray(p["coords"]), np.ascontiguousarray(p["elems"])
        self.mats, self.thick = np.ascontiguousarray(p["mats"]), p["thick"]
        self.c = L.Mesh(kind, self.cn.shape[1], self.coords.shape[0], self.coords.ctypes.data, self.elems.shape[0],
                        self.elems.ctypes.data, self.cn.ctypes.data, self.mats.ctypes.data,
                        self.thick.ctypes.data if self.thick is not None else None, None, None)

    def assemble(self):
        h, info = C.c_void_p(), L.AssemblyInfo()
        L.check(L.lib().sgpu_assemble(C.byref(self.c), C.byref(h), C.byref(info)))
        return gefel.DeviceMatrix.from_handle(h, info.n, 1)


ELEM = {"hex8": L.ELEM_HEX8, "hex20": L.ELEM_HEX20, "quad4": L.ELEM_QUAD4, "quad8": L.ELEM_QUAD8}


def prepare(case, seed):
    p = _problem(case, seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "heat":
        s["K"] = _Input(p, L.ELEM_HEX8T_K).assemble()
        s["C"] = _Input(p, L.ELEM_HEX8T_C).assemble()
        s["rhs"] = np.zeros(s["K"].n)
        L.check(L.lib().sgpu_assembly_lift(s["K"].h, p["hot"], s["rhs"]))
        s["d0"] = p["d0"]
        return s
    inp = _Input(p, ELEM[p["elem"]])
    if kind == "assemble":
        s["input"] = inp
        n = int(p["free"].sum())
        s["x"] = torch.from_numpy(np.random.default_rng([int(seed), 19]).standard_normal(n)).cuda()
        s["y"] = torch.empty(n, dtype=torch.float64, device="cuda")
        return s
    K = inp.assemble()
    if kind == "dropin":
        cls = gefel.symcomprow if case["storage"] == "scr" else gefel.comprow
        s["A"] = cls(*K.download(1 if case["storage"] == "scr" else 0))
        s["f"] = p["f"]
        K.close()
    elif kind == "noalloc":
        adr, ci, a = K.download(0)
        K.close()
        s["rowptr"], s["col"] = torch.from_numpy(adr).int().cuda(), torch.from_numpy(ci).int().cuda()
        s["val"], s["f"] = torch.from_numpy(a).cuda(), torch.from_numpy(p["f"]).cuda()
        s["x"] = torch.empty_like(s["f"])
    elif kind == "loads":
        s["K"] = K
        K.set_rigid_body_modes(inp.coords, inp.cn)
        s["F"] = torch.from_numpy(_load_block(case, p, seed)).pin_memory().numpy()
        s["X"] = torch.zeros(s["F"].shape, dtype=torch.float64).pin_memory().numpy()
    elif kind == "plates":
        s["K"], s["rows"], s["f"], s["x"] = K, p["rows"], p["f"], np.zeros(K.n)
        K.set_rigid_body_modes(inp.coords, inp.cn)
    else:
        s["K"], s["f"] = K, torch.from_numpy(p["f"]).cuda()
        s["x"] = torch.empty_like(s["f"])
        if kind == "agg":
            K.set_rigid_body_modes(inp.coords, inp.cn)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
MODE = {"fp64": L.FP64, "mixed": L.MIXED}


def _run_dropin(s):
    x = np.zeros(s["A"].n)
    if s["case"]["storage"] == "scr":
        r = s["A"].cg_prec(x, s["f"], 100000, 1e-20)
    else:  # comprow::cg_prec stops on sqrt(r.r / f.f)
        r = s["A"].cg_prec(x, s["f"], 100000, 1e-10)
    L.check(r.status)
    return x


def _run_pcg(s, prec, mode, crit, res):
    L.check(L.lib().sgpu_matrix_pcg_d(s["K"].h, s["x"].data_ptr(), s["f"].data_ptr(), 100000, res, 1e-30, 0, crit, prec,
                                      mode, None, None, None))
    return s["x"]


def _run_jacobi(s):
    return _run_pcg(s, L.PREC_JACOBI, L.FP64, L.CRIT_SCR_PREC, 1e-20)


def _run_agg(s):
    s["K"].precond_clear()  # new values each time in a user's program: the hierarchy is part of the solve
    return _run_pcg(s, L.PREC_AGG, MODE[s["case"]["mode"]], L.CRIT_TRUE, 1e-10)


def _run_loads(s):
    s["K"].precond_clear()
    X, out = gefel.pcg_multi_blocks(s["K"], s["F"], res=1e-20, prec="agg", mode=s["case"]["mode"], Xc=s["X"])
    return X


def _run_plates(s):
    K, nsys = s["K"], s["rows"].size
    if s["case"]["prec"] == "agg":
        K.precond_clear()
        L.check(L.lib().sgpu_matrix_pcg_batch_agg(K.h, nsys, s["rows"], s["x"], s["f"], 200000, 1e-20, 1e-30,
                                                  MODE[s["case"]["mode"]], None, None, None, None, None))
    else:
        L.check(L.lib().sgpu_matrix_pcg_batch(K.h, nsys, s["rows"], s["x"], s["f"], 200000, 1e-20, 1e-30, 0, None, None,
                                              None, None, None))
    return s["x"]


def _run_heat(s):
    # to 1e-12: the rates are differences of nearly equal temperatures
    d, v = s["d0"].copy(), np.zeros(s["K"].n)
    L.check(L.lib().sgpu_transient_dform(s["K"].h, s["C"].h, s["rhs"], d, v, s["case"]["dt"], 1.0, s["case"]["steps"],
                                         100000, 1e-24, 1e-30, 1, L.PREC_JACOBI, L.FP64, None, None))
    return d, v


def _run_assemble(s):
    with s["input"].assemble() as K:
        L.check(L.lib().sgpu_matrix_mxv_d(K.h, s["x"].data_ptr(), s["y"].data_ptr()))
    return s["y"]


def _run_noalloc(s):
    L.check(L.lib().sgpu_csr_pcg_noalloc_d(s["f"].numel(), s["rowptr"].data_ptr(), s["col"].data_ptr(),
                                           s["val"].data_ptr(), s["f"].data_ptr(), s["x"].data_ptr(), 100000, 1e-20,
                                           1e-30, 0, None, None, None, None))
    return s["x"]


RUN = dict(dropin=_run_dropin, jacobi=_run_jacobi, agg=_run_agg, loads=_run_loads, plates=_run_plates, heat=_run_heat,
           assemble=_run_assemble, noalloc=_run_noalloc)


def run(state):
    return RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------
# the least a pass must move and compute
# ---------------------------------------------------------------------------


def _counts(case):
    """(equations, stored entries of the full matrix, elements) of a case, boundary rows counted as inner ones'
    share of the grid."""
    if case["kind"] == "plates":
        side = 0.5 * (case["lo"] + case["hi"])
        cells, elem, reps = (side, side), "quad4", case["count"]
    elif case["kind"] == "heat":
        cells, elem, reps = (case["n"],) * 3, "hex8t", 1
    else:
        elem, reps = case["elem"], 1
        cells = (case["nx"], case["ny"], case["nz"]) if elem.startswith("hex") else (case["nx"], case["ny"])
    nd = {"hex8": 3, "hex20": 3, "hex8t": 1, "quad4": 2, "quad8": 2}[elem]
    ne, corners, links, edges = 1.0, 1.0, 1.0, 0.0
    for c in cells:
        ne, corners, links = ne * c, corners * (c + 1), links * (3 * c + 1)
    if elem in ("hex20", "quad8"):
        for a, c in enumerate(cells):
            e = c
            for b, o in enumerate(cells):
                e *= 1 if a == b else o + 1
            edges += e
        links = links + 2.0 * edges * (20 if elem == "hex20" else 8)
    return reps * nd * (corners + edges), reps * nd * nd * links, reps * ne


def work(case):
    """One pass: the matrix (values and 4-byte columns), right-hand sides and solutions once each; the assembly reads
    its elements and writes the matrix.  Operations: one product of the matrix with each vector, or the integration
    points' products of the element matrices."""
    n, nnz, ne = _counts(case)
    vec = case.get("nrhs", 1)
    if case["kind"] == "assemble":
        nne, pts = {"hex8": (8, 8), "hex20": (20, 27), "quad4": (4, 4), "quad8": (8, 9)}[case["elem"]]
        nd = 3 if case["elem"].startswith("hex") else 2
        return {"bytes": 12.0 * nnz + 16.0 * n + ne * (8.0 * nne + 16.0), "flops": ne * pts * (nne * nd) ** 2 * 2.0 * nd}
    if case["kind"] == "heat":
        return {"bytes": 24.0 * nnz + 32.0 * n, "flops": case["steps"] * 4.0 * nnz}
    return {"bytes": 12.0 * nnz + 16.0 * n * vec, "flops": 2.0 * nnz * vec}


# ---------------------------------------------------------------------------
# the same results in plain FP64 torch
# ---------------------------------------------------------------------------


def _shape_functions(elem):
    """Values (points x nodes), natural gradients (points x nodes x dim) and weights of the element's Gauss rule:
    the polynomial basis of the element's space, made 1 at its own node."""
    nodes = NODES[elem].astype(float)
    nne, dim = nodes.shape
    powers = [p for p in np.ndindex(*(3,) * dim)
              if sum(q for q in p if q == 2) <= (2 if elem in ("hex20", "quad8") else 0)]
    powers = np.array(powers, dtype=float)

    def mono(x):
        return np.prod(x[:, None, :] ** powers[None], axis=2)

    coef = np.linalg.inv(mono(nodes))  # basis k -> node value
    t, w = np.polynomial.legendre.leggauss(3 if elem in ("hex20", "quad8") else 2)
    pts = np.stack([g.ravel() for g in np.meshgrid(*(t,) * dim, indexing="ij")], axis=1)
    wts = np.prod(np.stack([g.ravel() for g in np.meshgrid(*(w,) * dim, indexing="ij")], axis=1), axis=1)
    grads = []
    for a in range(dim):
        low = powers.copy()
        low[:, a] = np.maximum(low[:, a] - 1.0, 0.0)
        grads.append((powers[:, a] * np.prod(pts[:, None, :] ** low[None], axis=2)) @ coef)
    return mono(pts) @ coef, np.stack(grads, axis=2), wts


def _element_matrices(p, capacity=False):
    """All element matrices (ne x d x d) on the GPU in FP64."""
    elem = p["elem"]
    N, dN, w = (torch.from_numpy(v).cuda() for v in _shape_functions(elem))
    dim = dN.shape[2]
    xyz = torch.from_numpy(p["coords"][:, :dim]).cuda()[torch.from_numpy(p["elems"]).cuda()]
    mats = torch.from_numpy(p["mats"]).cuda()
    ne, nne = xyz.shape[:2]
    nd = 1 if elem == "hex8t" else dim
    Ke = torch.zeros(ne, nne, nd, nne, nd, dtype=torch.float64, device="cuda")
    eye = torch.eye(nd, dtype=torch.float64, device="cuda")
    E, nu = mats[:, 0], mats[:, 1]
    mu = E / (2.0 * (1.0 + nu))
    lam = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)) if dim == 3 else E * nu / (1.0 - nu * nu)
    thick = torch.from_numpy(p["thick"]).cuda() if p["thick"] is not None else None
    for g in range(w.numel()):
        J = torch.einsum("nd,enk->edk", dN[g], xyz)
        det = torch.linalg.det(J).abs() * w[g]
        if thick is not None:
            det = det * thick
        if elem == "hex8t":
            if capacity:
                Ke[:, :, 0, :, 0] += (det * mats[:, 1])[:, None, None] * torch.outer(N[g], N[g])
                continue
            G = torch.linalg.solve(J, dN[g].T.expand(ne, dim, nne))
            Ke[:, :, 0, :, 0] += (det * mats[:, 0])[:, None, None] * (G.transpose(1, 2) @ G)
            continue
        G = torch.linalg.solve(J, dN[g].T.expand(ne, dim, nne))  # e, component, node
        gg = torch.einsum("eia,ejb->eaibj", G, G)
        Ke += (det * lam)[:, None, None, None, None] * gg
        Ke += (det * mu)[:, None, None, None, None] * gg.transpose(2, 4)
        Ke += (det * mu)[:, None, None, None, None] * torch.einsum("eab,ij->eaibj", G.transpose(1, 2) @ G, eye)
    return Ke.reshape(ne, nne * nd, nne * nd)


class _Operator:
    """y = A x over element matrices; fixed degrees of freedom share a last, zero entry.  Vectors are n x k."""

    def __init__(self, p, Ke):
        free = torch.from_numpy(p["free"]).cuda().reshape(-1)
        self.n = int(free.sum())
        cn = torch.where(free, torch.cumsum(free, 0) - 1, torch.full_like(free, self.n, dtype=torch.int64))
        nd = p["free"].shape[1]
        el = torch.from_numpy(p["elems"]).cuda()
        self.dof = cn[(el[:, :, None] * nd + torch.arange(nd, device="cuda")).reshape(el.shape[0], -1)]
        self.Ke = Ke
        d = torch.zeros(self.n + 1, dtype=torch.float64, device="cuda")
        d.index_add_(0, self.dof.reshape(-1), torch.diagonal(Ke, dim1=1, dim2=2).reshape(-1))
        self.diag = d[: self.n, None]

    def __call__(self, x):
        k = x.shape[1]
        xe = torch.cat([x, x.new_zeros(1, k)])[self.dof]
        y = x.new_zeros(self.n + 1, k)
        y.index_add_(0, self.dof.reshape(-1), torch.bmm(self.Ke, xe).reshape(-1, k))
        return y[: self.n]

    def solve(self, f, tol=1e-15, most=40000):
        """Jacobi-PCG on every column, restarted on the recomputed residual once."""
        x = torch.zeros_like(f)
        ff = (f * f).sum(0)
        for _ in range(2):
            r = f - self(x)
            h = r / self.diag
            d, rho = h.clone(), (r * h).sum(0)
            for it in range(most):
                q = self(d)
                alpha = rho / (d * q).sum(0).clamp_min(1e-300)
                x = x + alpha * d
                r = r - alpha * q
                h = r / self.diag
                new = (r * h).sum(0)
                d = h + (new / rho.clamp_min(1e-300)) * d
                rho = new
                if it % 50 == 49 and bool(((r * r).sum(0) <= tol * tol * ff).all()):
                    break
        return x


def exact(case, seed):
    p = _problem(case, seed)
    A = _Operator(p, _element_matrices(p))
    if case["kind"] == "assemble":
        x = torch.from_numpy(np.random.default_rng([int(seed), 19]).standard_normal(A.n)).cuda()
        return A(x[:, None])[:, 0]
    if case["kind"] == "loads":
        return A.solve(torch.from_numpy(_load_block(case, p, seed)).cuda().T.contiguous()).T.contiguous()
    if case["kind"] == "heat":
        Kfull = {**p, "free": np.ones_like(p["free"])}
        hot = torch.from_numpy(p["hot"]).cuda()[:, None]
        free = torch.from_numpy(p["free"][:, 0]).cuda()
        rhs = -_Operator(Kfull, A.Ke)(hot)[free]
        Ce = _element_matrices(p, capacity=True)
        M = _Operator(p, Ce)
        S = _Operator(p, Ce + case["dt"] * A.Ke)
        d = torch.from_numpy(p["d0"]).cuda()[:, None]
        v = torch.zeros_like(d)
        for _ in range(case["steps"]):
            new = S.solve(case["dt"] * rhs + M(d))
            v, d = (new - d) / case["dt"], new
        return d[:, 0], v[:, 0]
    return A.solve(torch.from_numpy(p["f"]).cuda()[:, None])[:, 0]
