"""The coarse levels of a cycle as one launch where level 1 is small, as launches of their own beyond: on both sides of
the line, with the same bits."""
import numpy as np
import pytest

from ssf_b200 import decks, mefel

pytestmark = pytest.mark.gpu

MESHES = {
    # name: (mesh, whether level 1 starts a program in FP64, in FP32)
    "conduction_1561": (lambda: decks.heat_cube(32), True, True),
    "conduction_3009": (lambda: decks.heat_cube(40), False, False),
    "plate_5278": (lambda: decks.plate_quad(200, 200), True, True),
    "plate_11803": (lambda: decks.plate_quad(300, 300), False, False),
    "bar_1025": (lambda: decks.cantilever_hex(60, 18, 18), True, False),
    "bar_5139": (lambda: decks.cantilever_hex(120, 30, 30), False, False),
}


@pytest.mark.parametrize("name", MESHES)
@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_form_and_bits(gpu_lib, monkeypatch, name, mode):
    make, fp64, fp32 = MESHES[name]
    mesh = make()
    heat = name.startswith("conduction")
    with (mefel.conductivity_matrix if heat else mefel.stiffness_matrix)(mesh) as K:
        if not heat:
            K.set_rigid_body_modes(mesh.coords, mesh.code_numbers())
        f = np.random.default_rng(1).standard_normal(K.n)
        K.pcg(f, prec="agg", mode=mode, res=1e-16)  # hierarchy and plans

        def solve():
            before = gpu_lib.sgpu_kernel_launches()
            x, r = K.pcg(f, prec="agg", mode=mode, res=1e-16)
            return x, r.info["iterations"], gpu_lib.sgpu_kernel_launches() - before

        x1, its1, launches1 = solve()
        monkeypatch.setenv("SGPU_AMG_TAIL", "0")
        x0, its0, launches0 = solve()
    assert np.array_equal(x0, x1) and its0 == its1
    # an iteration of the kernels' form has at least three launches a coarse level more
    assert (launches1 < launches0 - 3 * its0) == (fp64 if mode == "fp64" else fp32), (launches1, launches0)
