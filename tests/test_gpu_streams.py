"""A handle's work on streams of the caller's: the per-thread default stream, which means another stream in every
thread, and a product recorded into a graph after a solve."""
import numpy as np
import pytest

from ssf_b200 import _lib as L
from ssf_b200 import decks, mefel
from ssf_b200.gefel import DeviceMatrix

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread


@pytest.mark.parametrize("n", [1000, (4 << 20) // 8, 5 * ((4 << 20) // 8) + 7])
def test_copies_on_the_per_thread_default_stream(gpu_lib, n):
    """Below, at and above the size from which several threads copy.  The matrix is diagonal: products are exact."""
    rng = np.random.default_rng(n)
    with DeviceMatrix(np.arange(n + 1), np.arange(n), np.ones(n), 0) as K:
        L.check(gpu_lib.sgpu_matrix_set_stream(K.h, PER_THREAD))
        for _ in range(8):
            a, x = rng.standard_normal(n), rng.standard_normal(n)
            K.update_values(a)
            assert np.array_equal(K.mxv(x), a * x)


@pytest.mark.parametrize("make", [lambda: decks.cantilever_hex(17, 5, 3), lambda: decks.cantilever_hex(48, 16, 15),
                                  lambda: decks.plate_quad(33, 21)])
def test_product_recorded_after_a_solve(gpu_lib, make):
    """A solve leaves the handle ready for products on a capturing stream: nothing is timed or allocated there.
    The eager product may sum in another order."""
    import torch
    mesh = make()
    with mefel.stiffness_matrix(mesh) as K:
        _, r = K.pcg(np.ones(K.n), ni=5)
        assert r.status in (L.OK, L.NOT_CONVERGED)
        x = torch.randn(K.n, dtype=torch.float64, device="cuda")
        y = torch.zeros_like(x)
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        L.check(gpu_lib.sgpu_matrix_set_stream(K.h, stream.cuda_stream))
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            L.check(gpu_lib.sgpu_matrix_mxv_d(K.h, x.data_ptr(), y.data_ptr()))
        assert not y.any()
        graph.replay()
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        del graph
        want = K.mxv(x.cpu().numpy())
        # two sums of at most 243 products
        bound = 2 * 243 * 2.3e-16 * 243 * np.abs(K.download(0)[2]).max() * x.abs().max().item()
        assert np.abs(got - want).max() <= bound
