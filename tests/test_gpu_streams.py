"""A handle's work on streams of the caller's: the per-thread default stream, which is another stream in every
thread."""
import numpy as np
import pytest

from ssf_b200 import _lib as L
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
