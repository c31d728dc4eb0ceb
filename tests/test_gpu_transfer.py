"""Host arrays through the pinned slots: sizes below and at the line (4 MiB),
a last piece of one value, several rounds of every slot, two threads at once
(the second finds the slots in use), pinned arrays; and blocks that a handle
gave back.  The matrix is 2 I, so products are exact.
"""
import threading

import numpy as np
import pytest

from ssf_b200.gefel import DeviceMatrix

pytestmark = pytest.mark.gpu

LINE = (4 << 20) // 8  # values


def double(n, scale=2.0):
    return DeviceMatrix(np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int64), np.full(n, scale), 0)


@pytest.mark.parametrize("n", [1, 1000, LINE - 1, LINE, LINE + 1, 2 * LINE + 131071, 5 * LINE + 7])
def test_sizes(gpu_lib, n):
    x = np.random.default_rng(n).standard_normal(n)
    with double(n) as K:
        assert np.array_equal(K.mxv(x), 2.0 * x)
        K.update_values(np.arange(1.0, n + 1.0))
        assert np.array_equal(K.mxv(x), np.arange(1.0, n + 1.0) * x)


def test_pinned_arrays(gpu_lib):
    import torch
    x = torch.randn(LINE + 1, dtype=torch.float64).pin_memory().numpy()
    with double(x.size) as K:
        assert np.array_equal(K.mxv(x), 2.0 * x)


def test_two_threads(gpu_lib):
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        for k in range(6):
            n = 2 * LINE + int(rng.integers(1000))
            x = rng.standard_normal(n)
            with double(n, float(k + 1)) as K:
                if not np.array_equal(K.mxv(x), (k + 1) * x):
                    bad.append((seed, k))

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
