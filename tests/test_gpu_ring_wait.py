"""The bounded wait of a warp on the barrier of a bulk copy: one answer for all lanes, whatever poll each of them gives up
at.  The limits are the test's, from one poll up to about a second."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from ssf_b200 import build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
LONG = 1 << 20


@pytest.fixture(scope="module")
def answers(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ring") / "libring.so")
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-I", build.CSRC, "-shared",
                    "-Xcompiler", "-fPIC", os.path.join(HERE, "ring_wait.cu"), "-o", out], check=True)
    fn = C.CDLL(out).ring_wait_answers

    def call(mode, limit):
        limit, got = np.asarray(limit, dtype=np.int32), np.full(32, -1, dtype=np.int32)
        assert fn(mode, limit.ctypes.data_as(C.c_void_p), got.ctypes.data_as(C.c_void_p)) == 0
        return got
    return call


def test_done_before_the_wait(gpu_lib, answers):
    assert answers(0, [1] * 32).all()


def test_done_during_the_wait(gpu_lib, answers):
    assert answers(1, [LONG] * 32).all()


def test_never_done(gpu_lib, answers):
    assert not answers(2, [1000] * 32).any()


@pytest.mark.parametrize("lane", [0, 13, 31])
def test_one_lane_gives_up(gpu_lib, answers, lane):
    limit = [LONG] * 32
    limit[lane] = 0
    assert not answers(1, limit).any()
