"""The library's host code against a stand-in for the CUDA runtime (fake_cudart.cpp): which thread issues a copy on
which stream, and what a call that fails leads to.  No device is needed."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
SOURCES = ["sgpu_transfer.cu", "sgpu_alloc.cu", "sgpu_capi.cu"]
LARGE = 5 * (4 << 20) // 8 + 7  # values: several rounds of every copying thread
PER_THREAD = 2                  # cudaStreamPerThread


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """The host sources and the stand-in as one library, bound to each other whatever runtime the process has loaded; what
    they call in files of kernels returns 0 at once."""
    d = tmp_path_factory.mktemp("host")
    objs = []
    for src in [os.path.join(ROOT, "ssf_b200", "csrc", s) for s in SOURCES] + [os.path.join(HERE, "fake_cudart.cpp")]:
        objs.append(str(d / (os.path.basename(src) + ".o")))
        subprocess.run(["g++", "-x", "c++", "-std=c++17", "-O1", "-fPIC", "-I", os.path.join(CUDA, "include"), "-c", src,
                        "-o", objs[-1]], check=True)
    names = subprocess.run(["nm", "-g", *objs], check=True, capture_output=True, text=True).stdout.split("\n")
    names = [line.split()[-2:] for line in names if len(line.split()) >= 2 and not line.endswith(":")]
    defined = {n for kind, n in names if kind != "U"}
    missing = sorted({n for kind, n in names if kind == "U" and "sgpu" in n} - defined)
    stubs = d / "stubs.s"
    stubs.write_text(".text\n" + "".join(f".globl {n}\n{n}:\n" for n in missing) + "xorl %eax, %eax\nret\n"
                     ".section .note.GNU-stack,\"\",@progbits\n")
    out = str(d / "libhost.so")
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", out, *objs, str(stubs), "-lpthread"], check=True)
    lib = C.CDLL(out)
    yield lib


@pytest.fixture
def copies(host):
    """copy_in and copy_out, as (destination, source, bytes, stream) -> error"""
    host.fake_reset()
    out = []
    for name in ("_ZN4sgpu7copy_inEPvPKvmP11CUstream_st", "_ZN4sgpu8copy_outEPvPKvmP11CUstream_st"):
        fn = getattr(host, name)
        fn.argtypes, fn.restype = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p], C.c_int
        out.append(fn)
    yield out
    host.fake_reset()


@pytest.mark.parametrize("stream", [PER_THREAD, 0x1000])
@pytest.mark.parametrize("n", [1, (4 << 20) // 8, LARGE])
def test_every_piece_lands_on_the_callers_stream(host, copies, stream, n):
    """The per-thread default stream is another stream in another thread: only the caller may copy on it."""
    for fn in copies:
        src, dst = np.random.default_rng(n).standard_normal(n), np.zeros(n)
        assert fn(dst.ctypes.data, src.ctypes.data, 8 * n, stream) == 0
        assert np.array_equal(dst, src)
    assert stream != PER_THREAD or host.fake_foreign_copies(C.c_void_p(stream)) == 0


@pytest.mark.parametrize("call", ["cudaMemcpyAsync", "cudaEventRecord", "cudaEventSynchronize", "cudaSetDevice"])
@pytest.mark.parametrize("k", [1, 3, 7])
def test_one_failing_call_of_a_copy(host, copies, call, k):
    """A piece that fails sends the whole array once more, the plain way."""
    for fn in copies:
        host.fake_reset()
        src, dst = np.random.default_rng(k).standard_normal(LARGE), np.zeros(LARGE)
        host.fake_fail(call.encode(), k)
        assert fn(dst.ctypes.data, src.ctypes.data, 8 * LARGE, 0x1000) == 0
        assert np.array_equal(dst, src)


@pytest.mark.parametrize("n", [1, LARGE])
def test_a_copy_that_keeps_failing_says_so(host, copies, n):
    for fn in copies:
        host.fake_reset()
        src, dst = np.ones(n), np.zeros(n)
        host.fake_fail(b"cudaMemcpyAsync", 0)
        assert fn(dst.ctypes.data, src.ctypes.data, 8 * n, 0x1000) != 0


def test_no_copy_goes_unchecked():
    """The result of a copy of the caller's arrays is used wherever one is made."""
    found = 0
    for name in sorted(os.listdir(os.path.join(ROOT, "ssf_b200", "csrc"))):
        with open(os.path.join(ROOT, "ssf_b200", "csrc", name)) as f:
            text = "".join(line.split("//")[0] for line in f)
        for at in re.finditer(r"\bcopy_(in|out)\(", text):
            before = text[:at.start()].rstrip()
            found += 1
            assert before[-1] not in ";{})", (name, text[at.start():at.start() + 60])
    assert found > 20


def test_a_side_stream_that_is_not_to_be_had(host):
    """The values then take the handle's own stream, and no error stays behind for the next check of a launch."""
    n = 400000  # 3.2 MB of values: from 2 MB on they take a stream of their own
    adr, ci, a = np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int64), np.ones(n)
    create = host.sgpu_matrix_create
    create.argtypes = [C.c_int64] + [C.c_void_p] * 3 + [C.c_int32, C.c_void_p]
    for k in (0, 1, 2, 3):
        host.fake_reset()
        if k:
            host.fake_fail(b"cudaStreamCreateWithFlags", k)
        h = C.c_void_p()
        st = create(n, adr.ctypes.data, ci.ctypes.data, a.ctypes.data, 0, C.byref(h))
        if k == 1:  # the handle's own stream
            assert st == 4 and not h.value
            continue
        assert st == 0 and h.value
        assert host.fake_last_error() == 0
    host.fake_reset()
