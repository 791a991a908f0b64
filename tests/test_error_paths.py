"""Error paths of the library on the CPU: its own objects linked against a
runtime without a device (tests/c/fake_cudart.cpp), of which a test makes one
call fail."""
import ctypes
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

from cel_v3_b200 import celgpu

HERE = os.path.dirname(os.path.abspath(__file__))
OBJECTS = sorted(glob.glob(os.path.join(os.path.dirname(HERE), "cel_v3_b200", "_build", "*.o")))
CUDA = "/usr/local/cuda/include"
UNKNOWN = 999  # cudaErrorUnknown

pytestmark = pytest.mark.skipif(not OBJECTS or not shutil.which("g++") or not os.path.isdir(CUDA),
                                reason="needs the library's objects, g++ and the CUDA headers")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libcelgpu_fake.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CUDA, "-o", so,
                           os.path.join(HERE, "c", "fake_cudart.cpp"), *OBJECTS, "-ldl", "-Wl,-Bsymbolic"])
    lib = ctypes.CDLL(so)
    lib.fake_log.restype = ctypes.c_char_p
    return lib


def log(lib):
    return lib.fake_log().decode().splitlines()


def create(lib):
    h = ctypes.c_void_p()
    assert lib.celg_create(ctypes.byref(h), 0, None) == celgpu.OK
    return h


def identity(lib, h, n):
    """A diagonal matrix (its kernels do not run; the arrays are what counts)."""
    m = ctypes.c_void_p()
    rp, ci, v = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n)
    assert lib.celg_mat_from_csr(h, n, n, ctypes.c_void_p(rp.ctypes.data), ctypes.c_void_p(ci.ctypes.data),
                                 ctypes.c_void_p(v.ctypes.data), 0, ctypes.byref(m)) == celgpu.OK
    assert lib.celg_mat_jacobi(m) == celgpu.OK
    return m


def waited_for(lines):
    """Whether the host has waited for every launch in the log: by its stream,
    or by one that waits for an event recorded behind it."""
    done = {}  # stream -> launches not waited for
    events = {}
    for q, line in enumerate(lines):
        w = line.split()
        if w[0].startswith("cudaLaunch"):
            done.setdefault(w[1], set()).add(q)
        elif w[0] == "cudaEventRecord":
            events[w[2]] = set(done.get(w[1], ()))
        elif w[0] == "cudaStreamWaitEvent":
            done.setdefault(w[1], set()).update(events.get(w[2], ()))
        elif w[0] == "cudaStreamSynchronize":
            gone = done.pop(w[1], set())
            for s in done.values():
                s -= gone
    return not any(done.values())


@pytest.mark.parametrize("name", ["cudaLaunchCooperativeKernel", "cudaEventRecord", "cudaStreamWaitEvent"])
def test_batch_that_fails_half_way_leaves_nothing_running(lib, name):
    """Systems of every lane class: whichever call fails, the kernels launched
    before it have ended when the error is returned."""
    sizes = [950000, 600000, 300000, 100000, 90000, 80000]
    lib.fake_fail(b"", 0, 0)
    h = create(lib)
    mats = [identity(lib, h, n) for n in sizes]
    b = [np.ones(n) for n in sizes]
    ptrs = (ctypes.c_void_p * len(sizes))(*[m.value for m in mats])
    vec = (ctypes.c_void_p * len(sizes))(*[a.ctypes.data for a in b])
    p = celgpu.params(eps_rel=1e-8)
    res = (celgpu.Result * len(sizes))()
    lib.fake_int(1)  # the sliced copies are worth it

    def batch(nth):
        lib.fake_clear()
        lib.fake_fail(name.encode(), nth, UNKNOWN)
        st = lib.celg_pcg_batched(h, len(sizes), ptrs, vec, vec, ctypes.byref(p), res)
        return st, log(lib)

    st, lines = batch(0)
    assert st == celgpu.OK and waited_for(lines)
    kernels = [q for q in lines if q.startswith("cudaLaunchCooperative") and "pcg_" in q]
    assert len(kernels) == len(sizes) and len({q.split()[1] for q in kernels}) >= 4
    calls = sum(q.split()[0] == name for q in batch(0)[1])  # (the first batch also tried its grid)
    half_way = 0
    for nth in range(1, calls + 1):
        st, lines = batch(nth)
        assert st == celgpu.ERR_CUDA, nth
        before = any("pcg_" in q for q in lines[:lines.index("fail " + name)])
        half_way += before
        assert waited_for(lines), (nth, lines[-12:])
    assert half_way >= 4
    lib.fake_int(0)
    lib.fake_fail(b"", 0, 0)
    st, lines = batch(0)  # and the handle is usable
    assert st == celgpu.OK
    for m in mats:
        assert lib.celg_mat_destroy(m) == celgpu.OK
    assert lib.celg_destroy(h) == celgpu.OK
