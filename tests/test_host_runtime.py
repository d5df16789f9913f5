"""The C-ABI's host side on a fake CUDA runtime (tests/fake_cuda/fake_cuda.cpp).

bh_capi.cpp is compiled as it is and linked with a runtime whose streams are lists
of operations, so that what a driver or a full device does to a call can be made to
happen without a GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from blackhole_b200 import abi, workloads
from blackhole_b200.build import CSRC, INCLUDE

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"

XYZ = C.POINTER(abi.bh_xyz)
CFG = C.POINTER(abi.bh_render_config)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "libbh_fake.so")
    srcs = [os.path.join(HERE, "fake_cuda", "fake_cuda.cpp")] + [
        os.path.join(CSRC, f) for f in ("bh_capi.cpp", "bh_scene.cpp", "bh_adjoint_frame.cpp")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", INCLUDE,
                    "-I", CUDA_INCLUDE, "-o", so] + srcs, check=True)
    lib = C.CDLL(so)
    lib.bh_gpu_create.argtypes = [C.c_int, C.POINTER(C.c_void_p)]
    lib.bh_gpu_destroy.argtypes = [C.c_void_p]
    lib.bh_gpu_destroy.restype = None
    lib.bh_gpu_last_error.argtypes = [C.c_void_p]
    lib.bh_gpu_last_error.restype = C.c_char_p
    lib.bh_gpu_render_batch.argtypes = [C.c_void_p, CFG, C.c_int, C.POINTER(XYZ), C.POINTER(abi.bh_render_stats)]
    lib.fake_fail.argtypes = [C.c_char_p, C.c_int]
    lib.fake_memory.argtypes = [C.c_longlong]
    lib.fake_memory_used.restype = C.c_longlong
    lib.fake_count.argtypes = [C.c_char_p]
    lib.fake_count.restype = C.c_longlong
    return lib


@pytest.fixture
def ctx(lib):
    made = []

    def make():
        h = C.c_void_p()
        assert lib.bh_gpu_create(0, C.byref(h)) == abi.OK
        made.append(h)
        return h

    lib.fake_reset()
    yield make
    lib.fake_reset()
    for h in made:
        lib.bh_gpu_destroy(h)


def _cfg(width, height, precision=abi.PRECISION_MIXED):
    c = workloads.kerr_fp64_256()
    c.width, c.height, c.precision, c.star_count = width, height, precision, 100
    return c


class Batch:
    """Arguments of bh_gpu_render_batch over the frames `sizes` ((height, width))."""

    def __init__(self, sizes, precision=abi.PRECISION_MIXED):
        self.n = len(sizes)
        self.c = (abi.bh_render_config * self.n)(*[_cfg(w, h, precision).to_c() for h, w in sizes])
        self.px = [np.full((h, w, 3), -1.0) for h, w in sizes]
        self.ptr = (XYZ * self.n)(*[p.ctypes.data_as(XYZ) for p in self.px])
        self.stats = (abi.bh_render_stats * self.n)()

    def render(self, lib, h):
        return lib.bh_gpu_render_batch(h, self.c, self.n, self.ptr, self.stats)

    def whole(self):
        return all(np.array_equal(p[..., 1].reshape(-1), np.arange(p.shape[0] * p.shape[1])) for p in self.px) and all(
            s.rays == p.shape[0] * p.shape[1] for s, p in zip(self.stats, self.px))


EARLY = [(300, 500), (256, 513)]       # binary32 frames that are shaded and copied while the rest is traced


@pytest.mark.parametrize("missing", ["nothing", "wait_value", "event"])
def test_batch_without_what_the_row_bands_need(lib, ctx, missing):
    """A driver without stream waits on a value leaves the row-band pipeline out;
    the batch does not use them, and is whole.  Where an event cannot be made the batch
    takes the graph."""
    if missing == "wait_value":
        lib.fake_without_wait_value(1)
    h = ctx()
    if missing == "event":
        lib.fake_fail(b"cudaEventCreateWithFlags", 1)
    b = Batch(EARLY)
    assert b.render(lib, h) == abi.OK, lib.bh_gpu_last_error(h)
    assert b.whole()
    assert lib.fake_count(b"cudaGraphLaunch") == (missing == "event")
    assert lib.fake_outstanding_copies() == 0
