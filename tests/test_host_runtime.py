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
    S, U8, D = C.POINTER(abi.bh_render_stats), C.POINTER(C.c_uint8), C.POINTER(C.c_double)
    lib.bh_gpu_render.argtypes = [C.c_void_p, CFG, XYZ, S]
    lib.bh_gpu_trace_rays.argtypes = [C.c_void_p, CFG, C.POINTER(abi.bh_ray_result), S]
    lib.bh_gpu_render_rgb.argtypes = [C.c_void_p, CFG, C.POINTER(abi.bh_display), U8, D, S]
    lib.bh_gpu_render_batch_rgb.argtypes = [C.c_void_p, CFG, C.c_int, C.POINTER(abi.bh_display), C.POINTER(U8), D, S]
    lib.bh_gpu_develop.argtypes = [C.c_void_p, XYZ, C.c_int, C.c_int, C.POINTER(abi.bh_display), U8, D]
    lib.bh_gpu_adjoint_rays.argtypes = [C.c_void_p, CFG, C.POINTER(C.c_float), C.POINTER(abi.bh_grad4), D, D]
    lib.bh_gpu_eval.argtypes = [C.c_void_p, CFG, C.c_int, D, C.c_longlong, D]
    lib.bh_display_default.argtypes = [C.POINTER(abi.bh_display)]
    lib.bh_display_default.restype = None
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


def _calls(lib):
    """Every entry that copies into the caller's memory, as a function of the context."""
    d = abi.bh_display()
    lib.bh_display_default(C.byref(d))
    d.glare = 0.3
    u8, dp = C.POINTER(C.c_uint8), C.POINTER(C.c_double)
    small, tall, adj = _cfg(40, 30).to_c(), _cfg(60, 300).to_c(), _cfg(24, 20, abi.PRECISION_FP64).to_c()
    px = np.zeros((300, 60, 3))
    rays = np.zeros(40 * 30, dtype=abi.ray_result_dtype())
    rgb = [np.zeros((30, 40, 3), np.uint8) for _ in range(9)]
    developed = np.zeros((300, 60, 3), np.uint8)
    film = (abi.bh_render_config * 9)(*[small] * 9)
    films = (u8 * 9)(*[a.ctypes.data_as(u8) for a in rgb])
    ex, grad, lum, rhs = np.zeros(9), np.zeros((480, 4)), np.zeros(480), np.ones((5, 8))
    target, g = np.zeros((20, 24), np.float32), abi.bh_grad4()
    early, graph = Batch(EARLY), Batch([(30, 40), (20, 25)])
    p = lambda a, t: a.ctypes.data_as(t)  # noqa: E731
    return {
        "render": lambda h: lib.bh_gpu_render(h, C.byref(small), p(px, XYZ), None),
        "render in row bands": lambda h: lib.bh_gpu_render(h, C.byref(tall), p(px, XYZ), None),
        "trace_rays": lambda h: lib.bh_gpu_trace_rays(h, C.byref(small), p(rays, C.POINTER(abi.bh_ray_result)), None),
        "batch": lambda h: early.render(lib, h),
        "batch as a graph": lambda h: graph.render(lib, h),
        "develop": lambda h: lib.bh_gpu_develop(h, p(px, XYZ), 60, 300, C.byref(d), p(developed, u8), p(ex, dp)),
        "render_rgb": lambda h: lib.bh_gpu_render_rgb(h, C.byref(small), C.byref(d), p(rgb[0], u8), p(ex, dp), None),
        "film": lambda h, alive=rgb: lib.bh_gpu_render_batch_rgb(h, film, 9, C.byref(d), films, p(ex, dp), None),
        "adjoint": lambda h: lib.bh_gpu_adjoint_rays(h, C.byref(adj), p(target, C.POINTER(C.c_float)), C.byref(g),
                                                     p(grad, dp), p(lum, dp)),
        "eval": lambda h: lib.bh_gpu_eval(h, C.byref(small), abi.EVAL_RHS, p(rhs, dp), 5, p(rhs, dp)),
    }


FAILING = ["cudaMemcpyAsync", "cudaMemcpy2DAsync", "cudaMemsetAsync", "cudaEventRecord", "cudaStreamWaitEvent",
           "cudaStreamSynchronize", "cuStreamWaitValue32", "cudaGraphLaunch", "launch_trace", "launch_shade",
           "launch_reduce", "launch_display", "launch_adjoint"]


@pytest.mark.parametrize("call", ["render", "render in row bands", "trace_rays", "batch", "batch as a graph", "develop",
                                  "render_rgb", "film", "adjoint", "eval"])
def test_no_copy_into_the_callers_memory_outlives_a_failed_call(lib, ctx, call):
    """Whichever runtime call fails, an entry returns an error with nothing under way
    into memory that the caller may free, and the next call is whole."""
    h = ctx()
    run = _calls(lib)[call]
    assert run(h) == abi.OK, lib.bh_gpu_last_error(h)
    assert lib.fake_outstanding_copies() == 0
    failed = 0
    for name in FAILING:
        for nth in range(1, 200):
            lib.fake_reset()
            lib.fake_fail(name.encode(), nth)
            rc = run(h)
            assert lib.fake_outstanding_copies() == 0, (name, nth)
            lib.fake_reset()
            if rc == abi.OK:
                break
            failed += 1
        assert run(h) == abi.OK, (name, lib.bh_gpu_last_error(h))
    assert failed > 3


MB = 1 << 20


def _gradient(lib, h, n):
    """bh_gpu_adjoint_rays of an n x n frame."""
    c, g = _cfg(n, n, abi.PRECISION_FP64).to_c(), abi.bh_grad4()
    target, d = np.zeros(n * n, np.float32), np.zeros(4 * n * n)
    dp = d.ctypes.data_as(C.POINTER(C.c_double))
    return lib.bh_gpu_adjoint_rays(h, C.byref(c), target.ctypes.data_as(C.POINTER(C.c_float)), C.byref(g), dp, None)


def test_a_gradient_needs_no_more_than_its_rays(lib, ctx):
    """Records and stored states shrink to the memory there is: a gradient of 128^2 rays
    needs about 200 bytes a ray, whatever it takes on an empty device."""
    h = ctx()
    assert _gradient(lib, h, 8) == abi.OK            # the sky's tables
    lib.fake_memory(lib.fake_memory_used() + 16 * MB)
    assert _gradient(lib, h, 128) == abi.OK, lib.bh_gpu_last_error(h)


def test_what_a_gradient_keeps_is_given_back(lib, ctx):
    """A context that holds a gradient's record (0.94 GB at 128^2 x 512 steps) takes it
    back before another call fails for want of memory."""
    h = ctx()
    assert _gradient(lib, h, 128) == abi.OK
    held = lib.fake_memory_used()
    assert held > 400 * MB
    lib.fake_memory(held + MB)
    b = Batch([(600, 700), (500, 400)], abi.PRECISION_FP64)
    assert b.render(lib, h) == abi.OK, lib.bh_gpu_last_error(h)
    assert b.whole()
    lib.fake_memory(-1)
    assert _gradient(lib, h, 128) == abi.OK


def test_memory_of_a_gradient(lib, ctx):
    """The figures of bh_gpu.h: 7.5 GB of records and 0.2 GB of stored states at 512^2."""
    h = ctx()
    assert _gradient(lib, h, 8) == abi.OK
    before = lib.fake_memory_used()
    assert _gradient(lib, h, 512) == abi.OK
    used = (lib.fake_memory_used() - before) / 1e9
    assert 7.5 < used < 7.9
