"""The binary32 near-critical test of a mixed frame's rays against binary64, on the CPU.

The test may leave a ray undecided, and it may not decide it otherwise than the
value it stands for: R_min / r*^4 in (-0.1, 0) is traced in binary64, in (-0.2, -0.1]
at a quarter of the tolerances.  Compared ray by ray around the hole's image over
spins, inclinations, rolls, camera distances and directions: with the hole far off
the axis of a wide field the ray's direction is a difference of numbers of order
one, whose rounding in binary32 is 1e-7 of the distance at the hole."""
import ctypes as C
import math
import os
import random

import numpy as np
import pytest

from blackhole_b200 import abi, workloads
from blackhole_b200.build import CHECK_LIB, build_check

I, D = C.POINTER(C.c_int), C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def classes():
    if not os.path.exists(CHECK_LIB):
        build_check()
    f = C.CDLL(CHECK_LIB).bhx_near_critical
    f.argtypes = [C.POINTER(abi.bh_render_config), C.c_int, I, I, I, I, D]
    return f


def _hole(c):
    """The pixel (not rounded) at which the camera of `c` sees the hole's centre."""
    cam, tf, aspect = c.cam, math.tan(0.5 * c.cam.fov), c.width / c.height
    xr, yr = -math.tan(cam.yaw) / math.cos(cam.pitch), math.tan(cam.pitch)
    x = math.cos(cam.roll) * xr + math.sin(cam.roll) * yr
    y = -math.sin(cam.roll) * xr + math.cos(cam.roll) * yr
    return 0.5 * (x / tf + 1.0) * c.width, 0.5 * (1.0 - y * aspect / tf) * c.height


def _compare(classes, c, rng, n=3000):
    """Quick class and R_min / r*^4 of `n` rays around the hole's image."""
    hx, hy = _hole(c)
    S = c.sqrt_spp
    scale = c.width * S / (2.0 * c.cam.r * math.tan(0.5 * c.cam.fov))   # samples per M at the hole
    gx, gy = (np.floor(S * h + scale * rng.normal(0.0, 5.0, n)).astype(np.int64) for h in (hx, hy))
    ok = (gx >= 0) & (gx < c.width * S) & (gy >= 0) & (gy < c.height * S)
    gx, gy = gx[ok], gy[ok]
    px, py, k = (np.ascontiguousarray(v, dtype=np.int32) for v in (gx // S, gy // S, (gy % S) * S + gx % S))
    quick, rn = np.zeros(len(px), np.int32), np.zeros(len(px))
    cc = c.to_c()
    assert classes(C.byref(cc), len(px), px.ctypes.data_as(I), py.ctypes.data_as(I), k.ctypes.data_as(I),
                   quick.ctypes.data_as(I), rn.ctypes.data_as(D)) == abi.OK
    want = np.where((rn < 0.0) & (rn > -0.1), 1, np.where((rn < 0.0) & (rn > -0.2), 2, 0))
    wrong = (quick >= 0) & (quick != want)
    return len(px), int((want > 0).sum()), int((quick >= 0).sum()), wrong, rn


def _scene(spin, deg, r, fov, yaw, pitch, roll, size, spp=1):
    c = workloads.kerr_fp64_256()
    c.spin, c.cam.r, c.cam.theta, c.cam.fov = spin, r, math.radians(deg), fov
    c.cam.yaw, c.cam.pitch, c.cam.roll = yaw, pitch, roll
    c.width = c.height = size
    c.sqrt_spp = spp
    c.precision, c.r_escape, c.stars_enabled, c.star_count = abi.PRECISION_MIXED, 1.1 * r, False, 0
    return c


# (pixels across, samples across a pixel, M per pixel at the hole): a field around
# the hole, and wide fields with the hole anywhere in them
NARROW, WIDE, COARSE = (2048, 1, None), (65536, 1, 0.3), (65536, 64, 15.0)


@pytest.mark.parametrize("field", [NARROW, WIDE, COARSE])
@pytest.mark.parametrize("r", [30.0, 1000.0, 1e4, 5e4, 2e5, 1e6])
def test_quick_class_is_the_binary64_class(classes, r, field):
    size, spp, pixel = field
    pick, rng = random.Random(int(r) + size + spp), np.random.default_rng(int(r) + size + spp)
    rays = near = decided = 0
    for _ in range(24):
        fov = 2.0 * math.atan(min(1.0, 30.0 / r)) if pixel is None else min(1.4, 2.0 * math.atan(pixel * size / (2.0 * r)))
        aim = 5.0 / r if pixel is None else 0.25 * fov
        c = _scene(pick.choice([0.0, 0.5, 0.9, -0.9, 0.998]), pick.choice([5.0, 45.0, 85.0, 90.0, 150.0]), r, fov,
                   pick.uniform(-aim, aim), pick.uniform(-aim, aim), pick.choice([0.0, 0.0, 0.7, 2.0]), size, spp)
        n, k, d, wrong, rn = _compare(classes, c, rng)
        assert not wrong.any(), (c.spin, c.cam, rn[wrong][:5], int(wrong.sum()))
        rays, near, decided = rays + n, near + k, decided + d
    assert rays > 10000 and near > 100
    # it is there to decide: almost every ray of the cameras that programs use
    if field == NARROW or r <= 1e3:
        assert decided > 0.9 * rays, decided / rays
