"""The radius beyond which a step is left out of the jet's quadrature, on the CPU.

The trace kernels compare a step's cylindrical radius with jet_f_cut |z|^k in
binary32.  Where the frame gives a jet_f_cut, no point inside the profile's cut-off may
fall outside that, whatever the exponent: a radius that grows like a high power of
the height takes R_base / z_base^k or |z|^k out of binary32's range."""
import ctypes as C
import os

import numpy as np
import pytest

from blackhole_b200 import abi, workloads
from blackhole_b200.build import CHECK_LIB, build_check


@pytest.fixture(scope="module")
def jet_cut():
    if not os.path.exists(CHECK_LIB):
        build_check()
    f = C.CDLL(CHECK_LIB).bhx_jet_cut
    f.argtypes = [C.POINTER(abi.bh_render_config), C.POINTER(C.c_float)]
    return f


@pytest.mark.parametrize("z_base", [0.01, 0.4, 3.0, 50.0, 1e4])
@pytest.mark.parametrize("k", [0.0, 0.58, 1.0, 7.0, 20.0, 60.0, 78.0, 82.0, 100.0, 300.0])
def test_no_point_of_the_jet_is_left_out(jet_cut, z_base, k):
    cfg = workloads.quasar_jets(8, 8)
    j = cfg.jet
    j.z_base, j.z_top, j.R_base, j.k = z_base, 40.0 * z_base, 0.5 * z_base, k
    cfg.jet_enabled = True
    cut = C.c_float(0.0)
    assert jet_cut(C.byref(cfg.to_c()), C.byref(cut)) == abi.OK
    z = j.z_base * np.exp(np.linspace(0.0, np.log(40.0), 400))[:, None]
    with np.errstate(over="ignore", invalid="ignore"):
        # radii up to where the profile is 1e-9 of its peak, in jet radii
        rho = np.linspace(0.0, j.u_peak + 4.5 * j.u_wid, 50)[None, :] * (j.R_base * (z / j.z_base) ** k)
        inside = np.isfinite(rho) & (rho < 1e30)
        kept = (rho.astype(np.float32) < np.float32(cut.value) * z.astype(np.float32) ** np.float32(k)) | (cut.value < 0.0)
    assert inside.any() and kept[inside].all()
    if k <= 1.0:
        assert cut.value > 0.0          # the ordinary jets are cut
