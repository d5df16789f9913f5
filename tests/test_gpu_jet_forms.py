"""The jet's emission on the GPU against the CPU oracle over jet models at the
edges of the step test: radii that grow, stay or shrink with height, a sheath
wide enough to reach the bounding sphere, a base inside the ISCO, no spine, and
an index with which g does not matter.

The per-ray sums agree to the suite's binary64 bound (1e-6, 95th percentile);
a step wrongly left out would show as a ray without light, or in the frame's
sum, which is held to 1e-8: the rays differ by roundings alone, about 1e-12 per
ray, except where a hit's position is amplified near the photon shell."""
import numpy as np
import pytest

from blackhole_b200 import abi, workloads

pytestmark = pytest.mark.gpu

MODELS = {
    "quasar": dict(),
    "cylinder": dict(k=0.0, R_base=6.0),
    "narrowing": dict(k=-0.3, R_base=6.0),
    "fat": dict(R_base=8.0, u_wid=0.6),
    "low base": dict(z_base=0.4, R_base=0.8),
    "no spine": dict(spine=0.0, u_wid=0.08),
    "wide spine": dict(spine=0.8, spine_wid=1.5),
    "flat index": dict(alpha=-2.0, zeta=0.0),
}


@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_jet_sum_against_oracle(renderer, orc, name, precision):
    cfg = workloads.quasar_jets(41, 23)
    for k, v in MODELS[name].items():
        setattr(cfg.jet, k, v)
    cfg.setup_jet()
    assert cfg.jet_enabled
    cfg.r_escape = max(cfg.r_escape, 1.5 * cfg.jet.r_bound)
    cfg.star_count = 0
    chk, _ = orc.trace_rays(cfg)
    cfg.precision = precision
    got = renderer.trace_rays(cfg)
    same = got["what"] == chk["what"]
    assert (~same).sum() <= 2
    want, have = np.asarray(chk["jet"])[same], got["jet"][same]
    lit = want > 0.0
    assert lit.sum() > 50
    peak = want.max()
    # light where the oracle has light, and none where it has none
    assert (have[want > 1e-12 * peak] > 0.0).all() and (have[~lit] <= 1e-12 * peak).all()
    if precision == abi.PRECISION_FP64:
        assert np.quantile(np.abs(have[lit] / want[lit] - 1.0), 0.95) <= 1e-6
        assert abs(have.sum() / want.sum() - 1.0) <= 1e-8
    else:
        # the mixed path steps differently: the quadrature's own error
        assert abs(have.sum() / want.sum() - 1.0) <= 2e-2
