"""The forms of an integration attempt on the GPU.

  - the binary64 right-hand side against Hamilton's equations written out in
    numpy, for spins on both sides of a = 1 (Delta in factors or not), at
    ordinary angles and where the metric clamps sin(th);
  - frames whose rays pass close to the poles, where a stage can move the angle
    further than angle addition reaches and the attempt takes its general form,
    against the CPU oracle, in both precisions.
"""
import math

import numpy as np
import pytest


from blackhole_b200 import abi  # noqa: E402
from blackhole_b200.config import M_SUN, Camera, RenderConfig  # noqa: E402

pytestmark = pytest.mark.gpu


def _rates(a, y):
    """dy/dlambda of 2 Sigma H = Delta p_r^2 + p_th^2 + (L - a E sin^2)^2 / sin^2 - ((r^2 + a^2) E - a L)^2 / Delta, and
    the sum of the absolute values of each component's terms."""
    r, th, pr, pth, E, L = y[:, 1], y[:, 2], y[:, 5], y[:, 6], -y[:, 4], y[:, 7]
    sn, cs = np.sin(th), np.cos(th)
    sn = np.where(np.abs(sn) < 1e-9, np.where(sn < 0, -1e-9, 1e-9), sn)
    s2 = sn * sn
    S, D = r * r + a * a * cs * cs, r * r - 2 * r + a * a
    w = r * r + a * a
    K, P = w * E - a * L, L - a * E * s2
    B = [D * pr * pr, pth * pth, P * P / s2, -K * K / D]
    Bs, Ba = sum(B), sum(np.abs(b) for b in B)
    rows = [[a * P / S, w * K / (D * S)], [D * pr / S], [pth / S], [P / (s2 * S), a * K / (D * S)],
            [-(r - 1) * pr * pr / S, 2 * r * E * K / (D * S), -(r - 1) * (K / D) ** 2 / S, r * Bs / (S * S)],
            [-sn * cs * a * a * E * E / S, sn * cs * (L / s2) ** 2 / S, -sn * cs * a * a * Bs / (S * S)]]
    value = [sum(t) for t in rows]
    size = [sum(np.abs(t) for t in q) for q in rows]
    size[4] = size[4] + r * Ba / (S * S)
    size[5] = size[5] + np.abs(sn * cs) * a * a * Ba / (S * S)
    return np.stack(value, 1), np.stack(size, 1)


@pytest.mark.parametrize("spin", [0.0, 0.9, -0.7, 0.998, 1.0, 1.2])
def test_binary64_right_hand_side(renderer, spin):
    rng = np.random.default_rng(11)
    n = 257
    y = np.zeros((n, 8))
    y[:, 1] = 2.5 + np.exp(rng.uniform(-2.0, 6.0, n))
    y[:, 2] = rng.uniform(0.05, math.pi - 0.05, n)
    y[:8, 2] = [0.0, 1e-12, math.pi, 1e-4, math.pi - 1e-4, 0.5 * math.pi, 3.0, 0.01]
    y[:, 4] = -rng.uniform(0.5, 1.5, n)
    y[:, 5] = rng.normal(0.0, 1.0, n)
    y[:, 6] = rng.normal(0.0, 6.0, n)
    y[:, 7] = rng.normal(0.0, 6.0, n)
    y[:4, 7] = 0.0
    cfg = RenderConfig(spin=spin, cam=Camera(r=50.0, theta=1.0), width=4, height=4, disc_enabled=False, star_count=0,
                       quiet=True)
    got = renderer.eval(cfg, abi.EVAL_RHS, y)[:, [0, 1, 2, 3, 5, 6]]
    want, size = _rates(spin, y)
    # each term is a product of at most a dozen rounded factors; Delta in the
    # expanded form loses (r^2 + 1) / Delta <= 20 roundings at r >= 2.6, and
    # sin(th) at pi - 1e-4 one part in 1e-4 of an ulp of pi per factor
    tol = 64 * 2.0 ** -53 * (20.0 + np.pi / np.maximum(np.abs(np.sin(y[:, 2])), 1e-9))
    ok = np.abs(got - want) <= tol[:, None] * size
    ok |= np.abs(np.sin(y[:, 2]))[:, None] < 1e-9      # there sin is the clamp's: compared below
    assert ok.all(), np.argwhere(~ok)[:5]
    # where sin(th) is clamped the value is finite (and sign and size are the clamp's)
    clamped = np.abs(np.sin(y[:, 2])) < 1e-9
    assert clamped.sum() >= 3 and np.isfinite(got[clamped]).all()
    assert np.allclose(got[clamped][:, :3], want[clamped][:, :3], rtol=1e-9, atol=0.0)


@pytest.mark.parametrize("theta_deg,spin,precision", [
    (theta, spin, p) for theta, spin in ((0.3, 0.9), (179.6, 0.998), (2.0, 0.0), (90.0, 1.0))
    for p in (abi.PRECISION_FP64, abi.PRECISION_MIXED)
    # at a = 1 the mixed path's captured rays run out of steps: Delta has a
    # double root there, and no hand-over radius
    if not (spin == 1.0 and p == abi.PRECISION_MIXED)])
def test_rays_past_the_poles(renderer, orc, theta_deg, spin, precision):
    cfg = RenderConfig(
        M_kg=4.3e6 * M_SUN, spin=spin,
        cam=Camera(r=40.0, theta=math.radians(theta_deg), phi=0.7, fov=0.9), width=37, height=29, sqrt_spp=1,
        disc_r_out=20.0, rtol=1e-8, atol=1e-10, r_escape=220.0, star_count=0, quiet=True,
    )
    chk, _ = orc.trace_rays(cfg)
    cfg.precision = precision
    got = renderer.trace_rays(cfg)
    same = got["what"] == chk["what"]
    # the suite's bounds for a scene against the oracle: at most two rays of
    # another class; g and direction to 1e-6 (binary64) or the mixed targets
    assert (~same).sum() <= 2
    g_tol, d_tol = (1e-6, 1e-6) if precision == abi.PRECISION_FP64 else (1e-3, 1e-4)
    disc = same & (chk["what"] == abi.HIT_DISC) & (chk["g"] > 0)
    sky = same & (chk["what"] == abi.HIT_SKY)
    assert disc.sum() + sky.sum() > 500
    assert np.quantile(np.abs(got["g"][disc] / chk["g"][disc] - 1.0), 0.95) <= g_tol
    d = np.linalg.norm(got["dir"][sky] - chk["dir"][sky], axis=1)
    assert np.quantile(d, 0.95) <= d_tol


@pytest.mark.parametrize("width,height,jet", [(9, 4, False), (388, 390, False), (389, 390, False), (447, 254, True),
                                              (449, 254, True)])
def test_launch_shape_does_not_change_binary64_frames(width, height, jet):
    """On both sides of the ray counts where the library picks another register
    cap (four and three waves of lanes on 148 SMs), and at a frame of one partial
    warp: the same bits as under the tight cap."""
    from blackhole_b200 import Renderer, workloads

    cfg = workloads.quasar_jets(width, height) if jet else workloads.kerr_fp64_256()
    cfg.width, cfg.height, cfg.star_count = width, height, 20000
    with Renderer(0) as r:
        auto = r.trace_rays(cfg)
        r.set_launch(block_size=128, rays_per_thread=1, refill=32, reg_variant=1, precision=abi.PRECISION_FP64)
        tight = r.trace_rays(cfg)
    for k in ("what", "steps", "attempts", "y", "g", "dir"):
        assert np.array_equal(auto[k], tight[k]), k
    # the jet's sum is rounded by each kernel as it was compiled
    assert np.allclose(auto["jet"], tight["jet"], rtol=1e-11, atol=1e-14 * max(1e-300, tight["jet"].max()))


@pytest.mark.parametrize("centre,radius,fov", [
    ((0.0, 22.0, 0.0), 4.0, 1.2),          # beside the hole
    ((45.0, 5.0, 8.0), 0.3, 0.6),          # a small one close to the camera, between two steps
    ((-400.0, 60.0, 30.0), 40.0, 0.9),     # far behind, where the steps are long
    ((60.0, 0.0, 10.0), 12.0, 0.6),        # the camera just outside it
])
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_no_step_misses_the_sun(renderer, orc, centre, radius, fov, precision):
    """The binary32 test of a step against the Sun leaves out only steps that
    the oracle does not probe either: the same rays end on it (the suite's two
    flips allowed), at the same place."""
    from blackhole_b200.config import SunBody

    cfg = RenderConfig(
        M_kg=4.3e6 * M_SUN, spin=0.6, cam=Camera(r=60.0, theta=math.radians(80.0), phi=0.0, fov=fov, yaw=0.15),
        width=41, height=31, sqrt_spp=1, disc_r_out=20.0, sun_enabled=True, sun=SunBody(centre=centre, radius=radius),
        rtol=1e-9, atol=1e-11, r_escape=600.0, star_count=0, quiet=True,
    )
    chk, _ = orc.trace_rays(cfg)
    cfg.precision = precision
    got = renderer.trace_rays(cfg)
    sun = chk["what"] == abi.HIT_SUN
    assert sun.sum() > 5
    assert ((got["what"] == abi.HIT_SUN) != sun).sum() <= 2
    both = sun & (got["what"] == abi.HIT_SUN)
    tol = 1e-6 if precision == abi.PRECISION_FP64 else 1e-3
    assert np.quantile(np.abs(got["y"][both, 1] / chk["y"][both, 1] - 1.0), 0.95) <= tol


@pytest.mark.parametrize("turns", [1, -1000, 20000, 10 ** 6])
def test_no_step_misses_the_sun_after_many_turns(renderer, turns):
    """The camera's azimuth may be any number: with whole turns added to it the frame
    is the same but for the azimuth's own rounding (10^6 turns: 10^-9 rad), and so
    are its rays that end on a small Sun close to the camera, to two rays as above."""
    from blackhole_b200.config import SunBody

    def frame(phi):
        return renderer.trace_rays(RenderConfig(
            M_kg=4.3e6 * M_SUN, spin=0.6, cam=Camera(r=60.0, theta=math.radians(80.0), phi=phi, fov=0.6, yaw=0.15),
            width=161, height=121, sqrt_spp=1, disc_r_out=20.0, sun_enabled=True,
            sun=SunBody(centre=(45.0, 5.0, 8.0), radius=0.3), rtol=1e-9, atol=1e-11, r_escape=600.0, star_count=0,
            quiet=True))["what"]

    want, got = frame(0.0) == abi.HIT_SUN, frame(2.0 * math.pi * turns) == abi.HIT_SUN
    assert want.sum() > 50
    assert (want != got).sum() <= 2


@pytest.mark.parametrize("spin", [1.0, -1.0, 1.2])
def test_expanded_delta_is_rounded_like_the_reference(renderer, spin):
    """Without a pair of horizons Delta = r^2 - 2 r + a^2, in the reference's
    rounded steps: close to r = 1 at a^2 = 1 what is left is the roundings, and the
    rays that fall in follow it.  From dr / dlambda = Delta p_r / Sigma (a product of
    six rounded factors): Delta is one of the two values that r^2, rounded or
    exact, less 2 r, rounded, plus a^2, rounded, can have."""
    from fractions import Fraction

    rng = np.random.default_rng(5)
    n = 200
    y = np.zeros((n, 8))
    y[:, 1] = 1.0 + np.exp(rng.uniform(math.log(1.5e-8), math.log(3.0), n))
    y[:, 2] = 1.1
    y[:, 4], y[:, 5], y[:, 6], y[:, 7] = -1.0, 1.0, 0.3, 0.5
    cfg = RenderConfig(spin=spin, cam=Camera(r=50.0, theta=1.0), width=4, height=4, disc_enabled=False, star_count=0,
                       quiet=True)
    got = renderer.eval(cfg, abi.EVAL_RHS, y)[:, 1]
    a2 = spin * spin
    cs = math.cos(1.1)
    for r, d in zip(y[:, 1], got):
        exact = float(Fraction(r) ** 2 - 2 * Fraction(r)) + a2
        rounded = float(Fraction(r * r) - 2 * Fraction(r)) + a2
        want = [v / (r * r + a2 * cs * cs) for v in (exact, rounded) if v != 0.0]
        assert not want or min(abs(d / w - 1.0) for w in want) <= 16 * 2.0 ** -53, (r, d, want)


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_a_batch_of_spins_on_both_sides_of_one_equals_its_frames(precision):
    """A launch with a frame of a^2 >= 1 runs other binary64 kernels for all of its
    frames: bit for bit the single frames."""
    from blackhole_b200 import Renderer

    with Renderer(0) as r:
        cfgs = [RenderConfig(M_kg=4.3e6 * M_SUN, spin=s, cam=Camera(r=30.0, theta=th, fov=0.8), width=61, height=37,
                             disc_r_out=20.0, r_escape=60.0, star_count=1000, max_steps=2000, quiet=True,
                             precision=precision)
                for s, th in ((0.9, 1.0), (1.0, 1.2), (0.0, 0.02), (1.2, 0.5), (-0.998, 1.5))]
        batch = r.render_batch(cfgs)
        for c, px in zip(cfgs, batch):
            assert np.array_equal(px, r.render(c), equal_nan=True), c.spin
