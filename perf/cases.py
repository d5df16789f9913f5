"""The work a user of this library has it do, as measurable cases.

A case is a dict of plain values.  ``kind`` names the entry point's job:

  frame    one image through Renderer.render / render_into / render_device
  batch    frames of uneven size in one launch, Renderer.render_batch
  film     an animation to 8-bit sRGB, Renderer.render_batch_rgb
  adjoint  loss and gradient of a frame, autograd.luminance_loss

``listed()`` is the set that stands for the range, ``draw(rng)`` another case
of it.  Inputs (camera, hole, disc) are made from the seed around the scene
the case names; the sky (catalogue seed and size) stays the same from frame to
frame, as it does in a program that moves a camera through one sky.

Outputs are the images and the counts of what the rays ended on.  The counters
of how the work was done (steps, attempts, drift maxima, times, bytes copied)
are not part of the result.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from blackhole_b200 import Renderer, RenderStats, abi, autograd, workloads
from blackhole_b200.config import M_SUN, Camera, HotSpot, NeutronStar, RenderConfig, SunBody

STARS = 250000          # the library's default catalogue
SKY_SEED = 20240921

_renderer = None


def renderer() -> Renderer:
    """The one context a program keeps for the life of the process."""
    global _renderer
    if _renderer is None:
        _renderer = Renderer(0)
    return _renderer


# ---- the cases -----------------------------------------------------------------
def _frame(name, scene, precision, width, height, spp=1, entry="render", sky="uniform", **kw):
    c = dict(kind="frame", scene=scene, precision=precision, width=width, height=height, spp=spp, entry=entry, sky=sky,
             spin=0.9, incl=60.0, r_cam=1000.0, half=25.0, r_out=30.0, edd=0.1, mass=4.3e6, sense=1, roll=0.0,
             rtol=1e-8)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # an interactive preview while a scene is being set up: the smallest
        # frame, an odd number of columns, in the fast precision
        _frame("preview_161x90_mixed", "kerr", "mixed", 161, 90),
        # the plain binary64 frame of the package's own workloads
        _frame("kerr_256_fp64", "kerr", "fp64", 256, 256),
        # the headline frame, kept on the GPU for a torch program
        _frame("edge_on_1024_mixed", "kerr", "mixed", 1024, 1024, entry="device", spin=0.998, incl=85.0, r_out=50.0,
               edd=0.3, mass=10.0),
        # the same in the reference's arithmetic, into the caller's pinned host image
        _frame("edge_on_1024_fp64", "kerr", "fp64", 1024, 1024, entry="into", spin=0.998, incl=85.0, r_out=50.0,
               edd=0.3, mass=10.0),
        # a user who sets nothing: the reference's default camera, sky,
        # tolerances and four samples per pixel, at a quarter of its pixels
        _frame("default_640x360_spp2_fp64", "kerr", "fp64", 640, 360, spp=2, sky="galactic", incl=90.0, r_cam=60.0,
               half=18.6, r_out=24.0, mass=10.0, rtol=1e-9),
        # a close-up of the photon ring: the largest frame, dense in rays that
        # circle the hole
        _frame("photon_ring_2048_mixed", "ring", "mixed", 2048, 2048, entry="device", spin=0.998, incl=75.0, half=8.0,
               r_out=100.0, edd=0.5, mass=6.5e9),
        # the command line's jet presets: the reference's arithmetic at preview
        # size and the fast precision at film size
        _frame("quasar_jets_320x180_fp64", "quasar", "fp64", 320, 180, sky="galactic"),
        _frame("m87_jets_1024x576_mixed", "m87", "mixed", 1024, 576, sky="galactic", entry="into"),
        # the Sun beside the hole, an orbiting hot spot, four samples per
        # pixel, a ragged image
        _frame("sun_hotspot_333x217_fp64", "sun", "fp64", 333, 217, spp=2, sky="galactic", incl=80.0, r_cam=60.0,
               half=32.8, r_out=24.0, rtol=1e-9),
        # a parameter survey: uneven frames in one launch
        dict(name="survey_16_frames_mixed", kind="batch", precision="mixed", frames=16, sizes="256,512,1024"),
        # a hot-spot film as the command line makes it, glared, at the
        # exposure metered on its probe frame
        dict(name="film_24x512x288_mixed", kind="film", precision="mixed", frames=24, width=512, height=288, glare=0.2,
             glare_radius=3.0, metered=False),
        # one step of fitting spin, inclination, accretion rate and disc size
        # to an observed image
        dict(name="adjoint_512", kind="adjoint", width=512, height=512, spp=1, spin=0.7, incl=50.0, r_out=25.0,
             edd=0.2, stars=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["jet", "jet", "surface", "surface", "batch", "film", "adjoint", "adjoint"])
    precision = rng.choice(["fp64", "mixed"])
    aspect = rng.choice([1.0, 4.0 / 3.0, 16.0 / 9.0])
    if kind == "batch":
        return dict(kind="batch", precision=precision, frames=rng.randint(2, 12),
                    sizes=",".join(str(int(_log(rng, 96, 640))) for _ in range(3)))
    if kind == "film":
        w = int(_log(rng, 128, 640))
        return dict(kind="film", precision=precision, frames=rng.randint(4, 12), width=w, height=max(36, int(w / aspect)),
                    glare=rng.choice([0.0, 0.2, 0.5]), glare_radius=round(rng.uniform(1.0, 4.0), 2),
                    metered=rng.random() < 0.5)
    if kind == "adjoint":
        w = int(_log(rng, 96, 448))
        return dict(kind="adjoint", width=w, height=max(36, int(w / aspect)), spp=1 if w > 200 else rng.choice([1, 2]),
                    spin=round(rng.uniform(0.0, 0.95), 3), incl=round(rng.uniform(15.0, 80.0), 1),
                    r_out=round(rng.uniform(15.0, 40.0), 1), edd=round(_log(rng, 0.01, 0.5), 4),
                    stars=rng.random() < 0.5)
    entry = rng.choice(["render", "into", "device"])
    if kind == "jet":
        w = int(_log(rng, 128, 640))
        return _frame(None, rng.choice(["quasar", "m87"]), precision, w, max(36, int(w / aspect)), sky="galactic",
                      entry=entry)
    spp = rng.choice([1, 1, 1, 2])
    w = int(_log(rng, 96, (700 if precision == "fp64" else 1400) / spp))
    common = dict(spin=rng.choice([0.0, 0.5, 0.9, 0.998, round(rng.uniform(-0.95, 0.95), 3)]),
                  sense=rng.choice([1, 1, 1, -1]), edd=round(_log(rng, 1e-3, 0.5), 5), r_out=round(rng.uniform(12.0, 60.0), 1),
                  mass=float("%.3g" % _log(rng, 5.0, 1e9)), roll=rng.choice([0.0, 0.0, 0.2]), rtol=rng.choice([1e-8, 1e-9]),
                  sky=rng.choice(["uniform", "galactic"]))
    if kind == "surface":
        scene = rng.choice(["sun", "neutron"])
        w = min(w, 500 // spp)
        r_cam = round(rng.uniform(50.0, 90.0), 1)
        return _frame(None, scene, precision, w, max(36, int(w / aspect)), spp=spp, entry=entry, r_cam=r_cam,
                      half=round(r_cam * rng.uniform(0.15, 0.5), 2), incl=round(rng.uniform(30.0, 85.0), 1), **common)
    r_cam = round(_log(rng, 50.0, 2000.0), 1)
    return _frame(None, "kerr", precision, w, max(36, int(w / aspect)), spp=spp, entry=entry, r_cam=r_cam,
                  half=round(rng.uniform(8.0, 30.0), 2), incl=round(rng.uniform(8.0, 88.0), 1), **common)


# ---- inputs --------------------------------------------------------------------
def _precision(case):
    return abi.PRECISION_MIXED if case["precision"] == "mixed" else abi.PRECISION_FP64


def _frame_config(case, seed) -> RenderConfig:
    rng = random.Random(1000003 * int(seed) + 17)
    s, prec, w, h = case["scene"], _precision(case), case["width"], case["height"]
    turn, tilt = rng.uniform(0.0, 2.0 * math.pi), math.radians(rng.uniform(-1.0, 1.0))
    if s in ("quasar", "m87"):
        cfg = (workloads.quasar_jets if s == "quasar" else workloads.m87_jets)(w, h, prec)
        cfg.cam.phi = turn
        cfg.cam.theta += tilt
        cfg.sqrt_spp = case["spp"]
        return cfg
    cfg = RenderConfig(
        M_kg=case["mass"] * M_SUN, spin=case["spin"],
        cam=Camera(r=case["r_cam"] * rng.uniform(0.98, 1.02), theta=math.radians(case["incl"]) + tilt, phi=turn,
                   fov=2.0 * math.atan(case["half"] / case["r_cam"]), roll=case["roll"]),
        width=w, height=h, sqrt_spp=case["spp"], disc_r_out=case["r_out"], disc_sense=case["sense"],
        eddington=case["edd"] * rng.uniform(0.9, 1.1), star_count=STARS, seed=SKY_SEED,
        rtol=case["rtol"], atol=0.01 * case["rtol"], r_escape=1.1 * 1.02 * case["r_cam"], quiet=True, precision=prec,
    )
    if case["sky"] == "uniform":
        cfg.sky_mode, cfg.stop_mode, cfg.stop_epsilon = abi.SKY_UNIFORM, abi.STOP_RELATIVE, 1e-6
    if case["r_cam"] < 100.0:
        cfg.r_escape = 3.0 * case["r_cam"] + 100.0      # the command line's escape sphere
    if s == "ring":
        edge = workloads.critical_curve_prograde_edge(case["spin"], math.radians(case["incl"]))
        cfg.cam.yaw = math.atan(edge / case["r_cam"])
    if s == "sun":
        cfg.cam.phi, cfg.cam.yaw = 0.0, rng.uniform(0.1, 0.2)
        cfg.sun_enabled = True
        cfg.sun = SunBody(centre=(0.0, rng.uniform(20.0, 24.0), 0.0), radius=4.0)
        cfg.hotspot = HotSpot(enabled=True, phi0=rng.uniform(0.0, 6.0))
        cfg.hotspot.set_spin(cfg.spin, cfg.disc_sense)
        cfg.observer_time = rng.uniform(0.0, 80.0)
    if s == "neutron":
        cfg.spin, cfg.disc_enabled = 0.0, False
        cfg.star = NeutronStar(enabled=True, Omega=0.01, caps=True, cap_phase0=rng.uniform(0.0, 6.0))
        cfg.observer_time = rng.uniform(0.0, 80.0)
    return cfg


def _batch_configs(case, seed):
    rng = random.Random(1000003 * int(seed) + 29)
    sizes = [int(v) for v in case["sizes"].split(",")]
    out = []
    for i in range(case["frames"]):
        r_cam = rng.uniform(500.0, 2000.0)
        n = sizes[i % len(sizes)]
        out.append(_frame_config(_frame(None, "kerr", case["precision"], n, n, spin=(0.0, 0.5, 0.9, 0.998)[i % 4],
                                        incl=(15.0, 45.0, 70.0, 85.0)[(i // 4) % 4], r_cam=r_cam), rng.randrange(1 << 30)))
    random.Random(5).shuffle(out)      # uneven sizes in no order, the same for every seed
    return out


def _film_configs(case, seed):
    rng = random.Random(1000003 * int(seed) + 41)
    film = workloads.hotspot_orbit(frames=case["frames"], width=case["width"], height=case["height"],
                                   precision=_precision(case))
    tilt, start = math.radians(rng.uniform(-2.0, 2.0)), rng.uniform(0.0, 6.0)
    for c in film:
        c.cam.theta += tilt
        c.hotspot.phi0 = start
    return film


def prepare(case, seed):
    r = renderer()
    state = {"case": case, "r": r}
    if case["kind"] == "frame":
        cfg = state["cfg"] = _frame_config(case, seed)
        shape = (cfg.height, cfg.width, 3)
        if case["entry"] == "device":
            state["out"] = torch.empty(shape, dtype=torch.float64, device="cuda")
        elif case["entry"] == "into":
            state["pinned"] = torch.empty(shape, dtype=torch.float64, pin_memory=True)
            state["out"] = state["pinned"].numpy()
    elif case["kind"] == "batch":
        cfgs = state["cfgs"] = _batch_configs(case, seed)
        state["pinned"] = [torch.empty((c.height, c.width, 3), dtype=torch.float64, pin_memory=True) for c in cfgs]
        state["outs"] = [t.numpy() for t in state["pinned"]]
    elif case["kind"] == "film":
        film = state["cfgs"] = _film_configs(case, seed)
        exposure = 0.0
        if not case["metered"]:
            # the exposure a film is locked to, metered once on its probe frame
            # (the film's own sky, so that it is not rebuilt between the two)
            probe = workloads.exposure_probe(film[len(film) // 2])
            probe.star_count = film[0].star_count
            exposure = r.render_rgb(probe, meter_only=True)[1]
        state["display"] = r.display_settings(exposure=exposure, glare=case["glare"], glare_radius=case["glare_radius"])
    else:
        rng = random.Random(1000003 * int(seed) + 53)
        cfg = workloads.adjoint_512()
        cfg.width, cfg.height, cfg.sqrt_spp, cfg.stars_enabled = case["width"], case["height"], case["spp"], case["stars"]
        cfg.spin, cfg.cam.theta = case["spin"], math.radians(case["incl"] + rng.uniform(-1.0, 1.0))
        cfg.cam.phi = rng.uniform(0.0, 2.0 * math.pi)
        cfg.disc_r_out, cfg.eddington = case["r_out"], case["edd"]
        seen = cfg.replace(spin=min(0.97, cfg.spin + 0.04), eddington=1.1 * cfg.eddington, disc_r_out=1.08 * cfg.disc_r_out)
        seen.cam.theta += math.radians(2.0)
        state["cfg"] = cfg
        state["target"] = torch.from_numpy(r.render(seen)[..., 1].astype(np.float32))
        state["params"] = torch.tensor([cfg.spin, cfg.cam.theta, cfg.eddington, cfg.disc_r_out], dtype=torch.float64,
                                       requires_grad=True)
    return state


# ---- one pass ------------------------------------------------------------------
def _ends(st):
    return [st.rays, st.captured, st.disc_hits, st.sun_hits, st.star_hits, st.jet_rays, st.escaped, st.exhausted]


def run(state):
    case, r = state["case"], state["r"]
    if case["kind"] == "frame":
        if case["entry"] == "device":
            r.render_device(state["cfg"], state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
            return {"xyz": state["out"]}
        if case["entry"] == "into":
            st = abi.bh_render_stats()
            r.render_into(state["cfg"], state["out"], st)
            return {"xyz": state["out"], "ends": _ends(st), "flux": st.total_flux}
        st = RenderStats()
        xyz = r.render(state["cfg"], st)
        return {"xyz": xyz, "ends": _ends(st), "flux": st.total_flux}
    if case["kind"] == "batch":
        stats = []
        return {"xyz": r.render_batch(state["cfgs"], stats, state["outs"]), "ends": [_ends(s) for s in stats][:4]}
    if case["kind"] == "film":
        rgb, exposure = r.render_batch_rgb(state["cfgs"], state["display"])
        return {"rgb": rgb, "exposure": exposure if case["metered"] else exposure[0]}
    p = state["params"]
    p.grad = None
    loss = autograd.luminance_loss(p, state["target"], state["cfg"], r)
    loss.backward()
    return {"loss": loss.detach(), "grad": p.grad}


# ---- what a pass cannot do without -----------------------------------------------
def work(case):
    """Bytes: constants in, images out.  Operations: the accepted Dormand-Prince
    steps (957 operations each in binary64, 887 in binary32, as flops.py counts
    them) times the steps a ray takes in that precision (about 165 under the
    reference's step cap, 51 under the mixed path's)."""
    def ray_flops(precision):
        return 165 * 957.0 if precision == "fp64" else 51 * 887.0

    sky = 250000 * 64.0
    if case["kind"] == "frame":
        px = case["width"] * case["height"]
        capped = case["scene"] in ("quasar", "m87", "sun", "neutron")
        per_ray = 165 * (957.0 if case["precision"] == "fp64" else 887.0) if capped else ray_flops(case["precision"])
        if case["scene"] in ("quasar", "m87"):
            per_ray += 100 * 4 * 250.0      # the jet's quadrature along the steps near it
        return {"bytes": px * 24.0 + sky, "flops": px * case["spp"] ** 2 * per_ray}
    if case["kind"] == "batch":
        sizes = [int(v) for v in case["sizes"].split(",")]
        px = sum(sizes[i % len(sizes)] ** 2 for i in range(case["frames"]))
        return {"bytes": px * 24.0 + sky, "flops": px * ray_flops(case["precision"])}
    px = case["width"] * case["height"]
    if case["kind"] == "film":
        px *= case["frames"]
        taps = 4 * 3.0 * case["glare_radius"] * 4 + 4 if case["glare"] > 0 else 0.0
        return {"bytes": px * 3.0 + sky, "flops": px * (ray_flops(case["precision"]) + taps * 6)}
    # forward once, then the stages and their vector-Jacobian products backwards
    return {"bytes": px * 4.0 + sky, "flops": px * case["spp"] ** 2 * 165 * 957.0 * 4}


# ---- the same images in plain torch, binary64 --------------------------------------
PI = math.pi
CUT_RAYS = 1100000


def exact(case, seed):
    """A frame of a hole, its disc and the uniform sky, by the published scheme
    (Dormand-Prince 5(4) with PI step control and dense output on Hamilton's
    equations, Page-Thorne disc, Planck spectra under the CIE fit of Wyman et
    al.), in binary64 torch operations.  Other scenes, and frames too large for
    a few seconds, have no such value here."""
    if case["kind"] != "frame" or case["scene"] not in ("kerr", "ring") or case["sky"] != "uniform":
        return None
    if case["width"] * case["height"] * case["spp"] ** 2 > CUT_RAYS:
        return None
    xyz = _plain_frame(_frame_config(case, seed))
    if case["entry"] == "device":
        return {"xyz": xyz}
    return {"xyz": xyz, "ends": None, "flux": float(xyz[..., 1].sum())}


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _uniform(s0, k):
    """Draw k (from 1) of the splitmix64 stream of seed s0."""
    with np.errstate(over="ignore"):
        return (_mix(s0 + np.uint64(0x9E3779B97F4A7C15) * np.asarray(k, dtype=np.uint64)) >> np.uint64(11)) * 2.0 ** -53


def _lower(a, r, th):
    """g_tt, g_tphi, g_rr, g_thth, g_phiphi of Kerr in Boyer-Lindquist coordinates, and Sigma, Delta, A."""
    sn2, cs2 = math.sin(th) ** 2, math.cos(th) ** 2
    S, D = r * r + a * a * cs2, r * r - 2 * r + a * a
    A = (r * r + a * a) ** 2 - a * a * D * sn2
    return -(1 - 2 * r / S), -2 * a * r * sn2 / S, S / D, S, A * sn2 / S, S, D, A


def _photons(cfg):
    """(p_t, p_r, p_th, p_phi) of every sample's photon, pixel by pixel."""
    W, H, n = cfg.width, cfg.height, max(1, cfg.sqrt_spp)
    py, px, k = np.meshgrid(np.arange(H), np.arange(W), np.arange(n * n), indexing="ij")
    with np.errstate(over="ignore"):
        s0 = np.uint64(cfg.seed) ^ (py.astype(np.uint64) << np.uint64(32)) ^ (px.astype(np.uint64) * np.uint64(0x9E3779B97F4A7C15))
    jx = (k % n + _uniform(s0, 2 * k + 1)) / n
    jy = (k // n + _uniform(s0, 2 * k + 2)) / n
    t = math.tan(0.5 * cfg.cam.fov)
    x, y = (2 * (px + jx) / W - 1) * t, (1 - 2 * (py + jy) / H) * t / (W / H)
    c, s = math.cos(cfg.cam.roll), math.sin(cfg.cam.roll)
    x, y = c * x - s * y, s * x + c * y
    c, s = math.cos(cfg.cam.pitch), math.sin(cfg.cam.pitch)
    y, z = c * y - s, s * y + c
    c, s = math.cos(cfg.cam.yaw), math.sin(cfg.cam.yaw)
    x, z = c * x + s * z, -s * x + c * z
    d = np.stack([-z, -y, x]).reshape(3, -1)
    d /= np.sqrt((d * d).sum(0))
    a, r, th = cfg.spin, cfg.cam.r, cfg.cam.theta
    tt, tp, rr, hh, pp, S, D, A = _lower(a, r, th)
    lapse, drag = math.sqrt(S * D / A), 2 * a * r / A
    p0 = np.full(d.shape[1], -1 / lapse)
    p1, p2 = d[0] * math.sqrt(D / S), d[1] / math.sqrt(S)
    p3 = -drag / lapse + d[2] * math.sqrt(S / A) / math.sin(th)
    return np.stack([tt * p0 + tp * p3, rr * p1, hh * p2, tp * p0 + pp * p3])


def _rates(y, E, L, a):
    """Hamilton's equations; y = (t, r, th, phi, p_r, p_th)."""
    r, th, pr, ph = y[1], y[2], y[4], y[5]
    sn, cs = torch.sin(th), torch.cos(th)
    sn = torch.where(sn.abs() < 1e-9, torch.where(sn < 0, -1e-9, 1e-9).to(sn), sn)
    s2 = sn * sn
    S = r * r + a * a * cs * cs
    D = (r - (1 + math.sqrt(1 - a * a))) * (r - (1 - math.sqrt(1 - a * a)))
    w = r * r + a * a
    K, P = w * E - a * L, L - a * E * s2
    KD = K / D
    B = D * pr * pr + ph * ph + P * P / s2 - K * KD
    return torch.stack([
        (a * P + w * KD) / S, D * pr / S, ph / S, (P / s2 + a * KD) / S,
        -0.5 / S * ((2 * r - 2) * (pr * pr + KD * KD) - 4 * r * E * KD - 2 * r * B / S),
        -sn * cs / S * (a * a * E * E - L * L / (s2 * s2) + a * a * B / S)])


_A = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
      (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
      (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
      (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
_LOW = (5179 / 57600, 0.0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40)
_DENSE = (-12715105075 / 11282082432, 0.0, 87487479700 / 32700410799, -10690763975 / 1880347072,
          701980252875 / 199316789632, -1453857185 / 822651844, 69997945 / 29380423)


def _weighted(k, w):
    out = None
    for q, v in zip(k, w):
        if v:
            out = v * q if out is None else out + v * q
    return out


def _dense(y0, y1, k, h, s):
    """The fourth-order continuous extension at fraction s of the step."""
    r2 = y1 - y0
    r3 = h * k[0] - r2
    r4 = r2 - h * k[6] - r3
    return y0 + s * (r2 + (1 - s) * (r3 + s * (r4 + (1 - s) * h * _weighted(k, _DENSE))))


def _isco(a, sense):
    z1 = 1 + (1 - a * a) ** (1 / 3) * ((1 + a) ** (1 / 3) + (1 - a) ** (1 / 3))
    z2 = math.sqrt(3 * a * a + z1 * z1)
    return 3 + z2 - sense * math.sqrt(max(0.0, (3 - z1) * (3 + z1 + 2 * z2)))


def _plain_frame(cfg):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    a = cfg.spin
    p = torch.from_numpy(_photons(cfg)).to(dev)
    n = p.shape[1]
    r_h, r_in = 1 + math.sqrt(1 - a * a), _isco(a, cfg.disc_sense)
    r_out, r_stop = max(cfg.disc_r_out, 1.02 * r_in), r_h * (1 + cfg.stop_epsilon)
    full = lambda v: torch.full((n,), float(v), dtype=torch.float64, device=dev)  # noqa: E731
    ids, E, L = torch.arange(n, device=dev), -p[0], p[3]
    y = torch.stack([full(0), full(cfg.cam.r), full(cfg.cam.theta), full(cfg.cam.phi), p[1], p[2]])
    k1, h, prev, tries, steps = _rates(y, E, L, a), full(0.02 * max(1.0, cfg.cam.r)), full(1e-4), full(0), full(0)
    out = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    table = _planck_table(dev)
    sky = []
    while ids.numel():
        fresh = tries == 0
        h = torch.where(fresh, torch.minimum(h, 0.05 * torch.clamp(y[1] - r_h, min=1.0) + 0.01), h)
        k = [k1]
        for row in _A:
            yn = y + h * _weighted(k, row)
            k.append(_rates(yn, E, L, a))
        e = h * _weighted(k, tuple(u - v for u, v in zip(_A[5] + (0.0,), _LOW)))
        q = e / (cfg.atol + cfg.rtol * torch.maximum(y.abs(), yn.abs()))
        err = torch.sqrt((q * q).sum(0) / 8)
        err = torch.where(torch.isfinite(err), err, torch.full_like(err, 1e5))
        fac = (0.9 * torch.clamp(err, min=1e-16) ** -0.14 * prev ** 0.08).clamp(0.2, 5.0)
        ok = err <= 1
        tries = torch.where(ok, 0.0, tries + 1)
        steps = steps + ok
        rn = yn[1]
        dead = ~ok & ((tries > 40) | ((h * fac.clamp(max=1.0)).abs() < 1e-14))
        fell = ok & (rn <= r_stop)
        live = ok & ~fell
        cross = torch.nonzero(live & (torch.cos(y[2]) * torch.cos(yn[2]) < 0)).flatten() if cfg.disc_enabled else ids[:0]
        hit = torch.zeros_like(ok)
        if cross.numel():
            kc, hc, y0, y1 = [v[:, cross] for v in k], h[cross], y[:, cross], yn[:, cross]
            m = torch.where(y1[2] > y0[2], torch.ceil((y0[2] - PI / 2) / PI), torch.floor((y0[2] - PI / 2) / PI))
            goal = PI / 2 + m * PI
            lo, hi = torch.zeros_like(hc), torch.ones_like(hc)
            kt = [v[2] for v in kc]
            below = y0[2] < goal
            for _ in range(60):
                mid = 0.5 * (lo + hi)
                far = (_dense(y0[2], y1[2], kt, hc, mid) < goal) != below
                lo, hi = torch.where(far, lo, mid), torch.where(far, mid, hi)
            s = 0.5 * (lo + hi)
            rc = _dense(y0[1], y1[1], [v[1] for v in kc], hc, s)
            on = (rc >= r_in) & (rc <= r_out)
            hit[cross[on]] = True
            i = cross[on]
            out[ids[i]] = _disc(cfg, table, rc[on], E[i], L[i], r_in, r_out)
        gone = live & ~hit & (rn > cfg.r_escape)
        sky.append((ids[gone], yn[:, gone], E[gone], L[gone]))
        done = dead | fell | hit | gone | (live & (steps >= cfg.max_steps))
        keep = ~done
        y = torch.where(ok, yn, y)[:, keep]
        k1 = torch.where(ok, k[6], k1)[:, keep]
        h = (h * torch.where(ok, fac, fac.clamp(max=1.0)))[keep]
        prev = torch.where(ok, err.clamp(min=1e-4), prev)[keep]
        tries, steps, ids, E, L = tries[keep], steps[keep], ids[keep], E[keep], L[keep]
    at, ye, E, L = (torch.cat([s[j] for s in sky], dim=-1) for j in range(4))
    if at.numel() and cfg.stars_enabled:
        out[at] = _sky(cfg, table, ye, E, L)
    spp = max(1, cfg.sqrt_spp) ** 2
    return out.reshape(cfg.height, cfg.width, spp, 3).mean(2).cpu().numpy()


def _planck_table(dev):
    """ln of the CIE XYZ of a blackbody at 4096 temperatures from 50 K to 3e9 K, 360 to 830 nm by 1 nm."""
    nm = np.arange(360.0, 831.0)

    def lobe(mu, s1, s2):
        return np.exp(-0.5 * ((nm - mu) / np.where(nm < mu, s1, s2)) ** 2)

    cie = np.stack([1.056 * lobe(599.8, 37.9, 31.0) + 0.362 * lobe(442.0, 16.0, 26.7) - 0.065 * lobe(501.1, 20.4, 26.2),
                    0.821 * lobe(568.8, 46.9, 40.5) + 0.286 * lobe(530.9, 16.3, 31.1),
                    1.217 * lobe(437.0, 11.8, 36.0) + 0.681 * lobe(459.0, 26.0, 13.8)])
    lam, hp, c, kb = nm * 1e-9, 6.62607015e-34, 2.99792458e8, 1.380649e-23
    T = 10.0 ** np.linspace(math.log10(50.0), math.log10(3.0e9), 4096)[:, None]
    x = hp * c / (lam * kb * T)
    with np.errstate(over="ignore"):
        B = np.where(x > 700.0, 0.0, 2 * hp * c * c / (lam ** 5 * np.expm1(np.minimum(x, 700.0))))
    return torch.from_numpy(np.log(np.maximum((B * 1e-9) @ cie.T, 1e-300))).to(dev)


def _blackbody(table, T):
    lo, hi = math.log10(50.0), math.log10(3.0e9)
    f = (torch.log10(T.clamp(50.0, 3.0e9)) - lo) / (hi - lo) * 4095
    i = f.long().clamp(0, 4094)
    u = (f - i)[:, None]
    return torch.exp(table[i] * (1 - u) + table[i + 1] * u)


def _disc(cfg, table, r, E, L, r_in, r_out):
    """Page and Thorne's flux of a thin disc, as blackbody light at the redshifted effective temperature."""
    a, sg = cfg.spin, cfg.disc_sense
    x, x0 = torch.sqrt(r), math.sqrt(r_in)
    W = x - x0 - 1.5 * a * torch.log(x / x0)
    third = math.acos(a) / 3
    roots = [2 * math.cos(third - PI / 3), 2 * math.cos(third + PI / 3), -2 * math.cos(third)]
    for i in range(3):
        u, v, w = roots[i], roots[(i + 1) % 3], roots[(i + 2) % 3]
        if abs(u) >= 1e-13:
            W = W - 3 * (u - a) ** 2 / (u * (u - v) * (u - w)) * torch.log((x - u) / (x0 - u))

    def orbit(r, root):
        den = r * root(r * r - 3 * r + 2 * sg * a * root(r))
        return (r * r - 2 * r + sg * a * root(r)) / den, sg * root(r) * (r * r - 2 * sg * a * root(r) + a * a) / den

    Ec, Lc = orbit(r, torch.sqrt)
    d = x ** 3 + sg * a
    Om = sg / d
    flux = 1.5 * sg * x / (d * d) / (4 * PI * r * (Ec - Om * Lc) ** 2) * W
    G, c, sb = 6.67430e-11, 2.99792458e8, 5.670374419e-8
    eta = 1 - orbit(r_in, math.sqrt)[0]
    L_edd = 4 * PI * G * cfg.M_kg * 1.67262192369e-27 * c / 6.6524587321e-29
    mdot = cfg.eddington * L_edd / (eta * c * c)
    flux = flux * mdot * c * c / (G * cfg.M_kg / (c * c)) ** 2
    good = torch.isfinite(flux) & (flux > 0) & (r > r_in)
    T = torch.where(good, flux.clamp(min=0.0) / sb, 0.0) ** 0.25
    ut = d / torch.sqrt(r ** 3 - 3 * r * r + 2 * sg * a * x ** 3)
    ku = -E * ut + L * Om * ut
    good = good & (ku > 1e-12)
    T = torch.where(good, T / torch.where(good, ku, 1.0), 1.0)
    return torch.where(good[:, None], _blackbody(table, T), 0.0)


def _sky(cfg, table, y, E, L):
    """Stars under the Gaussian point-spread function, cut at three sigma, and the diffuse background."""
    a, r, th, ph = cfg.spin, y[1], y[2], y[3]
    d = _rates(y, E, L, a)
    sn, cs, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
    R = torch.sqrt(r * r + a * a)
    dR = r / R * d[1]
    v = torch.stack([dR * sn * cp + R * cs * d[2] * cp - R * sn * sp * d[3],
                     dR * sn * sp + R * cs * d[2] * sp + R * sn * cp * d[3], d[1] * cs - r * sn * d[2]], 1)
    v = v / v.norm(dim=1, keepdim=True)
    back = _blackbody(table, torch.tensor([4800.0], dtype=torch.float64, device=v.device))[0]
    diffuse = 3.24e-10 * 10 ** (-0.4 * 21.5) * 4.2545170296152206e10 if cfg.milky_way else 0.0
    out = (diffuse * back / back[1]).expand(v.shape[0], 3).clone()
    # the catalogue: four draws a star (z, longitude, magnitude, B-V)
    i = 4 * np.arange(cfg.star_count)
    z, lon, mag, bv = (_uniform(np.uint64(cfg.seed), i + j) for j in (1, 2, 3, 4))
    z, lon = 2 * z - 1, 2 * PI * lon
    rho = np.sqrt(np.maximum(0.0, 1 - z * z))
    mag = -1.5 + np.log10(mag * (10 ** (0.45 * 8.0) - 1) + 1) / 0.45
    bv = np.clip(-0.3 + 2.1 * bv, -0.4, 2.0)
    T = 4600 * (1 / (0.92 * bv + 1.7) + 1 / (0.92 * bv + 0.62))
    star = torch.from_numpy(np.stack([rho * np.cos(lon), rho * np.sin(lon), z], 1)).to(v.device)
    power = torch.from_numpy(3.64e-9 * 0.089 * 10 ** (-0.4 * mag)).to(v.device)
    colour = _blackbody(table, torch.from_numpy(T).to(v.device))
    colour = colour / colour[:, 1:2]
    sigma = 0.55 * cfg.cam.fov / cfg.width
    # stars sorted by height: each ray looks at the slab around its own
    order = torch.argsort(star[:, 2])
    star, power, colour = star[order], power[order], colour[order]
    heights = star[:, 2].contiguous()
    slab = 3.0 * sigma * 1.001
    lat = torch.asin(v[:, 2].clamp(-1, 1))
    first = torch.searchsorted(heights, torch.sin((lat - slab).clamp(min=-PI / 2)))
    last = torch.searchsorted(heights, torch.sin((lat + slab).clamp(max=PI / 2)))
    for k in range(0, v.shape[0], 4096):
        f, n = first[k:k + 4096], (last - first)[k:k + 4096]
        ray = torch.repeat_interleave(torch.arange(f.numel(), device=v.device), n)
        if not ray.numel():
            continue
        s = f[ray] + torch.arange(ray.numel(), device=v.device) - (torch.cumsum(n, 0) - n)[ray]
        ang = 2 * torch.asin((0.5 * (v[k + ray] - star[s]).norm(dim=1)).clamp(max=1.0))
        near = ang <= 3.0 * sigma
        ray, s, ang = ray[near], s[near], ang[near]
        w = power[s] * torch.exp(-ang * ang / (2 * sigma * sigma)) / (2 * PI * sigma * sigma)
        out.index_add_(0, k + ray, w[:, None] * colour[s])
    return out
