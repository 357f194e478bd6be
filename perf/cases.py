"""What a program that uses this framework has it do, as cases that can be timed
and compared: frames, batches, recorded trajectories, per-ray states and
gradients, through the package's public entry points.

Every case traces null geodesics with adaptive RKF45 from one camera (or from
one camera per frame) and colours them; the families are

  render   Context.render: host frames out (the 8-bit image, and the float one
           where the case says so)
  device   Context.render_device into device buffers
  graph    Graph.launch: a recorded camera trajectory
  rays     Context.trace_rays / trace_rays_f64: per-ray final states
  adjoint  Context.adjoint: the gradient of an image loss (the backward pass)

The seed moves cameras, spins, spheres and losses by a few per cent, so another
seed is another input of the same size and cost.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from parrelray_b200 import Context, Graph, LaunchConfig, abi, scenes

SHAPE_TUNED = (64, 0, 64, 1)  # what Context.autotune settles on for full-size frames

PRECISION = {"fp32": abi.PREC_FP32, "fp64": abi.PREC_FP64, "split": abi.PREC_SPLIT}
METRIC = {"flat": abi.METRIC_FLAT, "schwarzschild": abi.METRIC_SCHWARZSCHILD, "kerr": abi.METRIC_KERR}
SSAA = {"none": abi.SSAA_NONE, "regular": abi.SSAA_REGULAR, "random": abi.SSAA_RANDOM, "jittered": abi.SSAA_JITTERED}
CAMERA = {"spherical": abi.CAMERA_SPHERICAL, "pinhole": abi.CAMERA_PINHOLE, "panorama": abi.CAMERA_PANORAMA}

BASE = {"family": "render", "width": 320, "height": 180, "frames": 1, "samples": 1, "ssaa": "none", "metric": "kerr",
        "precision": "fp32", "mode": "physical", "tol": 1e-6, "r": 25.0, "incl": 80.0, "fov": 50.0, "spin": 0.9,
        "spheres": 1, "fxaa": False, "bilinear": False, "camera": "spherical", "emission": "none", "tuned": False,
        "floats": False, "uneven": False, "hmax": 0.1}


def _case(name=None, **kw) -> dict:
    c = dict(BASE)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed() -> list[dict]:
    return [
        # a preview while a scene is set up: a thumbnail on the default context; latency counts, the chip is not full
        _case("preview_96x54", width=96, height=54, floats=True),
        # the single-frame workload: Schwarzschild 320x180, one textured sphere, default context
        _case("single_schw_320x180", metric="schwarzschild", spin=0.0, r=30.0, incl=85.0, fov=60.0, floats=True),
        # the same deck in REFERENCE mode (the reference's own algorithm and tolerance), as its users first run it
        _case("reference_mode_320x180", metric="schwarzschild", spin=0.0, r=30.0, incl=85.0, fov=60.0, mode="reference"),
        # the headline frame: Kerr 1080p, 2x2 SSAA, FXAA, three spheres, tuned launch shape, into device memory
        _case("headline_kerr_1080p_ssaa4", family="device", width=1920, height=1080, samples=4, ssaa="regular", spin=0.95,
              spheres=3, fxaa=True, tuned=True),
        # an ordinary still of an odd size: 3x3 jittered SSAA through a pinhole camera, default context
        _case("still_613x347_jitter9", width=613, height=347, samples=9, ssaa="jittered", camera="pinhole", fov=60.0,
              spheres=2, r=18.0, incl=70.0),
        # a double-precision frame (the accuracy reference users render beside FP32)
        _case("fp64_640x360", family="device", width=640, height=360, precision="fp64", floats=True, tuned=True),
        # a server's batch of uneven requests in split precision at tolerance 1e-7 (FP32, FP64 near the photon orbit)
        _case("split_uneven_12", family="device", frames=12, width=420, height=300, precision="split", tol=1e-7,
              spheres=0, uneven=True, fov=60.0, tuned=True, floats=True),
        # a camera trajectory recorded once and replayed: 16 frames 960x540
        _case("trajectory_16x960x540", family="graph", frames=16, width=960, height=540, spin=0.9, r=14.0, incl=75.0,
              fov=60.0, tuned=True),
        # an image of a radiating disk, as for the EHT targets
        _case("disk_640x640", family="device", width=640, height=640, emission="disk", spin=0.94, r=50.0, incl=17.0,
              fov=27.0, camera="pinhole", spheres=0, floats=True, tuned=True),
        # per-ray double states for an analysis outside the renderer
        _case("rays_f64_161x91", family="rays", width=161, height=91, precision="fp64", spheres=0, tol=1e-7),
        # one gradient of an inverse fit (FP32 forward steps, FP64 reverse sweep)
        _case("adjoint_512x512", family="adjoint", width=512, height=512, spin=0.7, r=20.0, incl=60.0, fov=40.0,
              bilinear=True, tuned=True),
        # one gradient with FP64 forward steps, 2x2 SSAA, on the default context
        _case("adjoint_f64_160x120_ssaa4", family="adjoint", width=160, height=120, samples=4, ssaa="regular",
              precision="fp64", spin=0.5, r=16.0, incl=70.0, fov=40.0, bilinear=True),
    ]


def _log(rng, lo, hi) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    """One more case of these ranges: sizes log-uniform (odd ones among them), every option that the listed ones use,
    and no more work than the headline frame."""
    c = _draw(rng)
    weight = {"fp32": 1.0, "split": 1.5, "fp64": 3.0}[c["precision"]]
    while weight * work(c)["flops"] > 3.5e12:
        c["width"], c["height"] = int(0.85 * c["width"]), int(0.85 * c["height"])
    return c


def _draw(rng) -> dict:
    kind = rng.choice(["frame", "frame", "frame64", "batch", "graph", "disk", "grid", "rays", "adjoint", "reference"])
    spin = rng.uniform(0.0, 0.998)
    cam = dict(r=rng.uniform(9.0, 40.0), incl=rng.uniform(15.0, 88.0), fov=rng.uniform(35.0, 70.0))
    metric = rng.choice(["kerr", "kerr", "schwarzschild"])
    base = dict(metric=metric, spin=spin if metric == "kerr" else 0.0, tuned=rng.random() < 0.5, **cam)
    w = int(_log(rng, 64, 1280))
    h = max(36, int(w * rng.uniform(0.45, 1.0)))
    if kind in ("frame", "frame64"):
        ssaa, samples = rng.choice([("none", 1), ("none", 1), ("regular", 4), ("regular", 9), ("jittered", 4), ("random", 5)])
        if kind == "frame64":
            w, h = min(w, 640), min(h, 480)
            if samples > 4:
                ssaa, samples = "regular", 4
        return _case(family=rng.choice(["render", "device"]), width=w, height=h, ssaa=ssaa, samples=samples,
                     precision="fp64" if kind == "frame64" else "fp32", spheres=rng.randint(0, 3),
                     fxaa=kind == "frame" and rng.random() < 0.5, floats=kind == "frame64",
                     camera=rng.choice(["spherical", "spherical", "pinhole", "panorama"]),
                     tol=rng.choice([1e-6, 1e-7]), hmax=rng.choice([0.1, 0.1, 0.2, 0.05]), **base)
    if kind == "batch":
        return _case(family="device", frames=rng.randint(3, 16), width=int(_log(rng, 96, 480)), height=int(_log(rng, 96, 400)),
                     precision=rng.choice(["split", "split", "fp32"]), tol=1e-7, spheres=0, uneven=True, floats=True, **base)
    if kind == "graph":
        w = int(_log(rng, 128, 800))
        return _case(family="graph", frames=rng.randint(4, 12), width=w, height=int(w * 0.5625) | 1, spheres=1, **base)
    if kind in ("disk", "grid"):
        w = int(_log(rng, 64, 700))
        return _case(family="device", width=w, height=w, emission=kind, camera="pinhole", spheres=0, floats=True,
                     precision=rng.choice(["fp32", "fp32", "fp64"]) if w < 300 else "fp32",
                     **dict(base, r=rng.uniform(25.0, 50.0), fov=30.0))
    if kind == "rays":
        w = int(_log(rng, 48, 320))
        return _case(family="rays", width=w, height=int(w * 0.6) | 1, precision=rng.choice(["fp64", "fp32"]),
                     spheres=rng.randint(0, 2), tol=rng.choice([1e-6, 1e-7]), **base)
    if kind == "adjoint":
        w = int(_log(rng, 48, 512))
        prec = rng.choice(["fp32", "fp32", "fp64"])
        big = w > 256
        return _case(family="adjoint", width=w, height=int(w * rng.uniform(0.6, 1.0)), bilinear=True, spheres=1,
                     precision="fp32" if big else prec, **({} if big or rng.random() < 0.5 else dict(ssaa="regular", samples=4)),
                     **base)
    return _case(family="render", width=int(_log(rng, 64, 480)), height=int(_log(rng, 48, 270)), mode="reference",
                 spheres=rng.randint(0, 2), **base)


# ------------------------------------------------------------------ inputs

_textures: dict[int, np.ndarray] = {}


def _tex() -> dict[int, np.ndarray]:
    if not _textures:
        _textures.update(scenes.standard_textures())
    return _textures


def _frames(case: dict, seed: int) -> list[abi.FrameDesc]:
    rng = np.random.default_rng([seed, 17])
    out = []
    for k in range(case["frames"]):
        t = k / max(case["frames"] - 1, 1)
        j = rng.uniform(-1.0, 1.0, size=6)
        r = case["r"] * (1.0 + 0.02 * j[0])
        incl = min(max(case["incl"] + 1.5 * j[1], 5.0), 89.0)
        spin = min(abs(case["spin"]) * (1.0 + 0.002 * j[2]), 0.998) if case["spin"] else 0.0
        w, h = case["width"], case["height"]
        if case["uneven"]:  # request sizes 1/2 .. 2 of the nominal one, cameras and spins of their own
            u = np.random.default_rng([case["frames"], k])
            w, h = int(w * math.exp(u.uniform(-0.7, 0.7))), int(h * math.exp(u.uniform(-0.7, 0.7)))
            r, incl = float(u.uniform(8.0, 40.0)) * (1.0 + 0.02 * j[0]), float(u.uniform(10.0, 87.0)) + 1.5 * j[1]
            spin = float(u.uniform(0.05, 0.99)) if case["metric"] == "kerr" else 0.0
        if case["family"] == "graph":  # an approach towards the hole
            r, incl = r * (1.2 - 0.5 * t), max(incl - 12.0 * (1.0 - t), 5.0)
        sph = []
        for s in range(case["spheres"]):
            rad, orb, ph = scenes.KERR_1080P_SPHERES[s]
            sph.append((*scenes.orbit_point(orb, ph + 1.5 * k + 10.0 * j[3 + s]), rad, scenes.SPHERE_ID0 + s))
        d = scenes.make_frame(
            w, h, r=float(r), incl_deg=float(incl), fov_deg=case["fov"], metric=METRIC[case["metric"]], spin=float(spin),
            samples=case["samples"], fxaa=case["fxaa"], tol=case["tol"], precision=PRECISION[case["precision"]],
            mode=abi.MODE_REFERENCE if case["mode"] == "reference" else abi.MODE_PHYSICAL, spheres=sph, hmax=case["hmax"],
            bg_filter=abi.BG_BILINEAR if case["bilinear"] else abi.BG_RMS2X2, background=case["emission"] == "none")
        d.ssaa = SSAA[case["ssaa"]]
        d.camera = CAMERA[case["camera"]]
        d.ssaa_seed = 1 + seed % 1000
        if case["emission"] != "none":
            rp = 1.0 + math.sqrt(max(0.0, 1.0 - spin * spin))
            scenes.set_emission(d, abi.EMISSION_DISK if case["emission"] == "disk" else abi.EMISSION_GRID, r_in=scenes.f32(rp),
                                r_out=20.0, index=3.0, height=0.4, gain=2.0, absorb=0.0 if case["emission"] == "disk" else 0.02)
        out.append(d)
    return out


class _State:
    """A context with its textures (and plasma, launch shape, buffers, recorded graph), as a program keeps it."""

    def __init__(self, case: dict, seed: int):
        self.case, self.ctx, self.graph = case, Context(0), None
        self.frames = _frames(case, seed)
        self.ctx.upload_textures(_tex())
        if case["tuned"]:
            self.ctx.set_schedule(abi.SCHED_PERSISTENT, LaunchConfig(*SHAPE_TUNED))
        if case["emission"] == "grid":
            n = 48
            g = np.linspace(-20.0, 20.0, n, dtype=np.float32)
            z, y, x = np.meshgrid(g, g, g, indexing="ij")
            rr = np.sqrt(x * x + y * y + z * z) + 1.0
            rho = (rr / 3.0) ** -2 * np.exp(-(z / rr) ** 2 / 0.3) * (1.0 + 0.2 * np.sin(x + seed % 7))
            self.ctx.upload_plasma(rho.astype(np.float32), (-20.0,) * 3, (20.0,) * 3, temperature=(1.0 / rr).astype(np.float32))
        npx = sum(f.width * f.height for f in self.frames)
        fam = case["family"]
        self.rgb8 = self.rgbf = None
        if fam in ("device", "graph"):
            if case["floats"]:
                self.rgbf = torch.zeros(3 * npx, dtype=torch.float32, device="cuda")
            else:
                self.rgb8 = torch.zeros(3 * npx, dtype=torch.uint8, device="cuda")
        if fam == "graph":
            self.graph = Graph(self.ctx, self.frames, self.rgb8.data_ptr())
        if fam == "adjoint":
            f = self.frames[0]
            self.dl = np.random.default_rng([seed, 3]).standard_normal((f.height, f.width, 3)).astype(np.float32)

    def __del__(self):
        if getattr(self, "graph", None):
            self.graph.close()
        if getattr(self, "ctx", None):
            self.ctx.close()


def prepare(case: dict, seed: int) -> _State:
    return _State(dict(BASE, **case), seed)


def run(state: _State):
    c, ctx, f = state.case, state.ctx, state.frames
    fam = c["family"]
    if fam == "render":
        img8, imgf, _ = ctx.render(f, want_float=c["floats"])
        return (imgf if c["precision"] == "fp64" else [img8, imgf]) if c["floats"] else img8
    if fam == "device":
        out = state.rgb8 if state.rgbf is None else state.rgbf
        ctx.render_device(f, state.rgb8.data_ptr() if state.rgb8 is not None else None,
                          state.rgbf.data_ptr() if state.rgbf is not None else None,
                          torch.cuda.current_stream().cuda_stream)
        return out
    if fam == "graph":
        state.graph.launch(torch.cuda.current_stream().cuda_stream)
        return state.rgb8
    if fam == "rays":
        st, rgb, _ = ctx.trace_rays_f64(f[0]) if c["precision"] == "fp64" else ctx.trace_rays(f[0])
        return [st, rgb]
    grads, _ = ctx.adjoint(f[0], state.dl, 0 if c["spheres"] else -1)
    return grads


def work(case: dict) -> dict:
    """Floating-point operations of the rays' attempts, and the textures and outputs.  A ray flies about r + rout in
    steps of hmax (in steps of order 0.1 in REFERENCE mode); a step of the 4th-order solution takes five right-hand
    sides of about 95 operations, the sixth and the error estimate about 200 more."""
    c = dict(BASE, **case)
    frames = _frames(c, 0)
    rays = sum(f.nrays for f in frames)
    steps = sum(f.nrays * 0.93 * (math.hypot(*f.cam_pos) + f.rout) / f.hmax for f in frames)
    flops = steps * (5 * 95 + 100)
    if c["family"] == "adjoint":  # the reverse sweep: the five stages again and their vector-Jacobian products (x 2.5)
        flops *= 4.5
    out = 96 * rays if c["family"] == "rays" else sum(f.width * f.height for f in frames) * (12 if c["floats"] else 3)
    tex = 4 * 2048 * 1024 + c["spheres"] * 4 * 512 * 256
    return {"bytes": float(out + tex), "flops": float(flops)}


# ------------------------------------------------------------------ 64-bit values

def exact(case: dict, seed: int):
    """The same discrete algorithm in 64 bits (plain torch), for frames small enough; the 8-bit images, REFERENCE mode
    (its value is its FP32 operation order), stochastic sampling, plasma grids and gradients have no such value here."""
    c = dict(BASE, **case)
    frames = _frames(c, seed)
    rays = sum(f.nrays for f in frames)
    plain = c["mode"] == "physical" and c["ssaa"] in ("none", "regular") and c["emission"] != "grid" and not c["fxaa"]
    if not plain or rays > 450_000 or c["frames"] > 1 or c["family"] in ("adjoint", "graph"):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["family"] == "rays":
        st, rgb = _trace(frames[0], dev)
        return [st.cpu().numpy(), rgb.cpu().numpy()]
    if not c["floats"]:
        return None
    img = _combine(frames[0], _trace(frames[0], dev)[1])
    if c["family"] == "device":
        return img.reshape(-1)
    img = img.cpu().numpy()
    return [img] if c["precision"] == "fp64" else [[None], [img]]


def _combine(f, rgb: torch.Tensor) -> torch.Tensor:
    S = f.samples
    if S == 1:
        return rgb.clamp(0.0, 1.0).reshape(f.height, f.width, 3)
    return torch.sqrt((rgb * rgb).clamp(0.0, 1.0).reshape(f.height, f.width, S, 3).sum(2) / S)


def _ks(x, y, z, M, a):
    """Kerr-Schild r, f and l at (x, y, z)."""
    hb = 0.5 * (x * x + y * y + z * z - a * a)
    r2 = hb + torch.sqrt(hb * hb + a * a * z * z)
    r = torch.sqrt(r2)
    q = r2 + a * a
    return r, 2.0 * M * r * r2 / (r2 * r2 + a * a * z * z), ((r * x + a * y) / q, (r * y - a * x) / q, z / r)


def _rhs(s, pt, M, a):
    """dx = p - f Lam l, dp = 1/2 Lam^2 grad f + f Lam grad Lam for s = (x, y, z, px, py, pz)."""
    x, y, z, px, py, pz = s
    if M == 0.0:
        o = torch.zeros_like(x)
        return torch.stack((px, py, pz, o, o, o))
    a2 = a * a
    hb = 0.5 * (x * x + y * y + z * z - a2)
    Sh = torch.sqrt(hb * hb + a2 * z * z)
    r2 = hb + Sh
    r = torch.sqrt(r2)
    q, Sig = r2 + a2, r2 * r2 + a2 * z * z
    rx, ry, rz = x * r / (2.0 * Sh), y * r / (2.0 * Sh), z * q / (2.0 * Sh * r)
    f = 2.0 * M * r * r2 / Sig
    c1 = f * (3.0 / r - 4.0 * r * r2 / Sig)
    lx, ly, lz = (r * x + a * y) / q, (r * y - a * x) / q, z / r
    lp = lx * px + ly * py
    Lam = lp + lz * pz - pt
    Pp = (x * px + y * py - 2.0 * r * lp) / q - pz * lz / r
    h2, fL = 0.5 * Lam * Lam, f * Lam
    return torch.stack((px - fL * lx, py - fL * ly, pz - fL * lz,
                        h2 * c1 * rx + fL * (rx * Pp + (r * px - a * py) / q),
                        h2 * c1 * ry + fL * (ry * Pp + (a * px + r * py) / q),
                        h2 * (c1 * rz - 2.0 * f * a2 * z / Sig) + fL * (rz * Pp + pz / r)))


_A = [[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197], [439 / 216, -8.0, 3680 / 513, -845 / 4104],
      [-8 / 27, 2.0, -3544 / 2565, 1859 / 4104, -11 / 40]]
_B4 = [25 / 216, 0.0, 1408 / 2565, 2197 / 4104, -1 / 5, 0.0]
_B5 = [16 / 135, 0.0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]


def _texels(tex: torch.Tensor, i, j):
    h, w = tex.shape[:2]
    return tex[j.clamp(0, h - 1), i.clamp(0, w - 1)]


def _sky(f, u, dev):
    """The sky in direction u (3, n): RMS of the 2x2 block, or bilinear over texel centres."""
    if f.background_id < 0:
        return torch.zeros(u.shape[1], 3, dtype=torch.float64, device=dev)
    tex = torch.from_numpy(_tex()[f.background_id][:, :, :3].astype(np.float32) / np.float32(255.0)).to(dev).double()
    h, w = tex.shape[:2]
    n = u / torch.linalg.vector_norm(u, dim=0)
    theta, phi = torch.arccos(n[2].clamp(-1.0, 1.0)), torch.atan2(n[1], n[0])
    phi = torch.where(phi >= 0.0, phi, phi + 2.0 * math.pi)
    fx, fy = phi / (2.0 * math.pi) * w, theta / math.pi * h
    if f.bg_filter == abi.BG_BILINEAR:
        fx, fy = fx - 0.5, fy - 0.5
        x0, y0 = torch.floor(fx).long(), torch.floor(fy).long()
        wx, wy = (fx - x0)[:, None], (fy - y0)[:, None]
        t = lambda i, j: _texels(tex, i % w, j)  # noqa: E731
        return (t(x0, y0) * (1 - wx) * (1 - wy) + t(x0 + 1, y0) * wx * (1 - wy) + t(x0, y0 + 1) * (1 - wx) * wy
                + t(x0 + 1, y0 + 1) * wx * wy)
    i, j = torch.floor(fx).long().clamp(max=w - 1), torch.floor(fy).long().clamp(max=h - 1)
    a, b, c, d = (_texels(tex, i + p, j + q) for p, q in ((0, 0), (0, 1), (1, 0), (1, 1)))
    edge = ((i == w - 1) | (j == h - 1))[:, None]
    return torch.where(edge, a, torch.sqrt(0.25 * (a * a + b * b + c * c + d * d)))


def _sphere_colour(S, x, v, d, dev):
    c = torch.tensor([S.center[0], S.center[1], S.center[2]], dtype=torch.float64, device=dev)[:, None]
    i = x + v * d - c
    rad, PI = S.radius, 3.14159265359
    uu = ((torch.atan2(i[1], i[0]) + PI) / (2.0 * PI)).clamp(0.0, 0.999999999)
    vv = (torch.arccos(i[2] / rad) / PI).clamp(0.0, 0.999999999)
    tex = torch.from_numpy(_tex()[S.texture_id][:, :, :3].astype(np.float32) / np.float32(255.0)).to(dev).double()
    h, w = tex.shape[:2]
    ux, uy = torch.nan_to_num(uu * w), torch.nan_to_num(vv * h)
    ix, iy = torch.floor(ux).long(), torch.floor(uy).long()
    px, py = (ux - ix)[:, None], (uy - iy)[:, None]
    ix, iy = ix.clamp(0, w - 2), iy.clamp(0, h - 2)
    t = (tex[iy, ix] * (1 - px) * (1 - py) + tex[iy, ix + 1] * px * (1 - py) + tex[iy + 1, ix] * (1 - px) * py
         + tex[iy + 1, ix + 1] * px * py)
    return t * (0.5 + 0.5 * i[2] / rad).clamp(0.0, 1.0)[:, None]


def _start(f, dev):
    """Screen positions and null initial momenta (the ray directions are FP32 by definition of the path)."""
    W, H, S = f.width, f.height, f.samples
    n = W * H * S
    k = torch.arange(n, device=dev)
    s, pix = k % S, k // S
    x, y = (pix % W).float(), (pix // W).float()
    w32, h32 = np.float32(W), np.float32(H)
    if S == 1:
        uvx, uvy = x / W + float(np.float32(1) / w32 * np.float32(0.5)), y / H + float(np.float32(1) / h32 * np.float32(0.5))
    else:
        q = int(round(math.sqrt(S)))
        dux, duy = float(np.float32(1) / w32 / np.float32(q + 1)), float(np.float32(1) / h32 / np.float32(q + 1))
        uvx, uvy = x / W + (s % q + 1).float() * dux, y / H + (s // q + 1).float() * duy
    al, be, vf = f.cam_alpha, f.cam_beta, f.vfov
    if f.camera == abi.CAMERA_PINHOLE or f.camera == abi.CAMERA_PANORAMA:
        fw = np.array([math.cos(-be) * math.cos(al), math.cos(-be) * math.sin(al), math.sin(be)])
        up = np.array([math.cos(al) * math.sin(-be), math.sin(al) * math.sin(-be), math.cos(be)])
        rt = np.cross(fw, up)
        if f.camera == abi.CAMERA_PINHOLE:
            th = math.tan(vf / 2.0)
            c = (torch.ones_like(uvx), (2.0 * uvx - 1.0) * th * W / H, (1.0 - 2.0 * uvy) * th)
        else:
            mu, nu = (0.5 - uvy) * vf, (uvx - 0.5) * W / H * vf
            c = (torch.cos(mu) * torch.cos(nu), torch.cos(mu) * torch.sin(nu), torch.sin(mu))
        v = [c[0] * float(fw[m]) + c[1] * float(rt[m]) + c[2] * float(up[m]) for m in range(3)]
    else:
        nu, mu = (0.5 - uvy) * vf, (0.5 - uvx) * W / H * vf
        cb = torch.cos(be + nu)
        v = [cb * torch.cos(al + mu), cb * torch.sin(al + mu), torch.sin(be + nu)]
    v = torch.stack(v)
    return uvx, uvy, (v / torch.sqrt((v * v).sum(0))).double()


def _trace(f, dev):
    """Every ray of frame f integrated in 64 bits: (n, 12) states and (n, 3) colours, in the layout of trace_rays."""
    M = 0.0 if f.metric == abi.METRIC_FLAT else f.mass
    a = f.spin if f.metric == abi.METRIC_KERR else 0.0
    rp = 0.0 if M == 0.0 else M + math.sqrt(M * M - a * a)
    rstop = float(np.float32(np.float32(rp) + np.float32(f.horizon_eps)))
    uvx, uvy, dr = _start(f, dev)
    n = uvx.numel()
    full = lambda v: torch.full((n,), float(v), dtype=torch.float64, device=dev)  # noqa: E731
    pos = [full(f.cam_pos[k]) for k in range(3)]
    r, fc, l = _ks(*pos, M, a)
    ld = l[0] * dr[0] + l[1] * dr[1] + l[2] * dr[2]
    A, B, C = fc - 1.0, 2.0 * fc * ld, (dr * dr).sum(0) + fc * ld * ld
    rt = torch.sqrt(B * B - 4.0 * A * C)
    ut = torch.maximum((-B + rt) / (2.0 * A), (-B - rt) / (2.0 * A))
    ut = torch.where(ut < 0.0, torch.ones_like(ut), ut)
    Lu = ld + ut
    s = torch.stack((*pos, dr[0] + fc * l[0] * Lu, dr[1] + fc * l[1] * Lu, dr[2] + fc * l[2] * Lu))
    pt = -ut + fc * Lu
    nu_cam = -pt / torch.sqrt(1.0 - fc)
    out = torch.zeros(n, 12, dtype=torch.float64, device=dev)
    rgb = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    glow = torch.zeros(n, dtype=torch.float64, device=dev)
    out[:, 0], out[:, 1] = uvx.double(), uvy.double()
    ids = torch.arange(n, device=dev)
    h, th, path = full(f.h), full(f.h), full(0.0)
    tries, acc = torch.zeros_like(ids), torch.zeros_like(ids)
    inter = torch.zeros_like(ids, dtype=torch.bool)

    def velocity(s, pt):
        _, fc, l = _ks(s[0], s[1], s[2], M, a)
        fL = fc * (l[0] * s[3] + l[1] * s[4] + l[2] * s[5] - pt)
        return torch.stack((s[3] - fL * l[0], s[4] - fL * l[1], s[5] - fL * l[2])), fL - pt

    def end(m, result, st, colour=None, u=None):
        if not bool(m.any()):
            return
        k = ids[m]
        out[k, 2] = float(result)
        out[k, 3:6] = st[:3, m].T
        uu, ut = velocity(st[:, m], pt[m])
        out[k, 7:10], out[k, 10] = (uu.T, ut) if u is None else (u, torch.zeros_like(ut))
        out[k, 11] = acc[m].double()
        if colour is not None:
            rgb[k] = colour

    while ids.numel():
        done = ~(path < 1000.0)
        end(done, 3, s)
        tries = tries + 1
        ks = []
        for row in _A:
            z = s
            for c, k in zip(row, ks):
                z = z + c * k
            ks.append(h * _rhs(z, pt, M, a))
        d = sum(c * k for c, k in zip(_B4, ks) if c)
        e = sum((c5 - c4) * k for c5, c4, k in zip(_B5, _B4, ks) if c5 != c4)
        y = s + d
        err = (e.abs() / (f.atol + f.rtol * torch.maximum(s.abs(), y.abs()))).amax(0)
        hn = torch.nan_to_num(0.9 * h * err ** -0.2, nan=f.hmin, posinf=f.hmax).clamp(f.hmin, f.hmax)
        inter = inter & ~(tries > 10000)
        over = ~done & (tries > 8 * f.max_steps)
        end(over, 3, s)
        done = done | over
        live = ~done & ~((err > 1.0) & (h != f.hmin) & ~inter)
        retry = ~done & ~live
        bad = live & torch.isnan(y.sum(0))
        end(bad, 1, s)
        done, live = done | bad, live & ~bad
        hit = torch.zeros_like(inter)
        far = torch.full_like(h, 1e11)
        best = [[far.clone(), torch.full_like(ids, -1)] for _ in range(3)]
        v = None
        if f.nspheres:
            u, _ = velocity(y, pt)
            v = u / torch.sqrt((u * u).sum(0))
            for q in range(f.nspheres):
                S = f.spheres[q]
                dx = torch.stack([y[m] - S.center[m] for m in range(3)])
                b = (v * dx).sum(0)
                disc = b * b - ((dx * dx).sum(0) - S.radius * S.radius)
                dist = -2.0 * b - torch.sqrt(disc.clamp(min=0.0))
                for w, win in enumerate((h, hn, th)):
                    ok = (disc >= 0.0) & (dist >= 0.0) & ~(dist * dist > win) & (dist <= best[w][0])
                    best[w][0] = torch.where(ok, dist, best[w][0])
                    best[w][1] = torch.where(ok, q, best[w][1])
            hit = best[0][1] >= 0
        enter = live & hit & ~inter
        inter = inter | enter
        live = live & ~enter
        acc = acc + live
        if f.emission == abi.EMISSION_DISK:
            glow[ids] += torch.where(live, _disk(f, y, pt, nu_cam[ids], h, M, a), 0.0)
        s = torch.where(live, y, s)
        h = torch.where(enter, f.hmin, torch.where(retry | (live & ~hit & ~inter), hn, h))
        th = torch.where(live & ~hit, h, th)
        clear = ~hit
        cand = torch.where(clear, torch.where(inter, best[0][1], best[1][1]), best[2][1])
        dist = torch.where(clear, torch.where(inter, best[0][0], best[1][0]), best[2][0])
        r = _ks(s[0], s[1], s[2], M, a)[0]
        esc = live & (r >= f.rout)
        cap = live & ~esc & (r <= rstop) if M else torch.zeros_like(esc)
        if bool(esc.any()):
            end(esc, 0, s, _sky(f, velocity(s[:, esc], pt[esc])[0], dev))
        end(cap, 0, s)
        done = done | esc | cap
        for q in range(f.nspheres):
            m = live & ~done & (cand == q)
            if bool(m.any()):
                col = _sphere_colour(f.spheres[q], s[:3, m], v[:, m], dist[m], dev)
                end(m, 4, s, col, col)
            done = done | m
        live = live & ~done
        path = torch.where(live, path + h, path)
        cut = live & (acc >= f.max_steps)
        end(cut, 3, s)
        done = done | cut
        if bool(done.any()):
            m = ~done
            s, pt, ids, h, th, path, tries, acc, inter = (s[:, m], pt[m], ids[m], h[m], th[m], path[m], tries[m], acc[m],
                                                          inter[m])
    if f.emission == abi.EMISSION_DISK:
        g = (f.emis.gain * glow)[:, None]
        rgb += torch.cat(((2.0 * g).clamp(0, 1), (2.0 * g - 0.5).clamp(0, 1), (2.0 * g - 1.0).clamp(0, 1)), 1)
    return out, rgb


def _disk(f, y, pt, nu_cam, h, M, a):
    """The thick disk's contribution of one accepted step (optically thin, spectral index 0)."""
    e = f.emis
    r, fc, l = _ks(y[0], y[1], y[2], M, a)
    n = (r / e.r_in) ** -e.index * torch.exp(-((y[2] / r) ** 2) / (2.0 * e.height * e.height))
    om = e.sense * math.sqrt(M) / (r * torch.sqrt(r) + e.sense * a * math.sqrt(M))
    vx, vy = -om * y[1], om * y[0]
    lv = l[0] * vx + l[1] * vy + 1.0
    N = vx * vx + vy * vy - 1.0 + fc * lv * lv
    nu_e = -(y[3] * vx + y[4] * vy + pt) / torch.sqrt(torch.where(N < 0.0, -N, torch.ones_like(N)))
    ok = (r >= e.r_in) & (r <= e.r_out) & (N < 0.0) & (nu_e > 0.0)
    g = nu_cam / torch.where(nu_e > 0.0, nu_e, torch.ones_like(nu_e))
    return torch.where(ok, g * g * n * nu_cam * h, torch.zeros_like(n))
