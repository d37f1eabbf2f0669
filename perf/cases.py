"""The work that a program using the tracer has it do, as timed cases.

Each case is one call (or one batch of requests) through the public Python
binding: a tile of a progressive render, interactive previews, whole images in
both precisions, the Boyer-Lindquist path, multi-source scenes, the shaded
image read back to pinned memory, the volumetric torus, a table of cameras and
the request server.  Cameras are the repository's benchmark geometries; the
seed moves the observer and the hole's spin, so that every seed is another
image of the same kind and size.

`exact` integrates the same rays with torch in 64 bits (Dormand-Prince 5(4) at
a hundredth of the FP64 tracer's tolerance): Kerr-Schild rays from the
Hamiltonian of the Kerr-Schild form, Boyer-Lindquist rays from the separable
Kerr-Newman Hamiltonian in Mino time.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "relativity-simulator_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import relsim  # noqa: E402
import scenes  # noqa: E402

RECORD = ["status", "r", "theta", "phi", "r_hit", "g"]  # the record that the server keeps by default
FACE_ON = dict(spin=0.94, r_obs=100.0, incl=17.0, fov=12.0)   # the headline camera
EDGE_ON = dict(spin=0.998, r_obs=60.0, incl=80.0, fov=20.0)   # the near-extremal, grazing camera
CHARGED = dict(spin=0.9, charge=0.3, r_obs=50.0, incl=75.0, fov=30.0)  # the Kerr-Newman camera
WIDE = dict(spin=0.6, r_obs=40.0, incl=60.0, fov=35.0)        # a wide view, most rays escape


def listed():
    return [
        # one tile of a progressive 2048^2 render, read back to host arrays: the smallest call
        dict(name="tile64_fp64", kind="tile", precision="fp64", width=64, height=64, image=2048, **FACE_ON),
        # an interactive preview: a small odd image, latency and launches count
        dict(name="preview_mixed", kind="image", precision="mixed", width=213, height=119, **WIDE),
        # an ordinary image in the reference precision
        dict(name="kerr512_fp64", kind="image", precision="fp64", width=512, height=512, **FACE_ON),
        # an odd-sized widescreen frame of the grazing camera, mixed precision
        dict(name="wide_mixed", kind="image", precision="mixed", width=1279, height=717, **EDGE_ON),
        # the headline image, both precisions
        dict(name="kerr2048_mixed", kind="image", precision="mixed", width=2048, height=2048, **FACE_ON),
        dict(name="kerr2048_fp64", kind="image", precision="fp64", width=2048, height=2048, **FACE_ON),
        # the charged hole in Boyer-Lindquist coordinates
        dict(name="kn1024", kind="image_bl", width=1024, height=1024, **CHARGED),
        # a scene of five holes
        dict(name="scene5_480x270", kind="multi", precision="fp64", holes=5, width=480, height=270, spin=0.7, r_obs=70.0,
             incl=65.0, fov=25.0),
        # the displayed frame: shaded, with the sky, read back to pinned pixels
        dict(name="frame1536_sky", kind="frame", precision="mixed", model="sky", width=1536, height=1536, **FACE_ON),
        # the volumetric torus around the grazing hole
        dict(name="torus_640x360", kind="frame", precision="fp64", model="torus", width=640, height=360, **EDGE_ON),
        # a table of cameras of uneven size in one launch
        dict(name="table40_mixed", kind="table", precision="mixed", bundles=40),
        # a burst of requests to the server: small and ordinary images, and a scene of 16 holes
        dict(name="server_burst", kind="server", requests=24, multi_fraction=0.125, most_side=448),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    def camera():
        return dict(spin=round(rng.uniform(0.0, 0.998), 3), r_obs=round(rng.uniform(30.0, 150.0), 1),
                    incl=round(rng.uniform(10.0, 85.0), 1), fov=round(rng.uniform(8.0, 35.0), 1))

    kind = rng.choice(["tile", "image", "image", "image", "image_bl", "multi", "frame", "frame", "table", "server"])
    if kind == "tile":
        return dict(kind="tile", precision=rng.choice(["fp64", "mixed"]), width=_log(rng, 32, 256),
                    height=_log(rng, 32, 256), image=rng.choice([512, 1024, 2048]), **camera())
    if kind == "image":
        precision = rng.choice(["fp64", "mixed"])
        return dict(kind="image", precision=precision, width=_log(rng, 100, 1500), height=_log(rng, 100, 1500), **camera())
    if kind == "image_bl":
        c = camera()
        c["spin"] = min(c["spin"], 0.9)
        return dict(kind="image_bl", charge=round(rng.uniform(0.0, 0.4), 2), width=_log(rng, 64, 800),
                    height=_log(rng, 64, 800), **c)
    if kind == "multi":
        return dict(kind="multi", precision=rng.choice(["fp64", "mixed"]), holes=rng.randint(2, 9), width=_log(rng, 64, 320),
                    height=_log(rng, 64, 240), **camera())
    if kind == "frame":
        model = rng.choice(["sky", "sky", "disk", "torus"])
        most = 280 if model == "torus" else 1400
        return dict(kind="frame", precision=rng.choice(["fp64", "mixed"]), model=model, width=_log(rng, 100, most),
                    height=_log(rng, 100, most), **camera())
    if kind == "table":
        return dict(kind="table", precision=rng.choice(["fp64", "mixed"]), bundles=rng.randint(4, 32))
    return dict(kind="server", requests=rng.randint(4, 20), multi_fraction=0.1, most_side=rng.choice([192, 256, 384]))


def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, 977])


def _precision(case):
    return relsim.PRECISION_MIXED if case.get("precision") == "mixed" else relsim.PRECISION_FP64


def _camera(case, seed):
    g = _rng(case, seed)
    kw = dict(spin=min(max(case["spin"] + g.uniform(-0.01, 0.01), 0.0), 0.998), r_obs=case["r_obs"] * g.uniform(0.98, 1.02),
              incl_deg=case["incl"] + g.uniform(-1.0, 1.0), phi_obs=g.uniform(-3.0, 3.0), fov_deg=case["fov"],
              width=case["width"], height=case["height"], precision=_precision(case))
    if case["kind"] == "image_bl":
        kw.update(metric_form=relsim.METRIC_BOYER_LINDQUIST, charge=case["charge"], precision=relsim.PRECISION_FP64)
    if case["kind"] == "tile":
        kw.update(width=case["image"], height=case["image"])
    cam = relsim.make_camera(**kw)
    if case["kind"] == "tile":  # a tile over the hole's neighbourhood
        span_x, span_y = case["image"] - case["width"], case["image"] - case["height"]
        cam.tile_origin_x, cam.tile_origin_y = int(span_x * g.uniform(0.35, 0.65)), int(span_y * g.uniform(0.35, 0.65))
        cam.tile_extent_x, cam.tile_extent_y = case["width"], case["height"]
    return cam


def _holes(case, seed):
    """The bodies beside the camera's hole: as the request stream places them, in a tighter box."""
    g = _rng(case, seed)
    g.uniform(size=8)
    th = math.radians(case["incl"])
    placed, out = [((0.0, 0.0, 0.0), 1.0)], []
    while len(out) < case["holes"] - 1:
        m, chi, z, ph = g.uniform(0.2, 1.0), g.uniform(0.0, 0.9), g.uniform(-1.0, 1.0), g.uniform(0.0, 2.0 * math.pi)
        s = math.sqrt(max(0.0, 1.0 - z * z))
        pos = tuple(float(v) for v in g.uniform(-20.0, 20.0, 3))
        if all(math.dist(pos, q) > 3.0 * (m + mq) for q, mq in placed):
            out.append(dict(position=pos, mass=m, spin_parameter=chi, axis=(s * math.cos(ph), s * math.sin(ph), z),
                            disk_outer_units=8.0))
            placed.append((pos, m))
    return out


def _moved(bundle, g):
    """A drawn bundle seen from elsewhere: its size and field of view stay."""
    return scenes.BundleDraw(bundle.side, min(bundle.spin * g.uniform(0.9, 1.0), 0.998), bundle.incl_deg + g.uniform(-2.0, 2.0),
                             bundle.r_obs * g.uniform(0.97, 1.03), bundle.fov_deg)


def _table(case, seed):
    g = _rng(case, seed)
    return [_moved(b, g).camera(_precision(case)) for b in scenes.bundle_table(case["bundles"], seed=0)]


def _requests(case, seed):
    """(camera, bodies) of the stream's requests no larger than the case's side, moved by the seed."""
    g, got = _rng(case, seed), []
    for r in scenes.request_stream(n=8 * case["requests"], multi_fraction=case["multi_fraction"]):
        if r.bundle.side <= (case["most_side"] // 2 if r.multi_source else case["most_side"]):
            got.append((_moved(r.bundle, g).camera(), scenes.rt_sources(r.sources) if r.multi_source else None))
        if len(got) == case["requests"]:
            break
    return got


# A program keeps one handle (and one server) for its life; a handle's shading is set once.
_kept = {}


def _tracer(model=None):
    if model not in _kept:
        tr = relsim.Tracer(0)
        if model is not None:
            tr.set_shading(relsim.shading(**{"sky": dict(sky_enabled=1), "disk": {}, "torus": dict(hydro_model=2)}[model]))
        _kept[model] = tr
    return _kept[model]


def _server():
    if "server" not in _kept:
        _kept["server"] = relsim.Server(0, relsim.server_config(record=["status", "r_hit", "g"]))
    return _kept["server"]


def prepare(case, seed):
    kind = case["kind"]
    state = dict(kind=kind)
    if kind == "server":
        reqs = _requests(case, seed)
        n = sum(relsim.window_rays(cam) for cam, _ in reqs)
        out = {"status": torch.empty(n, dtype=torch.int32).pin_memory(),
               "r_hit": torch.empty(n, dtype=torch.float64).pin_memory(),
               "g": torch.empty(n, dtype=torch.float64).pin_memory()}
        jobs, at = [], 0
        for cam, sources in reqs:
            rays = relsim.window_rays(cam)
            jobs.append((cam, {f: t[at:at + rays].numpy() for f, t in out.items()}, sources))
            at += rays
        state.update(jobs=jobs, out=out, server=_server())
        return state
    if kind == "table":
        cams = _table(case, seed)
        n = relsim.bundle_rays(cams)
        ro, out = relsim.device_ray_out(n, RECORD)
        state.update(cams=cams, n=n, ro=ro, out=out, tracer=_tracer())
        return state
    cam = _camera(case, seed)
    state["cam"] = cam
    if kind == "tile":
        state["tracer"] = _tracer()
        return state
    n = relsim.window_rays(cam)
    state["n"] = n
    if kind == "frame":
        pix = torch.empty(n, 8, dtype=torch.float32).pin_memory()
        state.update(tracer=_tracer(case["model"]), pix=pix,
                     out={"rgba": pix[:, 0:4], "redshift": pix[:, 4], "affine": pix[:, 5],
                          "flags_iterations": pix.view(torch.int32)[:, 6:8]})
        return state
    ro, out = relsim.device_ray_out(n, RECORD)
    state.update(tracer=_tracer(), ro=ro, out=out)
    if kind == "multi":
        state["sources"] = [relsim.make_source(**h) for h in _holes(case, seed)]
    return state


def run(state):
    kind = state["kind"]
    if kind == "tile":
        return state["tracer"].dispatch(state["cam"], fields=RECORD, pixels=False, tile=True)
    if kind == "table":
        state["tracer"].trace_bundles_device(state["cams"], state["ro"], None, state["n"])
    elif kind == "multi":
        state["tracer"].dispatch_multi_device(state["cam"], state["sources"], state["ro"], None, state["n"])
    elif kind == "frame":
        tr = state["tracer"]
        st = tr.lib.rt_dispatch(tr.handle, state["cam"], state["pix"].data_ptr(), None, state["n"], None)
        if st != relsim.RT_OK:
            raise relsim.RelsimError(st, tr.lib.rt_last_error(tr.handle).decode())
    elif kind == "server":
        srv = state["server"]
        ids = [srv.submit(cam, out=part, sources=sources)[0] for cam, part, sources in state["jobs"]]
        srv.wait(ids)
    else:
        state["tracer"].dispatch_device(state["cam"], state["ro"], None, state["n"])
    return state["out"]


def work(case):
    """Record bytes of each ray once, and the DP45 attempts its tolerance asks for (mean of these
    cameras) at the operations of one attempt with shared stages: 1,221 FLOP for the Kerr-Schild
    equations (about 1,400 for each source of a superposition), 1,598 for Boyer-Lindquist."""
    kind, mixed = case["kind"], case.get("precision") == "mixed"
    if kind == "table":
        rays = float(sum(b.side ** 2 for b in scenes.bundle_table(case["bundles"], seed=0)))
    elif kind == "server":
        rays = 0.17 * case["most_side"] ** 2 * case["requests"]  # mean of the stream's sides up to that one
        mixed = True
    else:
        rays = float(case["width"] * case["height"])
    per_ray = {"fp64": 114.0, "mixed": 52.0}["mixed" if mixed else "fp64"] * 1221.0
    size = 44.0
    if kind == "image_bl":
        per_ray = 185.0 * 1598.0
    elif kind == "multi":
        per_ray = (75.0 if mixed else 186.0) * 1400.0 * case["holes"]
    elif kind == "frame":
        size = 32.0
    elif kind == "server":
        size = 20.0
    return {"bytes": rays * size, "flops": rays * per_ray}


# ---------------------------------------------------------------------------
# The same rays in plain torch, 64 bits.

_C = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9], [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656], [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_E = [71 / 57600, 0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40]
_TOL = 1e-12


def _dev():
    return "cuda:0" if torch.cuda.is_available() else "cpu"


def _combine(y, h, ks, row):
    acc = sum(k * w for k, w in zip(ks, row) if w)
    return y + h * acc


def _dp(f, y, h, k1):
    ks = [k1]
    for row in _C:
        y5 = _combine(y, h, ks, row)
        ks.append(f(y5))
    return y5, ks[-1], h * sum(k * w for k, w in zip(ks, _E) if w)


def _isco(m, a):
    z1 = 1 + (1 - (a / m) ** 2) ** (1 / 3) * ((1 + abs(a) / m) ** (1 / 3) + (1 - abs(a) / m) ** (1 / 3))
    z2 = math.sqrt(3 * (a / m) ** 2 + z1 * z1)
    return m * (3 + z2 - math.copysign(1.0, a) * math.sqrt((3 - z1) * (3 + z1 + 2 * z2)))


def _redshift(m, a, r, lz):
    """1 / (u^t (1 - Omega L)) of the circular equatorial orbit, as the disk's redshift factor is clamped."""
    sm, sr = m ** 0.5, torch.sqrt(r)
    r15 = r * sr
    bracket = (r15 - 3 * m * sr + 2 * a * sm).clamp_min(1e-9)
    den = (r15 + a * sm) / (torch.sqrt(r15) * torch.sqrt(bracket)) * (1 - sm / (r15 + a * sm) * lz)
    return torch.where(den.abs() > 1e-9, (1 / den).clamp(0.05, 4.0), torch.ones_like(den))


def _captured_for_certain(m, a, q2, rh, xi, eta):
    """Whether the radial potential keeps 1e-4 M off zero everywhere outside the horizon (impact parameter)."""
    K = eta + (xi - a) ** 2
    P, Q = a * a - xi * xi - eta, 2 * m * K
    # stationary points of r^4 + P r^2 + Q r + R0: the roots of r^3 + (P / 2) r + Q / 4
    p, q = P / 2, Q / 4
    disc = (q / 2) ** 2 + (p / 3) ** 3
    amp = 2 * torch.sqrt((-p / 3).clamp_min(0))
    th = torch.acos((3 * q / (p * amp)).clamp(-1, 1)) / 3
    sq = torch.sqrt(disc.clamp_min(0))
    cbrt = lambda v: torch.sign(v) * v.abs() ** (1 / 3)  # noqa: E731
    single = cbrt(-q / 2 + sq) + cbrt(-q / 2 - sq)
    best = torch.full_like(p, math.inf)
    at = torch.zeros_like(p)
    for k in range(3):
        r = torch.where(disc < 0, amp * torch.cos(th - 2 * math.pi * k / 3), single)
        for _ in range(2):
            r = r - (r ** 3 + p * r + q) / (3 * r * r + p)
        R = ((r * r + P) * r + Q) * r - a * a * eta - q2 * K
        use = (r > rh) & (12 * r * r + 2 * P > 0) & (R < best)
        best, at = torch.where(use, R, best), torch.where(use, r, at)
    delta = (at * at - 2 * m * at + a * a + q2).clamp_min(1e-30)
    return ~torch.isfinite(best) | (best / delta / (2 * torch.sqrt((eta + xi * xi).clamp_min(1e-30))) > 1e-4)


class _Hole:
    """A Kerr hole of unit mass in Kerr-Schild form; the spin is one number or one per ray."""

    def __init__(self, a):
        self.a = a
        self.rh = 1 + (1 - a * a) ** 0.5

    def rows(self, keep):
        return _Hole(self.a[keep])

    def geometry(self, x):
        """r, r^2, r^4 + a^2 z^2, 1 / (r^2 + a^2), the scalar h and the null direction k."""
        a2 = self.a * self.a
        z2 = x[2] * x[2]
        d = x[0] * x[0] + x[1] * x[1] + z2 - a2
        r2 = 0.5 * (d + torch.sqrt(d * d + 4 * a2 * z2))
        r = torch.sqrt(r2)
        den = r2 * r2 + a2 * z2
        w = 1 / (r2 + a2)
        k = torch.stack([(r * x[0] + self.a * x[1]) * w, (r * x[1] - self.a * x[0]) * w, x[2] / r])
        return r, r2, den, w, r2 * r / den, k

    def radius(self, x):
        return self.geometry(x)[0]

    def inward(self, y, w):
        """dr/dlambda along w."""
        r, r2, den, _, _, _ = self.geometry(y[:3])
        return (r2 * r * (y[0] * w[0] + y[1] * w[1]) + r * (r2 + self.a * self.a) * y[2] * w[2]) / den

    def flow(self, y):
        """(dx, dp) of H = |p|^2 / 2 - 1 / 2 - h s^2, s = 1 + k.p."""
        x, p = y[:3], y[3:]
        a, a2 = self.a, self.a * self.a
        r, r2, den, w, h, k = self.geometry(x)
        s = 1 + (k * p).sum(0)
        dr = torch.stack([r2 * r * x[0], r2 * r * x[1], r * (r2 + a2) * x[2]]) / den
        A = w * ((x[0] - 2 * r * k[0]) * p[0] + (x[1] - 2 * r * k[1]) * p[1]) - x[2] * p[2] / r2
        B = torch.stack([w * (r * p[0] - a * p[1]), w * (r * p[1] + a * p[0]), p[2] / r])
        dh = r2 * (3 * a2 * x[2] * x[2] - r2 * r2) / (den * den)
        dp = dr * (s * s * dh + 2 * h * s * A) + 2 * h * s * B
        dp[2] -= s * s * 2 * r2 * r * a2 * x[2] / (den * den)
        return torch.cat([p - 2 * h * s * k, dp])


def _directions(cam, tile):
    W, H = cam.screen_width, cam.screen_height
    x0, y0, w, h = (cam.tile_origin_x, cam.tile_origin_y, cam.tile_extent_x, cam.tile_extent_y) if tile else (0, 0, W, H)
    px = torch.arange(x0, x0 + w, dtype=torch.float64, device=_dev()) + 0.5
    py = torch.arange(y0, y0 + h, dtype=torch.float64, device=_dev()) + 0.5
    t = math.tan(0.5 * cam.field_of_view_rad)
    u, v = torch.meshgrid((2 * px / W - 1) * (W / H) * t, (1 - 2 * py / H) * t, indexing="xy")
    e = [torch.tensor(list(k)[1:], dtype=torch.float64, device=_dev())[:, None] for k in (cam.tetrad_e1, cam.tetrad_e2, cam.tetrad_e3)]
    d = e[0] + u.reshape(1, -1) * e[1] + v.reshape(1, -1) * e[2]
    return d / d.norm(dim=0)


def _start(hole, x0, d):
    """Null covectors (p_t = -1) of the static observer at x0 looking along d."""
    at = torch.tensor(x0, dtype=torch.float64, device=d.device)[:, None]
    _, _, _, _, h, k = hole.geometry(at)
    ell = torch.cat([torch.ones(1, dtype=torch.float64), k[:, 0].cpu()])
    g = torch.diag(torch.tensor([-1.0, 1, 1, 1], dtype=torch.float64)) + 2 * float(h[0]) * torch.outer(ell, ell)
    u = torch.zeros(4, dtype=torch.float64)
    u[0] = 1 / math.sqrt(-float(g[0, 0]))
    e = []
    for j in range(3):
        v = torch.zeros(4, dtype=torch.float64)
        v[1 + j] = 1
        v = v + (u @ g @ v) * u
        for q in e:
            v = v - (v @ g @ q) * q
        e.append(v / torch.sqrt(v @ g @ v))
    low = (torch.stack([u] + e) @ g).to(d.device)
    p = low[0][:, None] - low[1:].T @ d
    return torch.cat([at.expand(3, d.shape[1]), p[1:] / -p[0]])


def _to(f, y, dq, q_rate):
    """One step along the coordinate q (dy/dq = f / (dq/dlambda)) by dq."""
    def along(v):
        w = f(v)
        return w / q_rate(v, w)

    half = 0.5 * dq
    for _ in range(2):
        y = _dp(along, y, half, along(y))[0]
    return y


def _turn(p, q):
    return torch.atan2(p[0] * q[1] - p[1] * q[0], p[0] * q[0] + p[1] * q[1])


def _trace_ks(hole, y, r_in, cam):
    """Kerr-Schild rays to their end: (state, class, azimuth turned through, L)."""
    n = y.shape[1]
    end, cls, turned = torch.zeros_like(y), torch.zeros(n, dtype=torch.int64, device=y.device), torch.zeros_like(y[0])
    lz = y[0] * y[4] - y[1] * y[3]
    r = hole.radius(y)
    cos = y[2] / r
    sin2 = 1 - cos * cos
    pth = (y[0] * y[3] + y[1] * y[4]) * cos / torch.sqrt(sin2) - r * torch.sqrt(sin2) * y[5]
    eta = pth * pth + cos * cos * (lz * lz / sin2 - hole.a ** 2)
    sure = _captured_for_certain(1.0, hole.a, 0.0, hole.rh, lz, eta)
    idx, h, turn, k1 = torch.arange(n, device=y.device), torch.full_like(r, -1.0), torch.zeros_like(r), hole.flow(y)
    for _ in range(6000):
        if not y.shape[1]:
            break
        h = torch.maximum(h, -cam.step_cap_fraction * (r - hole.rh).clamp_min(0.01))
        y5, k7, err = _dp(hole.flow, y, h, k1)
        e = (err.abs() / (_TOL + _TOL * torch.maximum(y.abs(), y5.abs()))).amax(0).clamp_min(1e-10)
        ok = e <= 1
        h = h * (0.9 * e ** -0.2).clamp(0.2, 5.0)
        r5 = hole.radius(y5)
        done = torch.zeros_like(ok)

        def finish(rows, state, code):
            end[:, idx[rows]], cls[idx[rows]] = state, code
            turned[idx[rows]] = turn[rows] + _turn(y[:, rows], state)
            done[rows] = True

        hit = ok & (y[2] * y5[2] <= 0) & (y[2] != y5[2])
        if bool(hit.any()):
            i = hit.nonzero()[:, 0]
            one = hole.rows(i)
            root = _to(one.flow, y5[:, i], -y5[2, i], lambda s, w: w[2])
            rr = one.radius(root)
            on = (rr >= r_in[i]) & (rr <= cam.disk_outer_radius) & (rr > 1.02 * one.rh)
            finish(i[on], root[:, on], 3)
        for code, test, target in ((1, r5 < cam.capture_scale * hole.rh, cam.capture_scale * hole.rh),
                                   (2, r5 > cam.escape_radius, torch.full_like(r5, cam.escape_radius)),
                                   (1, sure & (hole.inward(y5, k7) > 0) & (r5 < r_in), r_in)):
            m = ok & ~done & test
            if bool(m.any()):
                i = m.nonzero()[:, 0]
                one = hole.rows(i)
                finish(i, _to(one.flow, y5[:, i], target[i] - r5[i], one.inward), code)
        step = ok & ~done
        turn = torch.where(step, turn + _turn(y, y5), turn)
        y, k1, r = torch.where(step, y5, y), torch.where(step, k7, k1), torch.where(step, r5, r)
        if bool(done.any()):
            keep = (~done).nonzero()[:, 0]
            hole, y, k1, r, r_in, sure = hole.rows(keep), y[:, keep], k1[:, keep], r[keep], r_in[keep], sure[keep]
            h, turn, idx = h[keep], turn[keep], idx[keep]
    return end, cls, turned, lz


def _exact_ks(cams, tile=False):
    ys, per_ray = [], []
    for cam in cams:
        _, r, th, ph = list(cam.observer_position)
        a = cam.metric_spin
        x0 = ((r * math.cos(ph) - a * math.sin(ph)) * math.sin(th), (r * math.sin(ph) + a * math.cos(ph)) * math.sin(th),
              r * math.cos(th))
        ys.append(_start(_Hole(a), x0, _directions(cam, tile)))
        numbers = torch.tensor([a, _isco(1.0, a), ph + math.atan2(a, r)], dtype=torch.float64, device=_dev())
        per_ray.append(numbers[:, None].expand(3, ys[-1].shape[1]))
    a, r_in, phi0 = torch.cat(per_ray, 1)
    hole = _Hole(a)
    end, cls, turned, lz = _trace_ks(hole, torch.cat(ys, 1), r_in, cams[0])
    r, hit = hole.radius(end), cls == 3
    return {"r": r, "theta": torch.atan2(torch.sqrt((r * r - end[2] ** 2).clamp_min(0)), end[2]),
            "phi": phi0 + turned - torch.atan2(a, r), "r_hit": torch.where(hit, r, math.nan),
            "g": torch.where(hit, _redshift(1.0, a, r, lz), 1.0)}


def _exact_bl(case, seed):
    """Kerr-Newman rays in Mino time: H = (D p_r^2 + p_th^2 - P^2 / D + (L / s - a E s)^2) / 2, E = 1."""
    cam = _camera(case, seed)
    _, r0, th0, ph0 = list(cam.observer_position)
    a, q2 = cam.metric_spin, cam.metric_charge ** 2
    d = _directions(cam, False)
    st, ct, sp, cp = math.sin(th0), math.cos(th0), math.sin(ph0), math.cos(ph0)
    er, et, ep = [torch.tensor(v, dtype=torch.float64, device=d.device) for v in
                  ((st * cp, st * sp, ct), (ct * cp, ct * sp, -st), (-sp, cp, 0.0))]
    nr, nt, np_ = er @ d, et @ d, ep @ d
    sig, dl = r0 * r0 + a * a * ct * ct, r0 * r0 - 2 * r0 + a * a + q2
    F = (2 * r0 - q2) / sig
    gtp, gpp = -a * st * st * F, st * st * (r0 * r0 + a * a + a * a * st * st * F)
    om = -gtp / gpp
    alpha = math.sqrt(-(F - 1.0 + om * gtp))
    ut, ur, uth = 1 / alpha, -nr * math.sqrt(dl / sig), -nt / math.sqrt(sig)
    up = om / alpha - np_ / math.sqrt(gpp)
    E, L = -((F - 1.0) * ut + gtp * up), gtp * ut + gpp * up
    L, pr, pth = L / E, ur * sig / dl / E, uth * sig / E
    eta = pth ** 2 + ct * ct * (L * L / st ** 2 - a * a)
    rh = 1 + math.sqrt(1 - a * a - q2)
    sure = _captured_for_certain(1.0, a, q2, rh, L, eta)
    n = L.shape[0]
    full = lambda v: torch.full((n,), v, dtype=torch.float64, device=d.device)  # noqa: E731
    y = torch.stack([full(r0), full(th0), full(ph0), pr, pth])
    r_in, r_out = _isco(1.0, a), cam.disk_outer_radius
    end, cls = torch.zeros_like(y), torch.zeros(n, dtype=torch.int64, device=y.device)
    idx, h, ell = torch.arange(n, device=y.device), full(-1e-5), L

    def flow(s, l):
        r, th, p, pt = s[0], s[1], s[3], s[4]
        D, dD = r * r - 2 * r + a * a + q2, 2 * r - 2
        P = r * r + a * a - a * l
        sn, cs = torch.sin(th), torch.cos(th)
        w = l / sn - a * sn
        return torch.stack([D * p, pt, a * P / D - a + l / (sn * sn),
                            -0.5 * dD * p * p + 2 * r * P / D - 0.5 * P * P * dD / (D * D), w * (l / (sn * sn) + a) * cs])

    k1 = flow(y, ell)
    for _ in range(6000):
        if not y.shape[1]:
            break
        f = lambda s: flow(s, ell)  # noqa: E731,B023
        y5, k7, err = _dp(f, y, h, k1)
        e = (err.abs() / (1e-13 + _TOL * torch.maximum(y.abs(), y5.abs()))).amax(0).nan_to_num(1e9, 1e9, 1e9).clamp_min(1e-10)
        ok = (e <= 1) & (y5[0] > rh) & ((y5[0] - y[0]).abs() < 0.25 * (y[0] - rh))
        h = torch.where(ok, h * (0.9 * e ** -0.2).clamp(0.2, 2.0), h * (0.9 * e ** -0.2).clamp(0.1, 0.5))
        done = torch.zeros_like(ok)
        c0, c1 = y[1] - 0.5 * math.pi, y5[1] - 0.5 * math.pi
        hit = ok & (c0 * c1 <= 0) & (c0 != c1)
        if bool(hit.any()):
            i = hit.nonzero()[:, 0]
            root = _to(lambda s: flow(s, ell[i]), y5[:, i], -c1[i], lambda s, w: w[1])  # noqa: B023
            on = (root[0] >= r_in) & (root[0] <= r_out) & (root[0] > 1.02 * rh)
            end[:, idx[i[on]]], cls[idx[i[on]]] = root[:, on], 3
            done[i[on]] = True
        for code, test, target in ((1, y5[0] < cam.capture_scale * rh, cam.capture_scale * rh), (2, y5[0] > cam.escape_radius, cam.escape_radius),
                                   (1, sure & (k7[0] > 0) & (y5[0] < r_in), r_in)):
            m = ok & ~done & test
            if bool(m.any()):
                i = m.nonzero()[:, 0]
                end[:, idx[i]] = _to(lambda s: flow(s, ell[i]), y5[:, i], target - y5[0, i], lambda s, w: w[0])  # noqa: B023
                cls[idx[i]] = code
                done[i] = True
        y, k1 = torch.where(ok, y5, y), torch.where(ok, k7, k1)
        if bool(done.any()):
            keep = (~done).nonzero()[:, 0]
            y, k1, h, idx, ell, sure = y[:, keep], k1[:, keep], h[keep], idx[keep], ell[keep], sure[keep]
    hit = cls == 3
    return {"r": end[0], "theta": end[1], "phi": end[2], "r_hit": torch.where(hit, end[0], math.nan),
            "g": torch.where(hit, _redshift(1.0, a, end[0], L), 1.0)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "table":
        return {"status": None, **_exact_ks(_table(case, seed))}
    if kind in ("image", "tile"):
        return {"status": None, **_exact_ks([_camera(case, seed)], kind == "tile")}
    if kind == "image_bl":
        return {"status": None, **_exact_bl(case, seed)}
    # Shaded pixels hold the procedural sky and disk patterns.  A multi-source ray starts off the zero
    # set of the superposed Hamiltonian and is projected onto it at its first accepted step, wherever
    # that ends: it has no value apart from the step sequence; so a burst of requests has none either.
    return None
