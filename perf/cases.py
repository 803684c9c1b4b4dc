"""What is measured of this framework: table builds, alone and in batches, and the use of the tables.

Each case is a dict of plain values. Kinds:
  build     Atmosphere.build of one atmosphere, its three tables as tensors
  dump      the same with half storage and the scattering table exported to the host
  batch     build_batch of several atmospheres, all their tables as tensors
  sky       the sky pass over finished tables, one image
  lighting  sun and sky irradiance at a batch of surface points

Table sizes are those of this repository's configurations (smoke, dump,
default, the half and double classes) or generic; atmospheres are drawn from
the seed, either near Earth ("earth") or over the planets that the batch
workloads cover ("wide").
"""
import math
import random

import numpy as np
import torch

from fuzzyblue_gb300.api import Atmosphere, Builder, build_batch
from fuzzyblue_gb300.params import (PRECISION_MIXED, PRECISION_PLAIN, STORAGE_F16, STORAGE_F32, DensityProfile,
                                    DensityProfileLayer, Parameters)
from fuzzyblue_gb300.render import DrawParameters

SIZE_KEYS = ("tr_mu", "tr_r", "tr_steps", "ir_mus", "ir_r", "sc_r", "sc_mu", "sc_mus", "sc_nu")
SIZES = {
    "smoke": (256, 64, 500, 64, 16, 8, 32, 8, 2),
    "dump": (256, 64, 500, 64, 16, 16, 64, 16, 4),
    "default": (256, 64, 500, 64, 16, 32, 128, 32, 8),
    "half": (128, 32, 500, 64, 16, 16, 64, 16, 4),
    "double": (512, 128, 2000, 128, 32, 64, 256, 64, 16),
}
DENSITY_SAMPLES = 16
IRRADIANCE_SAMPLES = 32
STEPS = 50  # of single and of multiple scattering


def _sized(name, cls, **kw):
    return dict(zip(SIZE_KEYS, SIZES[cls]), name=name, **kw)


def listed():
    return [
        # the smallest call: the reduced atmosphere of the integration test, where launches and latency count
        _sized("smoke_plain", "smoke", kind="build", order=4, precision="plain", planet="earth"),
        # the table dump example's sizes, written as half tables: build, then export to the host
        _sized("dump_half", "dump", kind="dump", order=4, precision="plain", planet="earth"),
        # an application that builds its one sky at start: the default parameters, in either precision
        _sized("default_plain", "default", kind="build", order=4, precision="plain", planet="earth"),
        _sized("default_mixed", "default", kind="build", order=4, precision="mixed", planet="wide"),
        # one bounce beyond single scattering, for a sky that is rebuilt while parameters are edited
        _sized("preview_plain", "default", kind="build", order=2, precision="plain", planet="earth"),
        # sizes that divide nothing
        dict(name="odd_mixed", kind="build", tr_mu=201, tr_r=51, tr_steps=333, ir_mus=47, ir_r=13, sc_r=21, sc_mu=90,
             sc_mus=27, sc_nu=7, order=5, precision="mixed", planet="wide"),
        # four times the default resolution, for a reference rendering
        _sized("double_mixed", "double", kind="build", order=4, precision="mixed", planet="wide"),
        # many planets of one class at once: at default sizes, and small ones of uneven order
        dict(name="uniform_batch", kind="batch", cls="default", count=16, order=4, precision="mixed"),
        dict(name="half_batch", kind="batch", cls="half", count=20, order=0, precision="mixed"),
        # a mixture of classes and orders, as a server's queue holds it
        dict(name="uneven_batch", kind="batch", cls="mixed", count=12, order=0, precision="mixed"),
        # a frame of the sky behind a scene, and the light on its surface points
        dict(name="sky_1080p", kind="sky", width=1920, height=1080, depth=True),
        dict(name="lighting", kind="lighting", points=200_003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "batch", "batch", "dump", "sky", "lighting"])
    if kind == "sky":
        return dict(kind=kind, width=_log(rng, 160, 2560), height=_log(rng, 90, 1440), depth=rng.random() < 0.6)
    if kind == "lighting":
        return dict(kind=kind, points=_log(rng, 1000, 1_000_000))
    if kind == "batch":
        cls = rng.choice(["default", "half", "mixed"])
        most = {"default": 18, "half": 20, "mixed": 12}[cls]
        return dict(kind=kind, cls=cls, count=_log(rng, 2, most), order=rng.choice([0, 2, 3, 4]),
                    precision=rng.choice(["mixed", "mixed", "plain"]))
    while True:
        c = dict(kind=kind, tr_mu=_log(rng, 48, 512), tr_r=_log(rng, 16, 128), tr_steps=_log(rng, 100, 2000),
                 ir_mus=_log(rng, 16, 128), ir_r=_log(rng, 4, 32), sc_r=_log(rng, 6, 64), sc_mu=2 * _log(rng, 8, 128),
                 sc_mus=_log(rng, 6, 64), sc_nu=_log(rng, 2, 16), order=rng.randint(1, 6),
                 precision=rng.choice(["plain", "mixed"]), planet="earth")
        if kind == "build" and c["precision"] == "mixed" and rng.random() < 0.6:
            c["planet"] = "wide"
        if c["precision"] == "plain":
            # where the packed slices have odd widths, the 32-bit texture coordinates of the plain mode bleed
            # into the next slice: it is used at the powers of two that the repository's configurations have
            c["sc_mus"], c["sc_nu"] = 2 ** rng.randint(3, 6), 2 ** rng.randint(1, 4)
        # no more than four times the default resolution's work at four orders
        if c["sc_r"] * c["sc_mu"] * c["sc_mus"] * c["sc_nu"] * c["order"] <= 64 * 256 * 64 * 16 * 4:
            return c


# ------------------------------------------------------------- inputs ---
EARTH_RAYLEIGH = (0.005802, 0.013558, 0.033100)
EARTH_OZONE = (6.5e-4, 1.881e-3, 8.5e-5)


def _f32(v):
    return tuple(float(np.float32(x)) for x in v) if isinstance(v, tuple) else float(np.float32(v))


def _planet(rng, planet):
    """The physical parameters of one atmosphere, lengths in km, as 32-bit values."""
    wide = planet == "wide"

    def logu(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    bottom = rng.uniform(3000.0, 8000.0) if wide else rng.uniform(6200.0, 6500.0)
    top = bottom + (rng.uniform(40.0, 120.0) if wide else rng.uniform(58.0, 80.0))
    h_r = rng.uniform(4.0, 12.0) if wide else rng.uniform(7.0, 9.0)
    h_m = rng.uniform(0.5, 3.0) if wide else rng.uniform(1.0, 1.5)
    f_r = logu(0.2, 5.0) if wide else logu(0.7, 1.4)
    mie = logu(1e-3, 5e-2) if wide else logu(2e-3, 8e-3)
    g = rng.uniform(0.6, 0.9) if wide else rng.uniform(0.7, 0.85)
    f_o = rng.uniform(0.0, 3.0) if wide else rng.uniform(0.5, 1.5)
    q = dict(
        solar=(1.474, 1.850, 1.91198), sun_radius=0.004675, bottom=bottom, top=top,
        rayleigh=tuple(f_r * c for c in EARTH_RAYLEIGH), mie_sca=(mie,) * 3,
        mie_ext=(mie / rng.uniform(0.8, 1.0),) * 3, g=g, albedo=(rng.uniform(0.02, 0.3),) * 3,
        absorption=tuple(f_o * c for c in EARTH_OZONE), mu_s_min=-0.207912, scale_r=-1.0 / h_r, scale_m=-1.0 / h_m)
    return {k: _f32(v) for k, v in q.items()}


def _parameters(q, s, order, precision, storage=STORAGE_F32):
    def exponential(scale):
        return DensityProfile([DensityProfileLayer(), DensityProfileLayer(exp_term=1.0, exp_scale=scale)])

    return Parameters(
        order=order, transmittance_mu_size=s["tr_mu"], transmittance_r_size=s["tr_r"], scattering_r_size=s["sc_r"],
        scattering_mu_size=s["sc_mu"], scattering_mu_s_size=s["sc_mus"], scattering_nu_size=s["sc_nu"],
        irradiance_mu_s_size=s["ir_mus"], irradiance_r_size=s["ir_r"], transmittance_steps=s["tr_steps"],
        solar_irradiance=q["solar"], sun_angular_radius=q["sun_radius"], bottom_radius=q["bottom"],
        top_radius=q["top"], rayleigh_density=exponential(q["scale_r"]), rayleigh_scattering=q["rayleigh"],
        mie_density=exponential(q["scale_m"]), mie_scattering=q["mie_sca"], mie_extinction=q["mie_ext"],
        mie_phase_function_g=q["g"], absorbtion_extinction=q["absorption"], ground_albedo=q["albedo"],
        mu_s_min=q["mu_s_min"], precision=PRECISION_MIXED if precision == "mixed" else PRECISION_PLAIN,
        storage=storage)


def _requests(case, seed):
    """(physical parameters, sizes, order) of every atmosphere of a build, dump or batch."""
    rng = random.Random(seed)
    if case["kind"] != "batch":
        return [(_planet(rng, case["planet"]), {k: case[k] for k in SIZE_KEYS}, case["order"])]
    got = []
    for i in range(case["count"]):
        cls = ("default", "half", "double")[i % 3] if case["cls"] == "mixed" else case["cls"]
        # a batch in plain precision holds Earth-like planets, where 32 bits are enough
        q = _planet(rng, "wide" if case["precision"] == "mixed" else "earth")
        order = rng.randint(2, 8)
        got.append((q, dict(zip(SIZE_KEYS, SIZES[cls])), case["order"] or order))
    return got


# Of the sky and lighting cases: the atmosphere, the camera and the points.
def _scene(case, seed):
    rng = random.Random(seed)
    q = _planet(rng, "earth")
    elevation, azimuth = rng.uniform(0.05, 1.2), rng.uniform(-0.6, 0.6)
    sun = np.array([math.cos(elevation) * math.cos(azimuth), math.sin(elevation), math.cos(elevation) * math.sin(azimuth)])
    return q, dict(zip(SIZE_KEYS, SIZES["dump"])), rng.uniform(0.2, 3.0), sun / np.linalg.norm(sun)


def _camera(case, q, altitude, sun):
    """The camera looks along x, slightly down, y up; (0, bottom, 0) is below it."""
    return DrawParameters.look_at((0.0, q["bottom"] + altitude, 0.0), (1.0, -0.05, 0.1), (0.0, 1.0, 0.0), 60.0,
                                  case["width"] / case["height"], sun)


def _depth(case, seed):
    """A depth image: sky (0) above a rough skyline, below it surfaces some hundred metres to 30 km away."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["height"], case["width"]
    distance = 300.0 * torch.exp(torch.rand((h, w), generator=g, device="cuda") * math.log(100.0))
    skyline = 0.35 + 0.2 * torch.rand((1, w), generator=g, device="cuda")
    y = (torch.arange(h, device="cuda").reshape(h, 1) + 0.5) / h
    return torch.where(y > skyline, 0.1 / distance, torch.zeros_like(distance)).contiguous()


def _points(case, q, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["points"]
    p = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    p = p / p.norm(dim=1, keepdim=True)
    normal = p + 0.5 * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    normal = normal / normal.norm(dim=1, keepdim=True)
    # up to 9 km above the ground
    p = p * (q["bottom"] + 0.01 + 9.0 * torch.rand((n, 1), generator=g, device="cuda", dtype=torch.float64))
    return p.float().contiguous(), normal.float().contiguous()


_builder = None


def _the_builder():
    global _builder
    if _builder is None:
        _builder = Builder(0)
    return _builder


def prepare(case, seed):
    builder = _the_builder()
    state = {"case": case, "builder": builder}
    if case["kind"] in ("sky", "lighting"):
        q, sizes, altitude, sun = _scene(case, seed)
        pending = Atmosphere.build(builder, _parameters(q, sizes, 4, "mixed"))
        state["atmosphere"] = pending.take()  # waits for the tables
        pending.release()
        if case["kind"] == "sky":
            state["draw"] = _camera(case, q, altitude, sun)
            state["depth"] = _depth(case, seed) if case["depth"] else None
        else:
            state["points"], state["normals"] = _points(case, q, seed)
            state["sun"] = tuple(float(x) for x in sun)
        return state
    storage = STORAGE_F16 if case["kind"] == "dump" else STORAGE_F32
    state["params"] = [_parameters(q, s, order, case["precision"], storage) for q, s, order in _requests(case, seed)]
    return state


def _tables(atmosphere):
    return {k: torch.as_tensor(v, device="cuda") for k, v in atmosphere.device_views().items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sky":
        color, through = state["atmosphere"].render_sky(state["draw"], case["width"], case["height"], depth=state["depth"])
        return {"radiance": color, "transmittance": through}
    if kind == "lighting":
        sun, sky = state["atmosphere"].sun_and_sky_irradiance(state["points"], state["normals"], state["sun"])
        return {"sun": sun, "sky": sky}
    if kind == "batch":
        pending = build_batch(state["builder"], state["params"])
        pending.acquire(torch.cuda.current_stream())
        return [_tables(pending.atmosphere(i)) for i in range(len(state["params"]))]
    pending = Atmosphere.build(state["builder"], state["params"][0])
    pending.acquire(torch.cuda.current_stream())
    tables = _tables(pending.atmosphere())
    if kind == "dump":
        tables["scattering"] = pending.atmosphere().export_scattering_f16()
    return tables


def _texels(s):
    return s["sc_r"] * s["sc_mu"] * s["sc_mus"] * s["sc_nu"]


def work(case):
    """Bytes: the tables written once. Operations: one multiply-add for each channel of each sample or
    direction of the quadratures that define the tables."""
    if case["kind"] == "sky":
        n = case["width"] * case["height"]
        tables = 16 * (_texels(dict(zip(SIZE_KEYS, SIZES["dump"]))) + 256 * 64)
        return {"bytes": n * (36 if case["depth"] else 32) + tables, "flops": n * (2 if case["depth"] else 1) * 2 * 4 * 16}
    if case["kind"] == "lighting":
        return {"bytes": case["points"] * 48 + 16 * (256 * 64 + 64 * 16), "flops": case["points"] * 2 * 3 * 8}
    size = flops = 0
    for _, s, order in _requests(case, 0):
        ntr, nir, nsc = s["tr_mu"] * s["tr_r"], s["ir_mus"] * s["ir_r"], _texels(s)
        size += 16 * (ntr + nir) + (8 if case["kind"] == "dump" else 16) * nsc
        flops += 6 * ntr * (s["tr_steps"] + 1) + 12 * nsc * (STEPS + 1)
        flops += (order - 1) * 6 * (nsc * (2 * DENSITY_SAMPLES * DENSITY_SAMPLES + STEPS + 1)
                                    + nir * IRRADIANCE_SAMPLES * IRRADIANCE_SAMPLES)
    return {"bytes": size, "flops": flops}


# ------------------------------------------- the tables in 64 bits ---
# The quadratures that define the tables, in plain torch. Samples along a ray
# are weighted by the trapezoid rule; tables are read with linear
# interpolation between texel centres.
F = torch.float64


def _lerp_axis(t, n):
    t = t.clamp(0.0, n - 1.0)
    i = t.floor().clamp(max=max(n - 2, 0)).long()
    return i, t - i


class _Exact:
    def __init__(self, q, s, order):
        self.q, self.s, self.order = q, s, order
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.R, self.T = q["bottom"], q["top"]
        self.H2 = (self.T - self.R) * (self.T + self.R)
        self.H = math.sqrt(self.H2)

    def vec(self, v):
        return torch.tensor(v, dtype=F, device=self.dev)

    def grid(self, n):
        return torch.arange(n, dtype=F, device=self.dev)

    # --- geometry; q = r^2 - bottom^2 and p = r mu keep what cancels apart
    def top_distance(self, q, p):
        root = (p * p + (self.H2 - q)).clamp(min=0).sqrt()
        return torch.where(p > 0, (self.H2 - q) / (p + root), root - p).clamp(min=0)

    def ground_distance(self, q, p):
        root = (p * p - q).clamp(min=0).sqrt()
        return (-p - root).clamp(min=0)

    def density(self, scale, h):
        return torch.exp(scale * h).clamp(0.0, 1.0)

    def ozone(self, h):
        below = (np.float32(0.066667).item() * h + np.float32(-0.666667).item()).clamp(0.0, 1.0)
        above = (np.float32(-0.066667).item() * h + np.float32(2.666667).item()).clamp(0.0, 1.0)
        return torch.where(h < 25.0, below, above)

    def altitude(self, q):
        return q / ((q + self.R * self.R).sqrt() + self.R)

    # --- transmittance
    def build_transmittance(self):
        s = self.s
        rho = (self.H * self.grid(s["tr_r"]) / (s["tr_r"] - 1)).reshape(-1, 1)
        q = rho * rho
        r = (q + self.R ** 2).sqrt()
        lo, hi = (self.H2 - q) / (self.T + r), rho + self.H
        d = lo + (self.grid(s["tr_mu"]) / (s["tr_mu"] - 1)).reshape(1, -1) * (hi - lo)
        p = torch.where(d == 0, r.expand_as(d), (self.H2 - q - d * d) / (2 * d))
        p = torch.minimum(torch.maximum(p, -r), r)
        n = s["tr_steps"]
        dx = self.top_distance(q, p) / n
        lengths = [0, 0, 0]
        for first in range(0, n + 1, 256):
            k = torch.arange(first, min(first + 256, n + 1), dtype=F, device=self.dev)
            w = torch.where((k == 0) | (k == n), 0.5, 1.0)
            k = k * dx[..., None]
            h = self.altitude((q[..., None] + k * (2 * p[..., None] + k)).clamp(min=0))
            for i, y in enumerate((self.density(self.q["scale_r"], h), self.density(self.q["scale_m"], h), self.ozone(h))):
                lengths[i] = lengths[i] + (w * y).sum(-1) * dx
        depth = sum(l[..., None] * self.vec(self.q[c]) for l, c in zip(lengths, ("rayleigh", "mie_ext", "absorption")))
        self.tr = torch.exp(-depth)

    def to_top(self, q, p):
        s = self.s
        q = q.clamp(0.0, self.H2)
        r, rho = (q + self.R ** 2).sqrt(), q.sqrt()
        lo, hi = (self.H2 - q) / (self.T + r), rho + self.H
        x, fx = _lerp_axis((self.top_distance(q, p) - lo) / (hi - lo) * (s["tr_mu"] - 1), s["tr_mu"])
        y, fy = _lerp_axis(rho / self.H * (s["tr_r"] - 1), s["tr_r"])
        flat, w = self.tr.reshape(-1, 3), s["tr_mu"]
        fx, fy, at = fx[..., None], fy[..., None], y * w + x
        near = flat[at] * (1 - fx) + flat[at + 1] * fx
        return near * (1 - fy) + (flat[at + w] * (1 - fx) + flat[at + w + 1] * fx) * fy

    def along(self, q, p, d, ground):
        """The point at distance d, and the transmittance to it."""
        qd, pd = (q + d * (2 * p + d)).clamp(0.0, self.H2), p + d
        rd = (qd + self.R ** 2).sqrt()
        pd = torch.minimum(torch.maximum(pd, -rd), rd)
        sign = torch.where(ground, -1.0, 1.0).to(F)
        a, b = self.to_top(q + 0 * d, sign * p + 0 * d), self.to_top(qd, sign * pd)
        g = ground[..., None].expand(a.shape)
        through = torch.where(g, b, a) / torch.where(g, a, b)
        return qd, pd, rd, through.clamp(max=1.0)

    def to_sun(self, q, r, mu_s):
        sine = self.R / r
        t = ((mu_s + q.clamp(min=0).sqrt() / r + sine * self.q["sun_radius"])
             / (2 * sine * self.q["sun_radius"])).clamp(0.0, 1.0)
        return self.to_top(q, r * mu_s) * (t * t * (3 - 2 * t))[..., None]

    # --- the scattering table's coordinates
    def build_axes(self):
        s = self.s
        M = s["sc_mu"] // 2
        rho = (self.H * self.grid(s["sc_r"]) / (s["sc_r"] - 1)).reshape(-1, 1)
        self.zq = (rho * rho).reshape(-1)
        q, r = rho * rho, (rho * rho + self.R ** 2).sqrt()
        self.zr = r.reshape(-1)
        x = (self.grid(M) / (M - 1)).reshape(1, -1)
        lo, hi = q / (r + self.R), rho
        d = lo + (hi - lo) * x.flip(1)
        pg = torch.where(d == 0, -r.expand_as(d), -(q + d * d) / (2 * d))
        lo, hi = (self.H2 - q) / (self.T + r), rho + self.H
        d = lo + (hi - lo) * x
        ps = torch.where(d == 0, r.expand_as(d), (self.H2 - q - d * d) / (2 * d))
        p = torch.cat([torch.maximum(pg, -r), torch.minimum(torch.maximum(ps, -r), r)], 1)
        self.row_p, self.row_mu = p, p / r  # [r][mu]
        self.row_ground = torch.arange(s["sc_mu"], device=self.dev) < M
        lo, hi = self.T - self.R, self.H
        A = -2 * self.q["mu_s_min"] * self.R / (hi - lo)
        x = self.grid(s["sc_mus"]) / (s["sc_mus"] - 1)
        d = lo + ((A - x * A) / (1 + x * A)).clamp(max=A) * (hi - lo)
        self.mu_s = ((self.H2 - d * d) / (2 * self.R * d)).clamp(-1.0, 1.0)
        self.nu = self.grid(s["sc_nu"]) / (s["sc_nu"] - 1) * 2 - 1

    def texel_nu(self, z):
        """[mu][nu][mu_s]: nu limited to the angles that mu and mu_s allow."""
        mu = self.row_mu[z].reshape(-1, 1, 1)
        mid, half = mu * self.mu_s, ((1 - mu * mu) * (1 - self.mu_s ** 2)).clamp(min=0).sqrt()
        return torch.minimum(torch.maximum(self.nu.reshape(1, -1, 1).expand(mid.shape[0], -1, mid.shape[2]), mid - half), mid + half)

    def mu_position(self, q, p, ground):
        M = self.s["sc_mu"] // 2
        rho, r = q.sqrt(), (q + self.R ** 2).sqrt()
        lo, hi = q / (r + self.R), rho
        xg = torch.where(hi == lo, torch.zeros_like(q), (self.ground_distance(q, p) - lo) / torch.where(hi == lo, torch.ones_like(q), hi - lo))
        lo, hi = (self.H2 - q) / (self.T + r), rho + self.H
        xs = (self.top_distance(q, p) - lo) / (hi - lo)
        return torch.where(ground, (M - 1) * (1 - xg.clamp(0, 1)), M + (M - 1) * xs.clamp(0, 1))

    def mu_s_position(self, mu_s):
        lo, hi = self.T - self.R, self.H
        a = (self.top_distance(torch.zeros_like(mu_s), self.R * mu_s) - lo) / (hi - lo)
        A = -2 * self.q["mu_s_min"] * self.R / (hi - lo)
        return (1 - a / A).clamp(min=0) / (1 + a) * (self.s["sc_mus"] - 1)

    def rows(self, table, tz, ty):
        """The table's rows at positions (tz, ty): [...][x][3]."""
        z, fz = _lerp_axis(tz, self.s["sc_r"])
        # rays that meet the ground and rays that do not have a half of the rows each
        M = self.s["sc_mu"] // 2
        half = (ty > M - 0.5).long() * M
        y, fy = _lerp_axis(ty - half, M)
        y = y + half
        flat, h = table.reshape(-1, *table.shape[2:]), self.s["sc_mu"]
        fz, fy, at = fz[..., None, None], fy[..., None, None], z * h + y
        up = min(1, M - 1)
        return (flat[at] * (1 - fy) + flat[at + up] * fy) * (1 - fz) + (flat[at + h] * (1 - fy) + flat[at + h + up] * fy) * fz

    # --- the passes
    def phases(self, nu):
        g = self.q["g"]
        k = 3 / (8 * math.pi) * (1 - g * g) / (2 + g * g)
        return 3 / (16 * math.pi) * (1 + nu * nu), k * (1 + nu * nu) * (1 + g * g - 2 * g * nu) ** -1.5

    def build_direct(self):
        s = self.s
        x = (self.grid(s["ir_r"]) / (s["ir_r"] - 1)).reshape(-1, 1)
        self.ir_h = x * (self.T - self.R)
        self.ir_mu_s = 2 * self.grid(s["ir_mus"]) / (s["ir_mus"] - 1) - 1
        q = self.ir_h * (2 * self.R + self.ir_h)
        m, a = self.ir_mu_s.reshape(1, -1), self.q["sun_radius"]
        cosine = torch.where(m < -a, torch.zeros_like(m), torch.where(m > a, m, (m + a) ** 2 / (4 * a)))
        r = self.R + self.ir_h
        return self.vec(self.q["solar"]) * self.to_top(q.expand(-1, m.shape[1]), r * m) * cosine[..., None]

    def samples(self, z):
        """The trapezoid samples of a slice's rows, [mu][sample]: the step, the distances, (q, p, r) there, the
        transmittance to them and the weights."""
        q, p = self.zq[z].expand(self.s["sc_mu"]), self.row_p[z]
        dx = torch.where(self.row_ground, self.ground_distance(q, p), self.top_distance(q, p)) / STEPS
        d = dx[:, None] * self.grid(STEPS + 1)
        q, p, ground = (v[:, None].expand(d.shape) for v in (q, p, self.row_ground))
        weight = torch.ones(STEPS + 1, dtype=F, device=self.dev)
        weight[0] = weight[-1] = 0.5
        return dx, d, *self.along(q, p, d, ground), weight

    def build_single(self):
        s = self.s
        shape = (s["sc_r"], s["sc_mu"], s["sc_nu"], s["sc_mus"], 3)
        ray, mie = (torch.empty(shape, dtype=F, device=self.dev) for _ in range(2))
        for z in range(s["sc_r"]):
            nu, r = self.texel_nu(z)[..., None], self.zr[z]
            dx, d, qd, _, rd, through, weight = self.samples(z)
            e = lambda v: v[:, None, None, :]  # noqa: E731
            mu_s_d = ((r * self.mu_s[:, None] + e(d) * nu) / e(rd)).clamp(-1.0, 1.0)
            light = self.to_sun(e(qd).expand(mu_s_d.shape), e(rd), mu_s_d) * through[:, None, None]
            h = self.altitude(qd)
            for out, scale, c in ((ray, "scale_r", "rayleigh"), (mie, "scale_m", "mie_sca")):
                w = weight * self.density(self.q[scale], h) * dx[:, None]
                out[z] = torch.einsum("mnsic,mi->mnsc", light, w) * self.vec(self.q["solar"]) * self.vec(self.q[c])
        return ray, mie

    def along_nu(self, rows, nu):
        """rows [direction row][nu][mu_s][3] at nu [direction row][mu][nu][mu_s][phi], between the slices."""
        L, n, m = rows.shape[:3]
        k, f = _lerp_axis((nu + 1) / 2 * (n - 1), n)
        at = k * m + self.grid(m).long()[:, None] + (self.grid(L).long() * (n * m)).reshape(-1, 1, 1, 1, 1)
        flat, f = rows.reshape(-1, 3), f[..., None]
        return flat[at] * (1 - f) + flat[at + m] * f

    def scattering_density(self, tables, irradiance):
        """tables: (ray, mie) of single scattering or (multiple,) of the order before."""
        s, N = self.s, DENSITY_SAMPLES
        out = torch.empty((s["sc_r"], s["sc_mu"], s["sc_nu"], s["sc_mus"], 3), dtype=F, device=self.dev)
        phi = (self.grid(2 * N) + 0.5) * math.pi / N
        theta = (self.grid(N) + 0.5) * math.pi / N
        wide = lambda v: v.reshape(-1, 1, 1, 1, 1)  # noqa: E731  per direction row
        ct, st = theta.cos(), theta.sin()
        for z in range(s["sc_r"]):
            r, q = self.zr[z], self.zq[z]
            mu = self.row_mu[z].reshape(-1, 1, 1)
            ox = (1 - mu * mu).clamp(min=0).sqrt()
            nu = self.texel_nu(z)
            sx = torch.where(ox == 0, torch.zeros_like(nu), (nu - mu * self.mu_s) / torch.where(ox == 0, torch.ones_like(ox), ox))
            sy = (1 - sx * sx - self.mu_s ** 2).clamp(min=0).sqrt()
            h = self.altitude(q)
            beta = [self.vec(self.q[c]) * self.density(self.q[k], h) for c, k in (("rayleigh", "scale_r"), ("mie_sca", "scale_m"))]
            qs, p = q.expand(N), r * ct
            ground = (p < 0) & (p * p - q >= 0)
            zpos = (q.sqrt() / self.H * (s["sc_r"] - 1)).expand(N)
            ypos = self.mu_position(qs, p, ground)
            nu1 = wide(ct) * self.mu_s[:, None] + wide(st) * (sx[..., None] * phi.cos() + sy[..., None] * phi.sin())
            light = []
            for table in tables:
                rows = self.rows(table.reshape(s["sc_r"], s["sc_mu"], -1, 3), zpos, ypos)
                light.append(self.along_nu(rows.reshape(N, s["sc_nu"], s["sc_mus"], 3), nu1))
            if len(light) == 2:
                fr, fm = self.phases(nu1)
                light = [light[0] * fr[..., None] + light[1] * fm[..., None]]
            light = light[0]
            dg = self.ground_distance(qs, p)
            tint = torch.where(ground[:, None], self.along(qs, p, dg, ground)[3] * self.vec(self.q["albedo"]) / math.pi, 0.0)
            if bool(ground.any()):
                cosine = (r * self.mu_s[:, None] + wide(dg) * nu1) / self.R
                i, f = _lerp_axis((cosine + 1) / 2 * (s["ir_mus"] - 1), s["ir_mus"])
                e, f = irradiance[0], f[..., None]
                light += (e[i] * (1 - f) + e[i + 1] * f) * tint.reshape(-1, 1, 1, 1, 1, 3)
            nu2 = (ox[..., None] * wide(st)) * phi.cos() + mu[..., None] * wide(ct)
            fr, fm = self.phases(nu2)
            weight = (fr[..., None] * beta[0] + fm[..., None] * beta[1]) * (wide(st) * (math.pi / N) ** 2)[..., None]
            out[z] = (light * weight).sum((0, 4))
        return out

    def indirect(self, tables):
        s, N = self.s, IRRADIANCE_SAMPLES
        J, L, m = s["ir_r"], N // 2, self.ir_mu_s
        phi = (self.grid(2 * N) + 0.5) * math.pi / N
        theta = (self.grid(L) + 0.5) * math.pi / N
        ct, st = theta.cos().reshape(1, -1), theta.sin()
        h = self.ir_h.reshape(-1, 1)
        q = (h * (2 * self.R + h)).clamp(0, self.H2).expand(J, L)
        zpos = q.sqrt() / self.H * (s["sc_r"] - 1)
        ypos = self.mu_position(q, (self.R + h) * ct, torch.zeros_like(q, dtype=torch.bool))
        ct = ct.reshape(1, 1, -1, 1)
        x, f = _lerp_axis(self.mu_s_position(m), s["sc_mus"])
        f = f[:, None]
        m = m.reshape(-1, 1, 1)
        nu = m * ct[0] + (1 - m * m).clamp(min=0).sqrt() * st.reshape(1, -1, 1) * phi.cos()  # [mu_s][theta][phi]
        k, fk = _lerp_axis((nu + 1) / 2 * (s["sc_nu"] - 1), s["sc_nu"])
        fk = fk[..., None]
        light = []
        for table in tables:
            rows = self.rows(table.reshape(s["sc_r"], s["sc_mu"], -1, 3), zpos, ypos)
            rows = rows.reshape(J, L, s["sc_nu"], s["sc_mus"], 3)
            rows = rows[..., x, :] * (1 - f) + rows[..., x + 1, :] * f  # [r][theta][nu][mu_s][3]
            i, l = (self.grid(n).long() for n in (x.shape[0], L))
            pick = lambda k: rows[:, l[:, None], k, i[:, None, None]]  # noqa: E731
            light.append(pick(k) * (1 - fk) + pick(k + 1) * fk)
        if len(light) == 2:
            fr, fm = self.phases(nu)
            light = [light[0] * fr[..., None] + light[1] * fm[..., None]]
        return (light[0] * (ct * st.reshape(1, 1, -1, 1) * (math.pi / N) ** 2)[..., None]).sum((2, 3))

    def multiple(self, density):
        s = self.s
        out = torch.empty_like(density)
        for z in range(s["sc_r"]):
            r, nu = self.zr[z], self.texel_nu(z)
            k, fk = _lerp_axis((nu + 1) / 2 * (s["sc_nu"] - 1), s["sc_nu"])
            k, fk = k[..., None], fk[..., None, None]
            dx, d, qd, pd, rd, through, weight = self.samples(z)
            ypos = self.mu_position(qd, pd, self.row_ground[:, None].expand(qd.shape))
            rows = self.rows(density.reshape(s["sc_r"], s["sc_mu"], -1, 3), qd.sqrt() / self.H * (s["sc_r"] - 1), ypos)
            e = lambda v: v[:, None, None, :]  # noqa: E731
            mu_s_i = ((r * self.mu_s[:, None] + e(d) * nu[..., None]) / e(rd)).clamp(-1.0, 1.0)
            x, fx = _lerp_axis(self.mu_s_position(mu_s_i), s["sc_mus"])
            fx = fx[..., None]
            flat, w, n = rows.reshape(-1, 3), s["sc_mus"], STEPS + 1  # rows [mu][sample][x][3]
            at = self.grid(s["sc_mu"]).long().reshape(-1, 1, 1, 1) * n + self.grid(n).long()
            at = at * (w * s["sc_nu"]) + k * w + x
            a = flat[at] * (1 - fx) + flat[at + 1] * fx
            b = flat[at + w] * (1 - fx) + flat[at + w + 1] * fx
            out[z] = torch.einsum("mnsic,mic->mnsc", a * (1 - fk) + b * fk, through * (weight * dx[:, None])[..., None])
        return out

    def build(self):
        s = self.s
        self.build_transmittance()
        self.build_axes()
        deltas = [self.build_direct()]
        ray, mie = self.build_single()
        scattering, irradiance = ray.clone(), torch.zeros_like(deltas[0])
        tables = (ray, mie)
        for n in range(2, self.order + 1):
            density = self.scattering_density(tables, deltas[-1])
            deltas.append(self.indirect(tables))
            irradiance += deltas[-1]
            tables = (self.multiple(density),)
            for z in range(s["sc_r"]):
                scattering[z] += tables[0][z] / self.phases(self.texel_nu(z))[0][..., None]
        one, zero = torch.ones_like(self.tr[..., :1]), torch.zeros_like(irradiance[..., :1])
        shape = (s["sc_r"], s["sc_mu"], s["sc_nu"] * s["sc_mus"], 4)
        return {"transmittance": torch.cat([self.tr, one], -1), "irradiance": torch.cat([irradiance, zero], -1),
                "scattering": torch.cat([scattering, mie[..., :1]], -1).reshape(shape)}

    # --- the use of finished tables
    def sky_lookup(self, table, q, p, mu_s, nu, ground):
        s = self.s
        n = q.shape[0]
        z, fz = _lerp_axis(q.sqrt() / self.H * (s["sc_r"] - 1), s["sc_r"])
        y, fy = _lerp_axis(self.mu_position(q, p, ground), s["sc_mu"])
        x, fx = _lerp_axis(self.mu_s_position(mu_s), s["sc_mus"])
        k, fk = _lerp_axis((nu + 1) / 2 * (s["sc_nu"] - 1), s["sc_nu"])
        flat, w = table.reshape(-1, 4), s["sc_nu"] * s["sc_mus"]
        total = torch.zeros((n, 4), dtype=F, device=self.dev)
        for bits in range(16):
            a, b, c, e = (bits >> i & 1 for i in range(4))
            weight = (fz if a else 1 - fz) * (fy if b else 1 - fy) * (fx if c else 1 - fx) * (fk if e else 1 - fk)
            total += weight[:, None] * flat[((z + a) * s["sc_mu"] + y + b) * w + (k + e) * s["sc_mus"] + x + c]
        mie = torch.where(total[:, :1] > 0, total[:, :3] * total[:, 3:] / total[:, :1], torch.zeros_like(total[:, :3]))
        return total[:, :3], mie * self.mie_ratio()

    def mie_ratio(self):
        ray, mie = self.vec(self.q["rayleigh"]), self.vec(self.q["mie_sca"])
        return ray[0] / mie[0] * (mie / ray)

    def sky(self, case, draw, depth, sun):
        t = self.build()
        s = self.s
        m = self.vec(np.asarray(draw.inverse_viewproj, np.float32).astype(np.float64).tolist())
        h, w = case["height"], case["width"]
        x = (2 * (self.grid(w) + 0.5) / w - 1).reshape(1, -1).expand(h, w).reshape(-1)
        y = (2 * (self.grid(h) + 0.5) / h - 1).reshape(-1, 1).expand(h, w).reshape(-1)
        z = torch.zeros_like(x) if depth is None else depth.reshape(-1).to(F)
        ray = x[:, None] * m[0] + y[:, None] * m[1] + m[3]
        view = ray[:, :3] / ray[:, :3].norm(dim=1, keepdim=True)
        point = ray + z[:, None] * m[2]
        camera = self.vec([float(np.float32(c)) for c in draw.camera_position])
        sun = self.vec([float(np.float32(c)) for c in sun])
        d = (point[:, :3] / point[:, 3:] * 1e-3 - camera).norm(dim=1)
        r = camera.norm()
        q = ((r - self.R) * (r + self.R)).expand(d.shape)
        p = view @ camera
        mu_s, nu = (camera @ sun / r).expand(d.shape), view @ sun
        ground = (p < 0) & (p * p - q >= 0)
        finite = d.isfinite()
        dd = torch.where(finite, d, torch.zeros_like(d))
        qd, pd, rd, through = self.along(q, p, dd, ground)
        # towards a point at infinity the ray leaves at the top; going down, the definition has no value there
        away = self.along(q, p, torch.full_like(d, 1e12), ground)[3]
        away = torch.where((p < 0)[:, None], torch.full_like(away, math.nan), away)
        through = torch.where(finite[:, None], through, away)
        table = t["scattering"]
        scattering, mie = self.sky_lookup(table, q, p, mu_s, nu, ground)
        mu_s_p = (r * mu_s + dd * nu) / rd
        scattering_p, mie_p = self.sky_lookup(table, qd, pd, mu_s_p, nu, ground)
        inner = scattering - through * scattering_p
        inner_mie = mie[:, :1] - through[:, :1] * mie_p[:, :1]
        extra = torch.where(inner[:, :1] > 0, inner * inner_mie / inner[:, :1], torch.zeros_like(inner)) * self.mie_ratio()
        e = (mu_s / 0.01).clamp(0, 1)
        extra = extra * (e * e * (3 - 2 * e))[:, None]
        scattering = torch.where(finite[:, None], inner, scattering)
        mie = torch.where(finite[:, None], extra, mie)
        fr, fm = self.phases(nu)
        color = scattering * fr[:, None] + mie * fm[:, None]
        zero, one = torch.zeros_like(color[:, :1]), torch.ones_like(color[:, :1])
        return {"radiance": torch.cat([color, zero], 1).reshape(h, w, 4),
                "transmittance": torch.cat([through, one], 1).reshape(h, w, 4)}

    def lighting(self, points, normals, sun):
        t = self.build()
        s = self.s
        points, normals = points.to(F), normals.to(F)
        sun = self.vec([float(np.float32(c)) for c in sun])
        r = points.norm(dim=1)
        mu_s = points @ sun / r
        q = (r - self.R) * (r + self.R)
        i, f = _lerp_axis((mu_s + 1) / 2 * (s["ir_mus"] - 1), s["ir_mus"])
        j, g = _lerp_axis((r - self.R) / (self.T - self.R) * (s["ir_r"] - 1), s["ir_r"])
        e, f, g = t["irradiance"], f[:, None], g[:, None]
        sky = (e[j, i] * (1 - f) + e[j, i + 1] * f) * (1 - g) + (e[j + 1, i] * (1 - f) + e[j + 1, i + 1] * f) * g
        sky = sky[:, :3] * ((1 + (normals * points).sum(1) / r) / 2)[:, None]
        direct = self.vec(self.q["solar"]) * self.to_sun(q, r, mu_s) * (normals @ sun).clamp(min=0)[:, None]
        return {"sun": direct, "sky": sky}


def exact(case, seed):
    if case["kind"] in ("sky", "lighting"):
        q, sizes, altitude, sun = _scene(case, seed)
        e = _Exact(q, sizes, 4)
        if case["kind"] == "lighting":
            return e.lighting(*_points(case, q, seed), sun)
        return e.sky(case, _camera(case, q, altitude, sun), _depth(case, seed) if case["depth"] else None, sun)
    left = 8.0e9  # directions of the density quadrature that some twenty seconds are enough for
    got = []
    for q, s, order in _requests(case, seed):
        need = _texels(s) * 2 * DENSITY_SAMPLES ** 2 * order + 1.5e8 * order
        if need > left:
            got.append({"transmittance": None, "irradiance": None, "scattering": None})
            continue
        left -= need
        got.append(_Exact(q, s, order).build())
    if all(g["scattering"] is None for g in got):
        return None
    return got if case["kind"] == "batch" else got[0]
