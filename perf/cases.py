"""The framework's performance cases: rebuilds of the atmosphere LUTs from the
smallest interactive ones to the high-resolution configuration, and the
render-time queries on them, each through the public entry points that a
program calls.

Planets are drawn around the Earth: radii 4000-7000 km, 50-100 km of air,
clear to hazy.  `exact` restates the
reference's integrals (functions.glsl of ebruneton/
precomputed_atmospheric_scattering) in plain FP64 torch.
"""
import math

import numpy as np
import torch

import precomputed_atmospheric_scattering_gb300 as atmo
from precomputed_atmospheric_scattering_gb300 import workloads as W

PI = math.pi
LAMBDAS = (680.0, 550.0, 440.0)
OZONE = (1.209e-25, 3.5e-25, 1.582e-26)   # cross sections at LAMBDAS, m^2
SHAPE_KEYS = ("tw", "th", "r", "mu", "mus", "nu", "iw", "ih")


def _case(name, kind, shape, orders=4, **more):
    return dict(name=name, kind=kind, orders=orders, **dict(zip(SHAPE_KEYS, shape)), **more)


def _shape(case):
    return tuple(case[k] for k in SHAPE_KEYS)


def listed():
    return [
        # An artist drags a slider: one planet at half the reference's LUT
        # sizes, single and double scattering only, rebuilt for every change.
        _case("edit_half_2", "batch", W.HALF, orders=2, n=1),
        # The same at the reference's sizes and its default of 4 orders.
        _case("edit_default_4", "batch", W.DEFAULT, n=1),
        # A program starts or swaps its atmosphere: constructor and Init of a
        # new model, as the reference's demo does on each parameter change.
        _case("model_init_default", "init", W.DEFAULT),
        # Many planets of one shape built together (offline, or a world list).
        _case("batch_default_8", "batch", W.DEFAULT, n=8),
        # A mixed batch: half, default and double-R shapes, 2 to 6 orders.
        _case("batch_mixed_9", "batch", W.DEFAULT, n=9, mixed=True),
        # Spectral precision: 15 wavelengths in 5 groups, FP16 LUTs, separate
        # single-Mie texture; Init repeated on a kept model.
        _case("spectral_15_half", "spectral", W.DEFAULT),
        # The high-resolution configuration, 8 orders.
        _case("hires_8", "batch", W.HIRES, orders=8, n=1),
        # One wavelength group into a caller's own buffers: odd sizes, a
        # luminance matrix, separate single-Mie texture.
        _case("precompute_odd", "precompute", (150, 37, 13, 46, 19, 5, 41, 11), orders=5),
        # A small environment map: sky luminance along 64 x 36 rays.
        _case("sky_2304", "sky", W.DEFAULT, n=2304),
        # Aerial perspective and lighting of a million scene points, with
        # shadow lengths: GetSkyRadianceToPoint and GetSunAndSkyIrradiance.
        _case("points_1000003", "points", W.DEFAULT, n=1000003),
        # One full-screen frame.
        _case("shade_1080p", "shade", W.DEFAULT, width=1920, height=1080),
        # The serving engine: four planets submitted together, each shaded
        # once built.
        _case("serve_4", "serve", W.DEFAULT, orders=3, n=4, width=640, height=360),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("batch", "batch", "batch", "precompute", "init", "sky", "points", "shade"))
    if kind in ("sky", "points"):
        return dict(_draw_shape(rng, 1 << 18), kind=kind, orders=2, n=_log(rng, 500, 2000000))
    if kind == "shade":
        return dict(_draw_shape(rng, 1 << 18), kind=kind, orders=2, width=_log(rng, 64, 2560),
                    height=_log(rng, 36, 1440))
    c = dict(_draw_shape(rng, 1 << 22), kind=kind, orders=rng.randint(2, 6))
    if kind == "batch":
        texels = c["r"] * c["mu"] * c["mus"] * c["nu"]
        c["n"] = _log(rng, 1, max(1, min(8, (1 << 23) // texels)))
    return c


def _draw_shape(rng, most):
    """LUT sizes between the tests' small shape and the high-resolution one."""
    while True:
        s = dict(tw=_log(rng, 64, 512), th=_log(rng, 16, 128), r=_log(rng, 4, 64),
                 mu=2 * _log(rng, 8, 128), mus=rng.choice((8, 16, 32, 64, _log(rng, 6, 70))),
                 nu=_log(rng, 3, 16), iw=_log(rng, 16, 128), ih=_log(rng, 4, 32))
        if s["r"] * s["mu"] * s["mus"] * s["nu"] <= most and _sound(s["r"]):
            return s


def _sound(r):
    """Whether the last of r radii is the top radius exactly in the reference's
    FP64 mapping: elsewhere (two sizes in five) the mu of its first upward row
    is the quotient of two rounding errors, and no two evaluations agree."""
    return ((r - 0.5) / r - 0.5 / r) / (1 - 1.0 / r) == 1.0


# --- inputs -----------------------------------------------------------------
def _planet(rng):
    """Parameters of one planet in km, per wavelength of LAMBDAS.  The radii
    are multiples of 1/8 km: their squares are exact in FP64, so that the
    distance of zero of the top radius's first upward row is zero however a
    compiler contracts the expression."""
    rb = int(rng.uniform(4000.0, 7000.0) * 8) / 8
    scale, mie = float(rng.uniform(0.3, 1.5)), float(rng.uniform(1e-3, 1e-2))
    ozone = bool(rng.random() < 0.5)
    return dict(
        rb=rb, rt=rb + int(rng.uniform(50.0, 100.0) * 8) / 8, solar=[1.5] * 3,
        ray=[1.24062e-3 * (l * 1e-3) ** -4 * scale for l in LAMBDAS],
        mie=[mie] * 3, mie_ext=[1.1 * mie] * 3,
        ozone=[300.0 * 2.687e20 / 15.0 * x if ozone else 0.0 for x in OZONE],
        albedo=[float(rng.uniform(0.0, 0.5))] * 3, sun=0.00935 / 2.0,
        hr=float(rng.uniform(6.0, 10.0)), hm=float(rng.uniform(0.8, 2.0)),
        g=float(rng.uniform(0.6, 0.9)), zenith=math.radians(102.0))


def _atmosphere(p):
    a = W.earth()
    for i in range(3):
        a.solar_irradiance[i], a.rayleigh_scattering[i] = p["solar"][i], p["ray"][i]
        a.mie_scattering[i], a.mie_extinction[i] = p["mie"][i], p["mie_ext"][i]
        a.absorption_extinction[i], a.ground_albedo[i] = p["ozone"][i], p["albedo"][i]
    a.sun_angular_radius, a.mie_phase_function_g = p["sun"], p["g"]
    a.bottom_radius, a.top_radius, a.mu_s_min = p["rb"], p["rt"], math.cos(p["zenith"])
    a.rayleigh_density.layers[1].exp_scale = -1.0 / p["hr"]
    a.mie_density.layers[1].exp_scale = -1.0 / p["hm"]
    return a


def _model(p, shape):
    """The planet through the reference's 19 constructor parameters (metres)."""
    up, L = (lambda v: np.array(v[::-1], np.float64)), atmo.DensityProfileLayer
    return atmo.Model(
        up(LAMBDAS), up(p["solar"]), p["sun"], p["rb"] * 1e3, p["rt"] * 1e3,
        [L(0.0, 1.0, -1e-3 / p["hr"], 0.0, 0.0)], up(p["ray"]) * 1e-3,
        [L(0.0, 1.0, -1e-3 / p["hm"], 0.0, 0.0)], up(p["mie"]) * 1e-3, up(p["mie_ext"]) * 1e-3,
        p["g"], [L(25000.0, 0.0, 0.0, 1.0 / 15000.0, -2.0 / 3.0),
                 L(0.0, 0.0, 0.0, -1.0 / 15000.0, 8.0 / 3.0)],
        up(p["ozone"]) * 1e-3, up(p["albedo"]), p["zenith"], 1000.0, 3, True, False,
        lut_shape=shape)


class _View:
    """A LUT's device buffer for torch, without a copy; the tensor made of it
    keeps it, and with it the owner of the buffer, alive."""

    def __init__(self, owner, v):
        self.owner = owner
        half = v.bytes == v.width * v.height * v.depth * 8
        self.__cuda_array_interface__ = dict(
            shape=(v.depth, v.height, v.width, 4), typestr="<f2" if half else "<f4",
            data=(v.device_ptr, False), version=2)


def _tensor(owner, view):
    return torch.as_tensor(_View(owner, view), device="cuda")


KINDS = (atmo.LUT_TRANSMITTANCE, atmo.LUT_SCATTERING, atmo.LUT_IRRADIANCE)


def _members(case, seed):
    """(planet, shape, orders) of a batch's or a server's instances."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["n"]):
        shape, orders = _shape(case), case["orders"]
        if case.get("mixed"):
            shape, orders = (W.HALF, W.DEFAULT, W.DOUBLE_R)[i % 3], 2 + i % 5
        elif case["kind"] == "serve" and i % 2:
            shape = W.HALF
        out.append((_planet(rng), shape, orders))
    return out


def _unit(rng, n):
    v = rng.normal(size=(n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _rays(case, seed):
    """Cameras up to 9 km high, view rays over the sphere, sun mostly up."""
    rng = np.random.default_rng(seed)
    p, n = _planet(rng), case["n"]
    up, view = _unit(rng, n), _unit(rng, n)
    sun = _unit(rng, n) * 0.8 + up * 0.6
    sun /= np.linalg.norm(sun, axis=1, keepdims=True)
    r = p["rb"] + np.exp(rng.uniform(math.log(0.05), math.log(9.0), n))
    cam = up * r[:, None]
    # Points along the view rays, short of the ground and of the top.
    rmu = (cam * view).sum(1)
    disc = rmu * rmu - r * r + p["rb"] ** 2
    top = -rmu + np.sqrt(rmu * rmu - r * r + p["rt"] ** 2)
    far = np.where((rmu < 0) & (disc >= 0), -rmu - np.sqrt(np.maximum(disc, 0)), top)
    d = far * rng.uniform(0.3, 0.98, n)
    shadow = np.where(rng.random(n) < 0.25, d * rng.uniform(0.0, 0.5, n), 0.0)
    normal = _unit(rng, n) * 0.5 + up
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    f = np.float32
    cam, view, sun = cam.astype(f), view.astype(f), sun.astype(f)
    point = (cam + view * d[:, None]).astype(f)
    return p, dict(cam=cam, view=view, sun=sun, point=point, normal=normal.astype(f),
                   shadow=shadow.astype(f))


def _frame(case, planet, rng):
    """A camera 0.1 to 5 km above the ground looking near the horizon, and
    the depth of each pixel's surface point."""
    w, h = case["width"], case["height"]
    up = _unit(rng, 1)[0]
    right = np.cross(up, _unit(rng, 1)[0])
    right /= np.linalg.norm(right)
    fwd = np.cross(up, right) + 0.1 * up
    fwd /= np.linalg.norm(fwd)
    cam = up * (planet["rb"] + rng.uniform(0.1, 5.0))
    v = W.random_view(np.random.default_rng(0), planet["rb"], w, h)
    sun = up * rng.uniform(0.1, 0.9) + np.cross(up, right) * 0.5 + right * rng.uniform(-0.5, 0.5)
    for name, x in (("camera", cam), ("right", right), ("up", np.cross(right, fwd)),
                    ("forward", fwd), ("sun_direction", sun / np.linalg.norm(sun))):
        setattr(v, name, (atmo.C.c_float * 3)(*x))
    cam, view = _pixel_rays(v)
    rmu, r2 = (view * cam).sum(-1), (cam * cam).sum(-1)
    disc = rmu * rmu - r2 + planet["rb"] ** 2
    hit = (rmu < 0) & (disc >= 0)
    far = torch.where(hit, -rmu - disc.clamp(min=0).sqrt(),
                      (-rmu + (rmu * rmu - r2 + planet["rt"] ** 2).sqrt()) * 0.3)
    return v, (far * 0.97).float().contiguous()


def _pixel_rays(v):
    """FP64 camera and unit view rays of a view's pixels, (H W, 3)."""
    t = lambda x: torch.tensor(list(x), dtype=torch.float64, device="cuda")   # noqa: E731
    w, h = v.width, v.height
    tan = float(np.float32(math.tan(0.5 * v.fov_y)))
    sx = ((2 * torch.arange(w, device="cuda", dtype=torch.float64) + 1) / w - 1) * tan * w / h
    sy = (1 - (2 * torch.arange(h, device="cuda", dtype=torch.float64) + 1) / h) * tan
    d = t(v.forward) + sx[None, :, None] * t(v.right) + sy[:, None, None] * t(v.up)
    d = (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)
    return t(v.camera).expand_as(d), d


def prepare(case, seed):
    kind, shape = case["kind"], _shape(case)
    rng = np.random.default_rng(seed)
    if kind == "batch":
        ms = _members(case, seed)
        atms = [_atmosphere(p) for p, _, _ in ms]
        batch = atmo.Batch(atms, [s for _, s, _ in ms], [o for _, _, o in ms])
        out = [_tensor(batch, batch.lut_view(i, k)) for i in range(len(ms)) for k in KINDS]
        return dict(kind=kind, batch=batch, atms=atms, out=out)
    if kind == "init":
        return dict(kind=kind, planet=_planet(rng), shape=shape, orders=case["orders"])
    if kind == "spectral":
        m = W.spectral_earth_model(shape, seed=seed)
        views = [_tensor(m, m.lut_view(k)) for k in (
            atmo.LUT_TRANSMITTANCE, atmo.LUT_SCATTERING, atmo.LUT_SINGLE_MIE,
            atmo.LUT_IRRADIANCE)]
        return dict(kind=kind, model=m, orders=case["orders"], out=views)
    if kind == "precompute":
        s = shape
        z = lambda *d: torch.zeros(*d, 4, device="cuda")   # noqa: E731
        return dict(kind=kind, atm=_atmosphere(_planet(rng)), shape=shape, orders=case["orders"],
                    lum=_lum(seed), out=[z(s[1], s[0]), z(s[2], s[3], s[5] * s[4]),
                                         z(s[2], s[3], s[5] * s[4]), z(s[7], s[6])])
    if kind in ("sky", "points"):
        p, x = _rays(case, seed)
        m = _model(p, shape)
        m.Init(case["orders"])
        x = {k: torch.from_numpy(v).cuda() for k, v in x.items()}
        return dict(kind=kind, model=m, luts=m.lut_set(), **x)
    if kind == "shade":
        p = _planet(rng)
        m = _model(p, shape)
        m.Init(case["orders"])
        v, depth = _frame(case, p, rng)
        return dict(kind=kind, model=m, luts=m.lut_set(), view=v, depth=depth)
    ms = _members(case, seed)
    frames = [_frame(case, p, rng) for p, _, _ in ms]
    bufs = [[torch.empty(case["height"], case["width"], 4, device="cuda") for _ in range(2)]
            for _ in ms]
    server = atmo.Server(hbm_budget_bytes=1 << 30)
    return dict(kind=kind, server=server, frames=frames, bufs=bufs,
                jobs=[(_atmosphere(p), s, o) for p, s, o in ms])


def run(state):
    kind = state["kind"]
    if kind == "batch":
        for i, a in enumerate(state["atms"]):
            state["batch"].set_atmosphere(i, a)
        state["batch"].run()
        return state["out"]
    if kind == "init":
        # The previous model lives while its LUTs are still referenced.
        m = _model(state["planet"], state["shape"])
        m.Init(state["orders"])
        return [_tensor(m, m.lut_view(k)) for k in KINDS]
    if kind == "spectral":
        state["model"].Init(state["orders"])
        return state["out"]
    if kind == "precompute":
        T, S, M, I = state["out"]
        atmo.precompute(state["atm"], state["shape"], state["orders"], T, S, M, I,
                        lum=state["lum"], combined=False)
        return state["out"]
    if kind == "sky":
        return state["luts"].sky_radiance(state["cam"], state["view"], state["sun"],
                                          luminance=True)
    if kind == "points":
        inscatter = state["luts"].sky_radiance_to_point(state["cam"], state["point"],
                                                        state["sun"], state["shadow"])
        light = state["luts"].sun_and_sky_irradiance(state["point"], state["normal"],
                                                     state["sun"])
        return [inscatter, light]
    if kind == "shade":
        return state["luts"].shade_view(state["view"], state["depth"])
    server = state["server"]
    built = [server.submit_rebuild(*job) for job in state["jobs"]]
    shaded = [server.submit_shade(t, v, depth, *bufs)
              for t, (v, depth), bufs in zip(built, state["frames"], state["bufs"])]
    for t in shaded:
        server.wait(t)
        server.release_ticket(t)
    return state["bufs"]   # the sets stay until the budget evicts them


def _lum(seed):
    return np.random.default_rng(seed + 99).uniform(-0.2, 1.0, (3, 3)).astype(np.float32)


def _rebuild_work(shape, orders, half=False, separate=False, groups=1):
    """Operations that the quadratures of the reference's sizes need per
    sample, with each lookup reduced to one line per channel."""
    tw, th, r, mu, mus, nu, iw, ih = shape
    texels = r * mu * mus * nu
    flops = tw * th * 501 * 15 + texels * 51 * 40
    flops += (orders - 1) * (texels * (512 * 16 + 51 * 40) + iw * ih * 1024 * 12)
    out = texels * (8 if half else 16) * (2 if separate else 1) + (tw * th + iw * ih) * 16
    return out, flops * groups


def work(case):
    kind, shape = case["kind"], _shape(case)
    lut = (shape[0] * shape[1] + shape[6] * shape[7]) * 16 + shape[2] * shape[3] * shape[4] * \
        shape[5] * 16
    if kind in ("batch", "serve"):
        parts = [_rebuild_work(s, o) for _, s, o in _members(case, 0)]
        out = sum(b for b, _ in parts), sum(f for _, f in parts)
        if kind == "batch":
            return dict(bytes=out[0], flops=out[1])
        pixels = case["n"] * case["width"] * case["height"]
        return dict(bytes=out[0] + pixels * 36, flops=out[1] + pixels * 600)
    if kind in ("init", "spectral", "precompute"):
        b, f = _rebuild_work(shape, case["orders"], kind == "spectral", kind != "init",
                             5 if kind == "spectral" else 1)
        return dict(bytes=b, flops=f)
    if kind == "shade":
        n = case["width"] * case["height"]
        return dict(bytes=n * 36 + min(lut, n * 256), flops=n * 600)
    n = case["n"]
    if kind == "sky":
        return dict(bytes=n * 60 + min(lut, n * 256), flops=n * 250)
    return dict(bytes=n * 148 + min(lut, n * 256), flops=n * 700)


# --- FP64 values ------------------------------------------------------------
class _Fp64:
    """The reference's precomputation and render functions in FP64 torch."""

    def __init__(self, planet, shape, rounded=False):
        # Model bakes its parameters into the shader with 6 decimals.
        q = (lambda x: float("%f" % x)) if rounded else float
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        v3 = lambda k: torch.tensor([q(x) for x in planet[k]], dtype=torch.float64,  # noqa: E731
                                    device=dev)
        self.dev, self.shape = dev, shape
        self.Rb, self.Rt, self.alpha, self.g = (q(planet[k]) for k in ("rb", "rt", "sun", "g"))
        self.H = math.sqrt(self.Rt * self.Rt - self.Rb * self.Rb)
        self.solar, self.ray, self.mie, self.mie_ext, self.oz, self.albedo = (
            v3(k) for k in ("solar", "ray", "mie", "mie_ext", "ozone", "albedo"))
        self.hr, self.hm = q(-1.0 / planet["hr"]), q(-1.0 / planet["hm"])
        lin, c0, c1 = q(1.0 / 15.0), q(-2.0 / 3.0), q(8.0 / 3.0)
        self.density = {
            "ray": lambda h: torch.where(h < 0, 0.0, (self.hr * h).exp().clamp(0, 1)),
            "mie": lambda h: torch.where(h < 0, 0.0, (self.hm * h).exp().clamp(0, 1)),
            "oz": lambda h: torch.where(h < 25.0, lin * h + c0, c1 - lin * h).clamp(0, 1)}
        D = self.to_top(self.t(self.Rb), self.t(q(math.cos(planet["zenith"]))))
        self.dmin_s = self.Rt - self.Rb
        self.A = float((D - self.dmin_s) / (self.H - self.dmin_s))

    def t(self, x):
        return torch.as_tensor(x, dtype=torch.float64, device=self.dev)

    def arange(self, n):
        return torch.arange(n, dtype=torch.float64, device=self.dev)

    def centre(self, n):
        """The texture coordinates of n texel centres."""
        return (self.arange(n) + 0.5) / self.t(n)

    def unit(self, u, n):
        """The unit-range value of texture coordinate u (by a tensor: torch
        divides by a number with a product on the GPU)."""
        return (u - 0.5 / n) / self.t(1 - 1.0 / n)

    def to_top(self, r, mu):
        return (-r * mu + (r * r * (mu * mu - 1) + self.Rt ** 2).clamp(min=0).sqrt()).clamp(min=0)

    def to_ground(self, r, mu):
        return (-r * mu - (r * r * (mu * mu - 1) + self.Rb ** 2).clamp(min=0).sqrt()).clamp(min=0)

    def hits_ground(self, r, mu):
        return (mu < 0) & (r * r * (mu * mu - 1) + self.Rb ** 2 >= 0)

    def phase_r(self, nu):
        return 3.0 / (16.0 * PI) * (1 + nu * nu)

    def phase_m(self, nu):
        g = self.g
        k = 3.0 / (8.0 * PI) * (1 - g * g) / (2 + g * g)
        return k * (1 + nu * nu) / (1 + g * g - 2 * g * nu) ** 1.5

    @staticmethod
    def taps(x, n):
        """Indices and upper weight of a clamped linear fetch at coordinate x."""
        f = x.floor()
        i = f.long()
        return i.clamp(0, n - 1), (i + 1).clamp(0, n - 1), x - f

    def bilinear(self, tex, x, y):
        h, w = tex.shape[:2]
        i0, i1, a = self.taps(x, w)
        j0, j1, b = self.taps(y, h)
        a, b, flat = a[..., None], b[..., None], tex.reshape(h * w, -1)
        return ((flat[j0 * w + i0] * (1 - a) + flat[j0 * w + i1] * a) * (1 - b) +
                (flat[j1 * w + i0] * (1 - a) + flat[j1 * w + i1] * a) * b)

    # Transmittance.
    def make_transmittance(self):
        w, h = self.shape[0], self.shape[1]
        unit = lambda n: self.unit(self.centre(n), n)   # noqa: E731
        rho = self.H * unit(h)[:, None]
        r = (rho * rho + self.Rb ** 2).sqrt()
        d = (self.Rt - r) + unit(w)[None, :] * (rho + self.H - (self.Rt - r))
        mu = torch.where(d == 0, 1.0, (self.H ** 2 - rho * rho - d * d) / (2 * r * d)).clamp(-1, 1)
        dx = self.to_top(r, mu) / 500
        tau = torch.zeros(h, w, 3, dtype=torch.float64, device=self.dev)
        sums = {k: torch.zeros(h, w, dtype=torch.float64, device=self.dev) for k in self.density}
        for i in range(501):
            di = i * dx
            alt = (di * di + 2 * r * mu * di + r * r).sqrt() - self.Rb
            for k, f in self.density.items():
                sums[k] += f(alt) * (0.5 if i in (0, 500) else 1.0)
        for k, beta in (("ray", self.ray), ("mie", self.mie_ext), ("oz", self.oz)):
            tau += (sums[k] * dx)[..., None] * beta
        self.T = (-tau).exp()

    def T_top(self, r, mu):
        rho = (r * r - self.Rb ** 2).clamp(min=0).sqrt()
        dmin, dmax = self.Rt - r, rho + self.H
        x = (self.to_top(r, mu) - dmin) / (dmax - dmin)
        return self.bilinear(self.T, x * (self.shape[0] - 1), rho / self.H * (self.shape[1] - 1))

    def T_segment(self, r, mu, d, ground):
        rd = (d * d + 2 * r * mu * d + r * r).sqrt().clamp(self.Rb, self.Rt)
        mud = ((r * mu + d) / rd).clamp(-1, 1)
        s = torch.where(ground, -1.0, 1.0)
        a, b = self.T_top(r, s * mu), self.T_top(rd, s * mud)
        up = ground[..., None]
        return (torch.where(up, b, a) / torch.where(up, a, b)).clamp(max=1)

    def T_sun(self, r, mu_s):
        sin_h = self.Rb / r
        e = sin_h * self.alpha
        x = ((mu_s + (1 - sin_h * sin_h).clamp(min=0).sqrt() + e) / (2 * e)).clamp(0, 1)
        return self.T_top(r, mu_s) * (x * x * (3 - 2 * x))[..., None]

    # Scattering coordinates.
    def make_texels(self):
        _, _, R, MU, MUS, NU = self.shape[:6]
        half = MU // 2
        # In the reference's own order of operations: at the top radius the
        # first upward row has a distance of zero or of a rounding error, and
        # its mu follows from which of the two it is.
        rho = self.H * self.unit(self.centre(R)[:, None], R)
        r = (rho * rho + self.Rb * self.Rb).sqrt()
        z = self.centre(MU)
        dg = (r - self.Rb) + (rho - (r - self.Rb)) * self.unit(1 - 2 * z[:half], half)
        dt = (self.Rt - r) + (rho + self.H - (self.Rt - r)) * self.unit(2 * z[half:] - 1, half)
        mug = torch.where(dg == 0, -1.0, -(rho * rho + dg * dg) / (2 * r * dg)).clamp(-1, 1)
        mut = torch.where(dt == 0, 1.0, (self.H * self.H - rho * rho - dt * dt) / (2 * r * dt))
        self.r = r.expand(R, MU).contiguous()
        self.mu = torch.cat([mug, mut.clamp(-1, 1)], 1)
        self.ground = (self.arange(MU) < half).expand(R, MU)
        xs = self.arange(MUS) / (MUS - 1)
        a = (self.A - xs * self.A) / (1 + xs * self.A)
        d = self.dmin_s + a.clamp(max=self.A) * (self.H - self.dmin_s)
        self.mu_s = ((self.H ** 2 - d * d) / (2 * self.Rb * d)).clamp(-1, 1)
        grid = (self.arange(NU) / (NU - 1) * 2 - 1)[:, None]
        mm = self.mu[..., None, None] * self.mu_s
        lim = ((1 - self.mu ** 2)[..., None, None] * (1 - self.mu_s ** 2)).clamp(min=0).sqrt()
        self.nu = torch.minimum(torch.maximum(grid - mm, -lim), lim) + mm   # (R, MU, NU, MUS)

    def row_coords(self, r, mu, ground):
        """(y, z) texel coordinates of (r, mu)."""
        R, half = self.shape[2], self.shape[3] // 2
        rho = (r * r - self.Rb ** 2).clamp(min=0).sqrt()
        rmu = r * mu
        disc = rmu * rmu - r * r + self.Rb ** 2
        dg = -rmu - disc.clamp(min=0).sqrt()
        xg = torch.where(rho == r - self.Rb, 0.0, (dg - (r - self.Rb)) / (rho - (r - self.Rb)))
        dt = -rmu + (disc + self.H ** 2).clamp(min=0).sqrt()
        xt = (dt - (self.Rt - r)) / (rho + self.H - (self.Rt - r))
        y = torch.where(ground, half - 1 - xg * (half - 1), half + xt * (half - 1))
        return y, rho / self.H * (R - 1)

    def sun_coord(self, mu_s):
        a = (self.to_top(self.t(self.Rb), mu_s) - self.dmin_s) / (self.H - self.dmin_s)
        return (1 - a / self.A).clamp(min=0) / (1 + a) * (self.shape[4] - 1)

    def fetch(self, tex, y, z, mu_s, nu):
        """The 4D lookup of tex (R, MU, NU * MUS, C)."""
        R, MU, MUS, NU = self.shape[2:6]
        Wd, flat = NU * MUS, tex.reshape(-1, tex.shape[-1])
        j0, j1, b = self.taps(y, MU)
        k0, k1, c = self.taps(z, R)
        x = self.sun_coord(mu_s)
        m0 = x.floor().clamp(0, MUS - 1)
        a, m0 = x - m0, m0.long()
        m1 = (m0 + 1).clamp(max=MUS - 1)
        v = (nu + 1) / 2 * (NU - 1)
        n0 = v.floor().clamp(0, NU - 1)
        l, n0 = v - n0, n0.long()
        n1 = (n0 + 1).clamp(max=NU - 1)
        out = 0
        for k, wk in ((k0, 1 - c), (k1, c)):
            for j, wj in ((j0, 1 - b), (j1, b)):
                row = (k * MU + j) * Wd
                for n, wn in ((n0, 1 - l), (n1, l)):
                    for m, wm in ((m0, 1 - a), (m1, a)):
                        out = out + flat[row + n * MUS + m] * (wk * wj * wn * wm)[..., None]
        return out

    def marched(self):
        """Samples of the ray of every LUT row: (weight x dx, d, r, mu)."""
        r, mu, g = self.r, self.mu, self.ground
        dx = torch.where(g, self.to_ground(r, mu), self.to_top(r, mu)) / 50
        for i in range(51):
            d = i * dx
            ri = (d * d + 2 * r * mu * d + r * r).sqrt().clamp(self.Rb, self.Rt)
            yield dx * (0.5 if i in (0, 50) else 1.0), d, ri, ((r * mu + d) / ri).clamp(-1, 1)

    def precompute(self, orders, lum=None, combined=True):
        _, _, R, MU, MUS, NU, IW, IH = self.shape
        lum = torch.eye(3, dtype=torch.float64, device=self.dev) if lum is None else self.t(lum)
        self.make_transmittance()
        self.make_texels()
        nu, e = self.nu, (lambda x: x[..., None, None])
        rmus = e(self.r) * self.mu_s
        irr_r = self.unit(self.centre(IH)[:, None], IH)
        irr_r = self.Rb + irr_r * (self.Rt - self.Rb)
        irr_r = irr_r.expand(IH, IW)
        irr_mu = (2 * self.arange(IW) / (IW - 1) - 1).expand(IH, IW)
        al = self.alpha
        f = torch.where(irr_mu < -al, 0.0, torch.where(irr_mu > al, irr_mu,
                                                       (irr_mu + al) ** 2 / (4 * al)))
        dI = self.solar * self.T_top(irr_r, irr_mu) * f[..., None]
        I = torch.zeros_like(dI)
        sr, sm = (torch.zeros(R, MU, NU, MUS, 3, dtype=torch.float64, device=self.dev)
                  for _ in range(2))
        for w, d, ri, _ in self.marched():
            t = e(self.T_segment(self.r, self.mu, d, self.ground).permute(2, 0, 1)).permute(
                1, 2, 3, 4, 0)
            mu_s = ((rmus + e(d) * nu) / e(ri)).clamp(-1, 1)
            t = t * self.T_sun(e(ri), mu_s)
            alt = ri - self.Rb
            sr += t * e(self.density["ray"](alt) * w)[..., None]
            sm += t * e(self.density["mie"](alt) * w)[..., None]
        dR, dM = (x.reshape(R, MU, NU * MUS, 3) for x in (sr * self.solar * self.ray,
                                                          sm * self.solar * self.mie))
        S, M = dR @ lum.T, dM @ lum.T
        mie_red = M[..., 0].clone()
        for order in range(2, orders + 1):
            J = self.scattering_density(dR, dM, dI, order)
            dI = self.indirect(dR, dM, order - 1, irr_r, irr_mu)
            I = I + dI @ lum.T
            acc = torch.zeros(R, MU, NU, MUS, 3, dtype=torch.float64, device=self.dev)
            for w, d, ri, mui in self.marched():
                y, z = self.row_coords(ri, mui, self.ground)
                mu_s = ((rmus + e(d) * nu) / e(ri)).clamp(-1, 1)
                t = self.T_segment(self.r, self.mu, d, self.ground) * w[..., None]
                acc += self.fetch(J, e(y), e(z), mu_s, nu) * t[:, :, None, None, :]
            dR = acc.reshape(R, MU, NU * MUS, 3)
            S = S + dR @ lum.T / self.phase_r(nu).reshape(R, MU, -1)[..., None]
        self.S = torch.cat([S, mie_red[..., None] if combined else torch.zeros_like(S[..., :1])],
                           -1)
        self.M, self.I = M, I
        return self

    def scattering_density(self, dR, dM, dI, order):
        R, MU, MUS, NU, IW = self.shape[2:7]
        phi = (self.arange(32) + 0.5) * PI / 16
        theta = (self.arange(16) + 0.5) * PI / 16
        J = torch.empty(R, MU, NU * MUS, 3, dtype=torch.float64, device=self.dev)
        cols = torch.arange(MUS, device=self.dev)[:, None]
        for k in range(R):
            r, mu, nu, mu_s = self.r[k, 0], self.mu[k], self.nu[k], self.mu_s
            ox = (1 - mu * mu).clamp(min=0).sqrt()
            sx = torch.where(ox[:, None, None] == 0, 0.0,
                             (nu - mu[:, None, None] * mu_s) / ox[:, None, None])
            sy = (1 - sx * sx - mu_s ** 2).clamp(min=0).sqrt()
            ground = self.hits_ground(r, theta.cos())
            y, _ = self.row_coords(r.expand(16), theta.cos(), ground)
            j0, j1, b = self.taps(y, MU)
            dist = torch.where(ground, self.to_ground(r, theta.cos()), 0.0)
            tg = self.T_segment(r.expand(16), theta.cos(), dist, ground) * self.albedo / PI
            b = b[:, None, None]
            lines = [x[k][j0] * (1 - b) + x[k][j1] * b for x in (dR, dM)]
            alt = r - self.Rb
            a_r, a_m = self.ray * self.density["ray"](alt), self.mie * self.density["mie"](alt)
            out = torch.zeros(MU, NU, MUS, 3, dtype=torch.float64, device=self.dev)
            for l in range(16):
                ct, st = theta[l].cos(), theta[l].sin()
                nu1 = (sx[..., None] * (phi.cos() * st) + sy[..., None] * (phi.sin() * st) +
                       (mu_s * ct)[:, None])
                v = (nu1.clamp(-1, 1) + 1) / 2 * (NU - 1)
                n0 = v.floor().clamp(0, NU - 2)
                fr, at = (v - n0)[..., None], n0.long() * MUS + cols
                L = lines[0][l]
                rad = L[at] * (1 - fr) + L[at + MUS] * fr
                if order == 2:
                    m = lines[1][l]
                    rad = (rad * self.phase_r(nu1)[..., None] +
                           (m[at] * (1 - fr) + m[at + MUS] * fr) * self.phase_m(nu1)[..., None])
                if bool(ground[l]):
                    mu_g = (r * mu_s[:, None] + dist[l] * nu1) / self.Rb
                    x = (mu_g + 1) / 2 * (IW - 1)
                    i0, i1, c = self.taps(x, IW)
                    c = c[..., None]
                    rad = rad + tg[l] * (dI[0][i0] * (1 - c) + dI[0][i1] * c)
                nu2 = ox[:, None] * phi.cos() * st + mu[:, None] * ct
                w = (self.phase_r(nu2)[..., None] * a_r + self.phase_m(nu2)[..., None] * a_m)
                out += torch.einsum("jncpe,jpe->jnce", rad, w) * (st * (PI / 16) ** 2)
            J[k] = out.reshape(MU, NU * MUS, 3)
        return J

    def indirect(self, dR, dM, order, r, mu_s):
        out = torch.zeros(*r.shape, 3, dtype=torch.float64, device=self.dev)
        phi = (self.arange(64) + 0.5) * PI / 32
        sky = torch.zeros_like(r, dtype=torch.bool)
        for j in range(16):
            th = (j + 0.5) * PI / 32
            y, z = self.row_coords(r, self.t(math.cos(th)).expand_as(r), sky)
            nu = (phi.cos() * math.sin(th) * (1 - mu_s ** 2).clamp(min=0).sqrt()[..., None] +
                  math.cos(th) * mu_s[..., None])
            at = y[..., None].expand_as(nu), z[..., None].expand_as(nu), mu_s[..., None].expand_as(
                nu), nu
            rad = self.fetch(dR, *at)
            if order == 1:
                rad = (rad * self.phase_r(nu)[..., None] +
                       self.fetch(dM, *at) * self.phase_m(nu)[..., None])
            out += rad.sum(-2) * (math.cos(th) * math.sin(th) * (PI / 32) ** 2)
        return out

    def luts(self, separate=False):
        pad = lambda x, a: torch.cat([x, torch.full_like(x[..., :1], a)], -1)   # noqa: E731
        out = [pad(self.T, 1.0)[None], self.S, pad(self.M, 0.0), pad(self.I, 0.0)[None]]
        return out if separate else [out[0], out[1], out[3]]

    # Render functions on the LUTs.
    def combined(self, r, mu, mu_s, nu, ground):
        y, z = self.row_coords(r, mu, ground)
        v = self.fetch(self.S, y, z, mu_s.clamp(-1, 1), nu)
        return v[..., :3], self.single_mie(v[..., :3], v[..., 3])

    def single_mie(self, rgb, alpha):
        k = torch.where(rgb[..., 0] > 0, alpha / rgb[..., 0], 0.0)[..., None]
        return rgb * k * (self.ray[0] / self.mie[0]) * (self.mie / self.ray)

    def start(self, cam, view, sun):
        r, rmu = cam.norm(dim=-1), (cam * view).sum(-1)
        mu = rmu / r
        return r, mu, (cam * sun).sum(-1) / r, (view * sun).sum(-1), self.hits_ground(r, mu)

    def phases(self, scattering, mie, nu):
        return scattering * self.phase_r(nu)[..., None] + mie * self.phase_m(nu)[..., None]

    def sky_radiance(self, cam, view, sun):
        r, mu, mu_s, nu, ground = self.start(cam, view, sun)
        T = torch.where(ground[..., None], 0.0, self.T_top(r, mu))
        return self.phases(*self.combined(r, mu, mu_s, nu, ground), nu), T

    def to_point(self, cam, point, sun, shadow):
        view = point - cam
        d = view.norm(dim=-1)
        r, mu, mu_s, nu, ground = self.start(cam, view / d[..., None], sun)
        T = self.T_segment(r, mu, d, ground)
        s, mie = self.combined(r, mu, mu_s, nu, ground)
        d = (d - shadow).clamp(min=0)
        rp = (d * d + 2 * r * mu * d + r * r).sqrt().clamp(self.Rb, self.Rt)
        sp, mie_p = self.combined(rp, (r * mu + d) / rp, (r * mu_s + d * nu) / rp, nu, ground)
        Ts = torch.where((shadow > 0)[..., None], self.T_segment(r, mu, d, ground), T)
        s = s - Ts * sp
        mie = self.single_mie(s, mie[..., 0] - Ts[..., 0] * mie_p[..., 0])
        x = (mu_s / 0.01).clamp(0, 1)
        return self.phases(s, mie * (x * x * (3 - 2 * x))[..., None], nu), T

    def irradiance(self, point, normal, sun):
        r = point.norm(dim=-1)
        mu_s = (point * sun).sum(-1) / r
        IW, IH = self.shape[6:]
        x_r = (r - self.Rb) / (self.Rt - self.Rb)
        sky = self.bilinear(self.I, (mu_s + 1) / 2 * (IW - 1), x_r * (IH - 1))
        sky = sky * ((1 + (normal * point).sum(-1) / r) * 0.5)[..., None]
        return self.solar * self.T_sun(r, mu_s) * (normal * sun).sum(-1).clamp(min=0)[..., None], \
            sky

    def frame(self, v, depth):
        cam, view = _pixel_rays(v)
        sun = self.t(list(v.sun_direction)).expand_as(cam)
        sky, t_sky = self.sky_radiance(cam, view, sun)
        point = cam + view * depth.reshape(-1, 1).double()
        scatter, t = self.to_point(cam, point, sun, torch.zeros_like(depth).double().reshape(-1))
        direct, ambient = self.irradiance(point, -view, sun)
        shaded = scatter + t * self.t(list(v.albedo)) / PI * (direct + ambient)
        dims = (v.height, v.width, 4)
        return [torch.cat([sky, t_sky[:, 1:2]], 1).reshape(dims),
                torch.cat([shaded, torch.ones_like(shaded[:, :1])], 1).reshape(dims)]


EXACT_SAMPLES = 6 << 30   # density samples that take a few seconds


def _costly(shape, orders):
    return shape[2] * shape[3] * shape[4] * shape[5] * 512 * (orders - 1) > EXACT_SAMPLES


def exact(case, seed):
    kind, shape, orders = case["kind"], _shape(case), case["orders"]
    rng = np.random.default_rng(seed)
    if kind == "spectral" or (kind != "batch" and _costly(shape, orders)):
        return None
    if kind == "batch":
        out, left = [], 2   # the first two instances
        for p, s, o in _members(case, seed):
            do = left > 0 and not _costly(s, o)
            left -= do
            out += _Fp64(p, s).precompute(o).luts() if do else [None] * 3
        return out if any(x is not None for x in out) else None
    if kind == "init":
        return _Fp64(_planet(rng), shape, rounded=True).precompute(orders).luts()
    if kind == "precompute":
        return _Fp64(_planet(rng), shape).precompute(orders, _lum(seed), False).luts(True)
    if kind in ("sky", "points"):
        p, x = _rays(case, seed)
        f = _Fp64(p, shape, rounded=True).precompute(orders)
        x = {k: torch.from_numpy(v).to(f.dev).double() for k, v in x.items()}
        if kind == "sky":
            # The luminance factors come from a table of the framework's.
            return [None, f.sky_radiance(x["cam"], x["view"], x["sun"])[1]]
        return [list(f.to_point(x["cam"], x["point"], x["sun"], x["shadow"])),
                list(f.irradiance(x["point"], x["normal"], x["sun"]))]
    if kind == "shade":
        p = _planet(rng)
        v, depth = _frame(case, p, rng)
        return _Fp64(p, shape, rounded=True).precompute(orders).frame(v, depth)
    ms = _members(case, seed)
    frames = [_frame(case, p, rng) for p, _, _ in ms]
    return [_Fp64(p, s).precompute(o).frame(*fr) for (p, s, o), fr in zip(ms, frames)]
