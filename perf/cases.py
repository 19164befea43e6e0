"""The work that users of this package have it do, as measurable cases.

Every case goes through a public entry point: the lookup-table builds
(`atmosphere_lut.build`, `build_device`, `build_batch`, `Plan`), the queries of
a built atmosphere (`query.Context`), the surrogate's inference and its
training gradients, and the cloud-noise builders (`noise`).

`exact` is the same result in 64 bits from plain torch: the atmosphere's
definition (ray and sphere quadratures over clamped multilinear tables)
restated array by array, without this package's code.
"""
import math

import numpy as np
import torch

from sfsim_gb300 import atmosphere_lut, config, noise, query

# Table shapes and quadrature steps of config.py's named workloads (T, E, S/M
# shapes, ray steps, sphere steps, iterations, atmosphere height in km).
SMALL = dict(t0=32, t1=32, e0=16, e1=32, n0=8, n1=16, n2=8, n3=4, steps=64, sphere=16, iters=2, height_km=100)
REFERENCE = dict(t0=64, t1=255, e0=16, e1=63, n0=32, n1=127, n2=32, n3=8, steps=100, sphere=15, iters=5, height_km=35)
PRODUCTION = dict(t0=255, t1=255, e0=16, e1=64, n0=32, n1=255, n2=32, n3=8, steps=128, sphere=32, iters=5,
                  height_km=100)
SWEEP = dict(t0=255, t1=255, e0=16, e1=64, n0=16, n1=128, n2=16, n3=8, steps=128, sphere=32, iters=4, height_km=100)
RAGGED = dict(t0=65, t1=129, e0=13, e1=37, n0=21, n1=95, n2=19, n3=6, steps=90, sphere=21, iters=3, height_km=60)


def _build(name, how, shape, precision="f32", batch=1):
    return dict(name=name, op="build", how=how, precision=precision, batch=batch, **shape)


def listed():
    return [
        # a preview-size table, where launches and latencies count
        _build("build_small_f32", "device", SMALL),
        # the same table in the 64-bit mode that results are judged by, as a prepared plan
        _build("build_small_f64", "plan", SMALL, precision="f64"),
        # odd sizes on every axis, a whole build into device tensors
        _build("build_ragged", "device", RAGGED),
        # the reference's own settings, into host arrays as generate_atmosphere_luts takes them
        _build("build_reference", "host", REFERENCE),
        # the production tables, kept on the device
        _build("build_production", "device", PRODUCTION),
        # a parameter sweep: many atmospheres in one batched call, to host arrays
        _build("build_sweep", "batch", SWEEP, batch=16),
        # a frame's worth of sky lookups against the reference's tables
        dict(name="query_in_scatter", op="table", kind=4, n=1049353, **REFERENCE),
        # a frame's ground pixels attenuated along their view rays
        dict(name="query_attenuation", op="attenuation", kind=1, n=524309, **REFERENCE),
        # the rendered in-scatter by direct quadrature (the judge of the other two)
        dict(name="query_direct", op="direct", n=65557, **REFERENCE),
        # the surrogate network over a frame of queries
        dict(name="surrogate_query", op="surrogate", n=1049353, **REFERENCE),
        # loss and gradients of one training batch
        dict(name="surrogate_gradients", op="gradients", n=65536, **SMALL),
        # the cloud-noise build tasks: Worley, Perlin and the blue-noise dither array
        dict(name="cloud_noise", op="noise", size=64, divisions=8, blue=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: builds twice as often as queries, each over its whole range."""
    op = rng.choice(["build"] * 6 + ["table", "attenuation", "direct", "surrogate", "gradients", "noise"])
    if op == "build":
        case = dict(t0=_log_int(rng, 16, 255), t1=_log_int(rng, 16, 255), e0=rng.randint(4, 16),
                    e1=_log_int(rng, 16, 64), n0=rng.randint(6, 32), n1=_log_int(rng, 15, 255),
                    n2=rng.choice([7, 8, 12, 16, 19, 24, 31, 32]), n3=rng.choice([3, 4, 5, 6, 8]),
                    steps=_log_int(rng, 24, 128), sphere=rng.randint(12, 32), iters=rng.randint(1, 5),
                    height_km=rng.choice([35, 60, 100]))
        precision = "f32"
        if case["n0"] * case["n1"] * case["n2"] * case["n3"] <= 40000 and rng.random() < 0.4:
            precision = "f64"
        how = rng.choice(["device", "device", "plan", "host", "batch"])
        return dict(op="build", how=how, precision=precision, batch=rng.randint(2, 6) if how == "batch" else 1, **case)
    shape = dict(REFERENCE, n1=rng.choice([63, 95, 127]), n0=rng.choice([16, 24, 32]), height_km=rng.choice([35, 100]))
    if op == "table":
        return dict(op=op, kind=rng.choice([1, 3, 4]), n=_log_int(rng, 1000, 1050000), **shape)
    if op == "attenuation":
        return dict(op=op, kind=rng.choice([0, 1, 3]), n=_log_int(rng, 1000, 500000), **shape)
    if op == "direct":
        return dict(op=op, n=_log_int(rng, 500, 60000), **shape)
    if op == "surrogate":
        return dict(op=op, n=_log_int(rng, 1000, 1000000), **shape)
    if op == "gradients":
        return dict(op=op, n=1024 * _log_int(rng, 2, 64), **SMALL)
    divisions = rng.choice([4, 5, 8])
    return dict(op=op, size=divisions * rng.randint(3, 8), divisions=divisions, blue=rng.randint(16, 72))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _physics(case, seed):
    """An atmosphere of the sweep's distribution (config.parameter_sweep) with its own ground and sun."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 17]))
    s_r, s_m = np.exp(rng.uniform(math.log(0.5), math.log(2.0), 2))
    return dict(radius=rng.uniform(3000e3, 7000e3), height=1000.0 * case["height_km"],
                brightness=tuple(rng.uniform(0.1, 0.5, 3)), intensity=tuple(rng.uniform(0.8, 1.2, 3)),
                ray_base=tuple(s_r * b for b in (5.8e-6, 13.5e-6, 33.1e-6)), ray_scale=rng.uniform(6000.0, 10000.0),
                mie_base=(s_m * 2e-5,) * 3, mie_scale=rng.uniform(800.0, 2000.0), mie_quot=0.9,
                mie_g=rng.uniform(0.6, 0.85))


def _config(case, seed):
    p = _physics(case, seed)
    return config.make_config(
        radius=p["radius"], height=p["height"], brightness=p["brightness"], intensity=p["intensity"],
        mie=config.component(p["mie_base"], p["mie_scale"], p["mie_quot"], p["mie_g"]),
        rayleigh=config.component(p["ray_base"], p["ray_scale"]),
        transmittance_shape=(case["t0"], case["t1"]), surface_radiance_shape=(case["e0"], case["e1"]),
        ray_scatter_shape=(case["n0"], case["n1"], case["n2"], case["n3"]), ray_steps=case["steps"],
        sphere_steps=case["sphere"], iterations=case["iters"],
        precision=config.FP64 if case.get("precision") == "f64" else config.FP32)


def _generator(seed, device):
    return torch.Generator(device=device).manual_seed(int(seed) * 1000003 + 11)


def _unit(n, g, device):
    v = torch.randn((n, 3), generator=g, device=device, dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _query_points(case, seed, device):
    """Positions uniform in height inside the atmosphere, views and suns uniform on the sphere."""
    p, g, n = _physics(case, seed), _generator(seed, device), case["n"]
    r = p["radius"] + p["height"] * torch.rand((n, 1), generator=g, device=device, dtype=torch.float64)
    return r * _unit(n, g, device), _unit(n, g, device), _unit(n, g, device), g


def _mlp_parameters(seed):
    """Weights of the size a trained surrogate has: corrections of a few percent of the table's value."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 23]))
    parts = []
    for k in range(4):
        parts += [rng.normal(0, math.sqrt(1.5 / 256), 256 * 256), rng.normal(0, 0.05, 256)]
    parts += [rng.normal(0, 0.01, 4 * 256), np.array([0.0, 0.0, 0.0, -7.0])]
    return np.concatenate(parts).astype(np.float32)


def _training_batch(case, seed):
    """Coordinates in [0, 1] and log-space corrections of a few percent."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 29]))
    coords = rng.random((case["n"], 10), dtype=np.float32)
    coords[:, 5] = coords[:, 5] > 0.5
    return coords, rng.normal(0, 0.05, (case["n"], 3)).astype(np.float32)


def _noise_inputs(case, seed):
    rng = np.random.Generator(np.random.PCG64([int(seed), 31]))
    m = case["blue"]
    return (noise.random_point_grid(case["divisions"], case["size"], rng),
            noise.random_gradient_grid(case["divisions"], rng),
            rng.permutation(m * m)[:m * m // 10].astype(np.int32))


def prepare(case, seed):
    op = case["op"]
    if op == "build":
        if case["how"] == "batch":
            return dict(case=case, cfgs=[_config(case, 1000 * int(seed) + b) for b in range(case["batch"])])
        cfg = _config(case, seed)
        out = None
        if case["how"] in ("device", "plan"):
            out = [torch.empty(s, dtype=torch.float32, device="cuda") for s in atmosphere_lut.table_shapes(cfg)]
        return dict(case=case, cfg=cfg, out=out, plan=atmosphere_lut.Plan(cfg) if case["how"] == "plan" else None)
    if op == "noise":
        grid, gradients, seeds = _noise_inputs(case, seed)
        return dict(case=case, grid=grid, gradients=gradients, seeds=seeds)
    state = dict(case=case, ctx=query.Context(_config(case, seed)))
    if op == "gradients":
        state["ctx"].surrogate_parameters(set_to=_mlp_parameters(seed))
        state["coords"], state["targets"] = _training_batch(case, seed)
        return state
    x, v, l, g = _query_points(case, seed, "cuda")
    if op in ("table", "attenuation"):
        x, v, l = x.float(), v.float(), l.float()
    state.update(x=x, v=v, l=l)
    if op == "attenuation":
        state["segment"] = _segments(case, seed, x, v)
        state["incoming"] = torch.rand((case["n"], 4), generator=g, device="cuda", dtype=torch.float32)
    if op == "surrogate":
        state["ctx"].surrogate_parameters(set_to=_mlp_parameters(seed))
    return state


def _segments(case, seed, x, v):
    """(start, length) of the part of each view ray up to the ground or 200 km, as a scene's pixels have it."""
    p = _physics(case, seed)
    x, v = x.double(), v.double()
    b, c = (x * v).sum(1), (x * x).sum(1)
    ground = b * b - (c - p["radius"] ** 2)
    top = (-b + torch.sqrt((b * b - (c - (p["radius"] + p["height"]) ** 2)).clamp(min=0))) * 0.98
    near = torch.where((ground > 0) & (b < 0), (-b - torch.sqrt(ground.clamp(min=0))) * 0.98, top)
    return torch.stack([torch.zeros_like(near), near.clamp(0.0, 2e5)], 1).float().contiguous()


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

TABLES = ("transmittance", "surface_radiance", "ray_scatter", "mie_strength")


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "build":
        if case["how"] == "device":
            return dict(zip(TABLES, atmosphere_lut.build_device(state["cfg"], state["out"])))
        if case["how"] == "plan":
            return dict(zip(TABLES, state["plan"].build(state["out"])))
        if case["how"] == "batch":
            return atmosphere_lut.build_batch(state["cfgs"])
        return atmosphere_lut.build(state["cfg"])
    if op == "noise":
        return dict(worley=noise.worley_noise(case["divisions"], case["size"], grid=state["grid"]),
                    perlin=noise.perlin_noise(case["divisions"], case["size"], gradients=state["gradients"]),
                    blue=noise.blue_noise(case["blue"], seed_pixels=state["seeds"]))
    ctx = state["ctx"]
    if op == "table":
        return ctx.table(case["kind"], state["x"], state["v"], state["l"])
    if op == "attenuation":
        return ctx.attenuation(case["kind"], state["l"], state["x"], state["v"], state["segment"], state["incoming"])
    if op == "direct":
        return ctx.direct(state["x"], state["v"], state["l"])
    if op == "surrogate":
        return ctx.surrogate(state["x"], state["v"], state["l"])[0]
    loss, grads = ctx.surrogate_gradients(state["coords"], state["targets"])
    return dict(loss=loss, grads=grads)


def _sphere_rings(theta_steps, phi_steps, span):
    return [math.ceil(math.sin(span * ((0.5 + k) / theta_steps)) * phi_steps) for k in range(theta_steps)]


def work(case):
    """Bytes of the inputs and results; operations of the quadratures, counting each sum once per node it is
    defined at: about 24 per extinction sample, 16 per interpolated direction or ray sample."""
    op = case["op"]
    if op == "noise":
        n, m2 = case["size"] ** 3, case["blue"] ** 2
        return dict(bytes=8 * n + 4 * m2, flops=27 * 8 * n + 120 * n + 2.0 * m2 * m2)
    if op == "gradients":
        flops = 3 * case["n"] * 2 * (4 * 256 * 256 + 256 * 4)
        return dict(bytes=case["n"] * 13 * 4 + 8 * 264196, flops=flops)
    nodes = case["n0"] * case["n1"] * case["n2"] * case["n3"]
    rows, S = case["n0"] * case["n1"], case["steps"]
    table_bytes = 12 * (case["t0"] * case["t1"] + case["e0"] * case["e1"] + 2 * nodes)
    if op == "build":
        P = sum(_sphere_rings(case["sphere"] >> 1, case["sphere"], math.pi))
        half = sum(_sphere_rings(S >> 2, S, math.pi / 2))
        flops = (24 * (rows * S * S + case["t0"] * case["t1"] * S) + 40 * nodes * S / 3 +
                 case["iters"] * 16 * (nodes * P + nodes * S + case["e0"] * case["e1"] * half))
        return dict(bytes=case["batch"] * table_bytes, flops=case["batch"] * flops)
    n = case["n"]
    if op == "direct":
        return dict(bytes=n * 84 + table_bytes, flops=n * S * (24 * S * 1.3 + 100))
    if op == "surrogate":
        return dict(bytes=n * 84 + table_bytes, flops=n * 2 * (4 * 256 * 256 + 256 * 4))
    return dict(bytes=n * (68 if op == "attenuation" else 48) + table_bytes, flops=n * 250)


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

def _limit_quot(a, b, lower, upper):
    a, b = torch.where(b < 0, -a, a), b.abs()
    q = a / torch.where(b == 0, torch.ones_like(b), b)
    r = torch.where(a < b * upper, torch.where(a > b * lower, q, torch.as_tensor(lower).to(a)), torch.as_tensor(upper).to(a))
    return torch.where(a == 0, torch.zeros_like(a), r)


def _interp(table, coords):
    """Clamped multilinear interpolation of table[n0]..[nk][3] at broadcastable coordinates."""
    shape = table.shape[:-1]
    flat, size = table.reshape(-1, table.shape[-1]), 1
    terms = [(0, 1.0)]
    for n in reversed(range(len(shape))):
        c = torch.nan_to_num(coords[n]).clamp(0, shape[n] - 1)
        u = c.floor()
        f, u = c - u, u.long()
        w = (u + 1).clamp(max=shape[n] - 1)
        terms = [(o + size * i, s * k) for o, s in terms for i, k in ((u, 1 - f), (w, f))]
        size *= shape[n]
    return sum(flat[o] * s.unsqueeze(-1) for o, s in terms)


def _dot(a, b):
    return (a * b).sum(-1)


def _vec(*c):
    return torch.stack(torch.broadcast_tensors(*c), -1)


class Atmosphere64:
    """The tables of one atmosphere by their definition, in 64 bits."""

    def __init__(self, case, physics, device):
        self.case, self.p, self.device = case, physics, device
        self.R, self.H = physics["radius"], physics["height"]
        self.top = self.R + self.H
        self.Hh = math.sqrt(self.top ** 2 - self.R ** 2)
        self.S = case["steps"]
        self.ray_base, self.mie_base = self.t(physics["ray_base"]), self.t(physics["mie_base"])
        self.mie_ext = self.mie_base / physics["mie_quot"]

    def t(self, v):
        return torch.as_tensor(v, dtype=torch.float64, device=self.device)

    def range(self, n):
        return torch.arange(n, dtype=torch.float64, device=self.device)

    # geometry

    def exit_point(self, x, v, above):
        b, c = _dot(x, v), _dot(x, x)
        far = -b + torch.sqrt((b * b - c + self.top ** 2).clamp(min=0))
        disc = b * b - c + self.R ** 2
        near = torch.where(disc > 0, (-b - torch.sqrt(disc.clamp(min=0))).clamp(min=0), (-b).clamp(min=0))
        return x + v * torch.where(above, far, near).unsqueeze(-1)

    def above_horizon(self, x, v):
        s = _dot(x, v)
        return (s >= 0) | (s * s <= _dot(x, x) - self.R ** 2)

    def rho(self, r):
        return torch.sqrt((r * r - self.R ** 2).clamp(min=0))

    def radius(self, n):
        return torch.sqrt(self.R ** 2 + (self.range(n) / (n - 1) * self.Hh) ** 2)

    def views(self, r, n):
        """sin, cos and above flag of the n elevation nodes at each radius r."""
        hd, i, r = self.rho(r)[:, None], (self.range(n) / (n - 1))[None, :], r[:, None]
        below = (i < 0.5) | ((i == 0.5) & (2 * r < self.R + self.top))
        g, s = hd * (1 - 2 * i), (hd + self.Hh) * (2 * i - 1)
        a = _limit_quot(self.R ** 2 - r * r - g * g, 2 * r * g, -1.0, 1.0)
        b = _limit_quot(self.top ** 2 - r * r - s * s, 2 * r * s, -1.0, 1.0)
        sin = torch.where(below, a, b)
        return sin, torch.sqrt(1 - sin * sin), ~below

    def height_index(self, r, n):
        return (n - 1) * self.rho(r) / self.Hh

    def elevation_index(self, r, rs, above, n):
        rho = self.rho(r)
        delta = rs * rs - rho * rho
        up = 0.5 - _limit_quot(rs - torch.sqrt((delta + self.Hh ** 2).clamp(min=0)), 2 * rho + 2 * self.Hh, -0.5, 0.0)
        down = 0.5 + _limit_quot(rs + torch.sqrt(delta.clamp(min=0)), 2 * rho, -0.5, 0.0)
        return (n - 1) * torch.where(above, up, down)

    def sun_sin(self, n):
        return (torch.log(1 - self.range(n) / (n - 1) * (1 - math.exp(-3.6))) + 0.6) / -3.0

    def sun_index(self, sin, n):
        return (n - 1) * ((1 - torch.exp(-3 * sin - 0.6)) / (1 - math.exp(-3.6))).clamp(min=0)

    @staticmethod
    def phase(g, mu):
        return 3 * (1 - g * g) * (1 + mu * mu) / (8 * math.pi * (2 + g * g) * (1 + g * g - 2 * g * mu) ** 1.5)

    # optical depths

    def sums(self, q, b, length):
        """Midpoint integrals of both densities from a point with q = |p|^2 - R^2 along a ray with p.d = b."""
        dt = length / self.S
        ray, mie = torch.zeros_like(q + b), torch.zeros_like(q + b)
        for n in range(self.S):
            t = dt * (n + 0.5)
            h = t.add(b, alpha=2).mul_(t).add_(q)
            h = h.div_(h.add(self.R ** 2).clamp_(min=0).sqrt_().add_(self.R))
            ray += torch.exp(h * (-1 / self.p["ray_scale"]))
            mie += torch.exp(h.mul_(-1 / self.p["mie_scale"]))
        return ray * dt, mie * dt

    def transmittance(self, x, end):
        d = end - x
        length = d.norm(dim=-1)
        r = x.norm(dim=-1)
        b = _dot(x, d) / torch.where(length > 0, length, torch.ones_like(length))
        ray, mie = self.sums((r - self.R) * (r + self.R), b, length)
        return torch.exp(-(ray[..., None] * self.ray_base + mie[..., None] * self.mie_ext))

    def sphere(self, theta_steps, phi_steps, span):
        """Directions (frame of x = (r, 0, 0)) and weights of the ring quadrature."""
        d, w = [], []
        half = span / theta_steps / 2
        for k in range(theta_steps):
            theta = span * ((0.5 + k) / theta_steps)
            n = math.ceil(math.sin(theta) * phi_steps)
            for i in range(n):
                phi = 2 * math.pi * ((0.5 + i) / n)
                d.append((math.cos(theta), -math.sin(theta) * math.sin(phi), math.sin(theta) * math.cos(phi)))
                w.append((math.cos(theta - half) - math.cos(theta + half)) * 2 * math.pi / n)
        return self.t(d), self.t(w)

    # the build

    def rows(self):
        c = self.case
        n0, n1, n2, n3 = (c[k] for k in ("n0", "n1", "n2", "n3"))
        r = self.radius(n0)
        sin, cos, above = self.views(r, n1)
        self.row_r = r[:, None].expand(n0, n1).reshape(-1)
        self.sin, self.cos, self.above = sin.reshape(-1), cos.reshape(-1), above.reshape(-1)
        zero = torch.zeros_like(self.row_r)
        x, v = _vec(self.row_r, zero, zero), _vec(self.sin, self.cos, zero)
        self.end = self.exit_point(x, v, self.above)
        self.x, self.v, self.D = x, v, self.end - x
        self.step = self.D.norm(dim=-1) / self.S
        ss = self.sun_sin(n2)
        most = torch.sqrt((1 - ss * ss).clamp(min=0))
        dvs = 2 * self.range(n3) / (n3 - 1) - 1
        s1 = _limit_quot(dvs[None, None, :] - self.sin[:, None, None] * ss[None, :, None],
                         self.cos[:, None, None].expand(-1, n2, n3), -2.0, 2.0)
        s1 = torch.minimum(torch.maximum(s1, -most[None, :, None]), most[None, :, None])
        s2 = torch.sqrt((1 - s1 * s1 - (ss * ss)[None, :, None]).clamp(min=0))
        self.light = _vec(ss[None, :, None], s1, s2)  # [row][n2][n3][3]
        self.mu = _dot(self.v[:, None, None, :], self.light)
        self.row_T = {}

    def samples(self, lo, hi):
        """Points p_s [row][S][3], T(x, p_s), q and radius of the rows lo..hi."""
        s = (self.range(self.S) + 0.5) / self.S
        p = self.x[lo:hi, None, :] + self.D[lo:hi, None, :] * s[None, :, None]
        if lo not in self.row_T:  # the same in every iteration
            self.row_T[lo] = self.transmittance(self.x[lo:hi, None, :].expand_as(p), p)
        r = p.norm(dim=-1)
        return p, self.row_T[lo], (r - self.R) * (r + self.R), r

    def first_order(self):
        c = self.case
        cells = c["n2"] * c["n3"]
        out_r, out_m = [], []
        light = self.light.reshape(-1, cells, 3)
        step = max(1, 3_000_000 // (self.S * cells))
        for lo in range(0, light.shape[0], step):
            hi = min(lo + step, light.shape[0])
            p, T, q, r = self.samples(lo, hi)
            b = torch.einsum("rsc,rkc->rks", p, light[lo:hi])
            qq = q[:, None, :].expand_as(b)
            lit = (b >= 0) | (b * b <= qq)
            bl, ql = b[lit], qq[lit]
            root = torch.sqrt((bl * bl - ql + self.Hh ** 2).clamp(min=0))
            far = torch.where(bl >= 0, (self.Hh ** 2 - ql) / (bl + root).clamp(min=1e-300), root - bl).clamp(min=0)
            ray, mie = self.sums(ql, bl, far)
            h = r - self.R
            er, em = torch.exp(-h / self.p["ray_scale"]), torch.exp(-h / self.p["mie_scale"])
            sr, sm = [], []
            for ch in range(3):
                t = torch.zeros_like(b)
                t[lit] = torch.exp(-(self.ray_base[ch] * ray + self.mie_ext[ch] * mie))
                t *= T[:, None, :, ch]
                sr.append((t * er[:, None, :]).sum(-1))
                sm.append((t * em[:, None, :]).sum(-1))
            scale = self.step[lo:hi, None, None] * self.t(self.p["intensity"])
            out_r.append(torch.stack(sr, -1) * scale * self.ray_base)
            out_m.append(torch.stack(sm, -1) * scale * self.mie_base)
        shape = (c["n0"], c["n1"], c["n2"], c["n3"], 3)
        phase = self.phase(0.0, self.mu).reshape(shape[:-1] + (1,))
        return torch.cat(out_r).reshape(shape) * phase, torch.cat(out_m).reshape(shape)

    def point_scatter(self, dS, M, dE):
        c = self.case
        n0, n1, n2, n3 = (c[k] for k in ("n0", "n1", "n2", "n3"))
        dirs, weight = self.sphere(c["sphere"] >> 1, c["sphere"], math.pi)
        light = self.light.reshape(n0, n1, n2, n3, 3)
        ss = self.sun_sin(n2)
        J = torch.empty((n0, n1, n2, n3, 3), dtype=torch.float64, device=self.device)
        for i in range(n0):
            r = self.radius(n0)[i]
            x = _vec(r, 0 * r, 0 * r).expand_as(dirs)
            above = self.above_horizon(x, dirs)
            end = self.exit_point(x, dirs, above)
            surface = 2 * (end.norm(dim=-1) - self.R) < self.H
            hx = self.height_index(r, n0)
            el = self.elevation_index(r.expand(len(dirs)), _dot(x, dirs), ~surface, n1)
            sun = self.sun_index(ss, n2)
            at = [hx.reshape(1, 1, 1), el[:, None, None], sun[None, :, None], self.range(n3)[None, None, :]]
            rows, rows_m = _interp(dS, at), _interp(M, at) if M is not None else None  # [P][n2][n3][3]
            view = self.v.reshape(n0, n1, 3)[i] @ dirs.T  # [n1][P]
            w = torch.stack([self.phase(0.0, view) * weight, self.phase(self.p["mie_g"], view) * weight], 1)
            ground = self.transmittance(x, end) * self.t(self.p["brightness"]) / math.pi * surface[:, None]
            h = r - self.R
            beta_r = self.ray_base * torch.exp(-h / self.p["ray_scale"])
            beta_m = self.mie_base * torch.exp(-h / self.p["mie_scale"])
            gr = end.norm(dim=-1)
            dirs_at = torch.arange(len(dirs), device=self.device)
            g = torch.nonzero(surface).squeeze(1)
            step = max(1, 20_000_000 // (n1 * n3 * len(dirs)))
            for lo in range(0, n2, step):
                k = torch.arange(lo, min(lo + step, n2), device=self.device)
                lk = light[i].transpose(0, 1)[k].reshape(-1, 3)  # [k n1 n3][3]
                k, each = k.repeat_interleave(n1 * n3)[:, None], len(k)
                mu = lk @ dirs.T  # [k n1 n3][P]
                a = torch.nan_to_num((n3 - 1) * (1 + mu) / 2).clamp(0, n3 - 1)
                u = a.floor().long()
                f, up = (a - u)[..., None], (u + 1).clamp(max=n3 - 1)
                val = rows[dirs_at, k, u] * (1 - f) + rows[dirs_at, k, up] * f
                if rows_m is not None:
                    m = rows_m[dirs_at, k, u] * (1 - f) + rows_m[dirs_at, k, up] * f
                    val = val + m * self.phase(self.p["mie_g"], mu)[..., None]
                if len(g):
                    sun_g = (lk @ end[g].T) / gr[g]
                    e = _interp(dE, [self.height_index(gr[g], c["e0"])[None, :].expand_as(sun_g),
                                     self.sun_index(sun_g, c["e1"])])
                    val[:, g] += e * ground[g]
                val = val.reshape(each, n1, n3, len(dirs), 3).transpose(2, 3).reshape(each, n1, len(dirs), n3 * 3)
                ray, mie = (w @ val).reshape(each, n1, 2, n3, 3).unbind(2)
                J[i, :, lo:lo + each] = (ray * beta_r + mie * beta_m).transpose(0, 1)
        return J

    def surface_radiance(self, dS, M):
        c = self.case
        dirs, weight = self.sphere(self.S >> 2, self.S, math.pi / 2)
        r = self.radius(c["e0"])
        sun = self.sun_sin(c["e1"])
        light = _vec(sun, torch.sqrt((1 - sun * sun).clamp(min=0)), 0 * sun)
        mu = light @ dirs.T  # [e1][P]
        out = []
        for i in range(c["e0"]):
            ri = r[i].expand(len(dirs))
            above = torch.ones_like(ri, dtype=torch.bool)
            el = self.elevation_index(ri, ri * dirs[:, 0], above, c["n1"])
            at = [self.height_index(ri, c["n0"])[None, :].expand_as(mu), el[None, :].expand_as(mu),
                  self.sun_index(sun, c["n2"])[:, None].expand_as(mu), (c["n3"] - 1) * (1 + mu) / 2]
            v = _interp(dS, at)
            if M is not None:
                v = v + _interp(M, at) * self.phase(self.p["mie_g"], mu)[..., None]
            out.append((v * (weight * dirs[:, 0])[None, :, None]).sum(1))
        return torch.stack(out)

    def ray_scatter(self, J):
        c = self.case
        cells = c["n2"] * c["n3"]
        light, out = self.light.reshape(-1, cells, 3), []
        angle = ((c["n3"] - 1) * (1 + self.mu) / 2).reshape(-1, cells)
        step = max(1, 3_000_000 // (self.S * cells))
        for lo in range(0, light.shape[0], step):
            hi = min(lo + step, light.shape[0])
            p, T, q, r = self.samples(lo, hi)
            h = self.height_index(r, c["n0"])
            el = self.elevation_index(r, _dot(p, self.v[lo:hi, None, :]), self.above[lo:hi, None], c["n1"])
            planes = _interp(J.reshape(c["n0"], c["n1"], cells * 3), [h, el])  # [row][S][cells 3]
            planes = planes.reshape(-1, c["n2"], c["n3"], 3)
            sin = torch.einsum("rsc,rkc->rsk", p, light[lo:hi]) / r[..., None]
            at = torch.arange(planes.shape[0], dtype=torch.float64, device=self.device).reshape(hi - lo, self.S, 1)
            v = _interp(planes, [at.expand_as(sin), self.sun_index(sin, c["n2"]),
                                 angle[lo:hi, None, :].expand_as(sin)])
            out.append((v * T[:, :, None, :]).sum(1) * self.step[lo:hi, None, None])
        return torch.cat(out).reshape(c["n0"], c["n1"], c["n2"], c["n3"], 3)

    def build(self):
        c = self.case
        self.rows()
        # transmittance and the ground's direct light
        rt = self.radius(c["t0"])
        sin, cos, above = self.views(rt, c["t1"])
        x = _vec(rt[:, None].expand_as(sin), 0 * sin, 0 * sin)
        v = _vec(sin, cos, 0 * sin)
        T = self.transmittance(x, self.exit_point(x, v, above))
        at_t = [self.height_index(rt, c["t0"])[:, None].expand_as(sin),
                self.elevation_index(rt[:, None], rt[:, None] * sin, above, c["t1"])]
        re = self.radius(c["e0"])
        sun = self.sun_sin(c["e1"])
        re, sun = re[:, None].expand(-1, c["e1"]), sun[None, :].expand(c["e0"], -1)
        x, l = _vec(re, 0 * re, 0 * re), _vec(sun, torch.sqrt((1 - sun * sun).clamp(min=0)), 0 * sun)
        dE = (self.transmittance(x, self.exit_point(x, l, torch.ones_like(sun, dtype=torch.bool))) *
              self.t(self.p["intensity"]) * sun.clamp(min=0)[..., None])
        at_e = [self.height_index(re, c["e0"]), self.sun_index(sun, c["e1"])]
        shape = (c["n0"], c["n1"], c["n2"], c["n3"])
        at_s = [self.height_index(self.row_r, c["n0"]).reshape(c["n0"], c["n1"], 1, 1).expand(shape),
                self.elevation_index(self.row_r, self.row_r * self.sin, self.above, c["n1"])
                .reshape(c["n0"], c["n1"], 1, 1).expand(shape),
                self.sun_index(self.sun_sin(c["n2"]), c["n2"]).reshape(1, 1, -1, 1).expand(shape),
                ((c["n3"] - 1) * (1 + self.mu) / 2).reshape(shape)]
        first, strength = self.first_order()
        dS, M, S, E = first, strength, first, torch.zeros_like(dE)
        self.Jsum = torch.zeros_like(first)
        for _ in range(c["iters"]):
            J = self.point_scatter(dS, M, dE)
            dE, dS, M = self.surface_radiance(dS, M), self.ray_scatter(J), None
            E, S = _interp(E + dE, at_e), _interp(S + dS, at_s)
            self.Jsum += J
        self.T, self.E, self.Sc, self.M = _interp(T, at_t), _interp(E, at_e), _interp(S, at_s), _interp(strength, at_s)

    def files(self):
        """The four tables in the files' layout: 4-D tables tiled [n0 n2][n1 n3]."""
        c = self.case

        def tile(t):
            return t.permute(0, 2, 1, 3, 4).reshape(c["n0"] * c["n2"], c["n1"] * c["n3"], 3)
        return dict(zip(TABLES, (self.T, self.E, tile(self.Sc), tile(self.M))))

    # lookups, as the renderer's shaders define them

    def look_transmittance(self, p, d, above):
        c, r = self.case, p.norm(dim=-1)
        return _interp(self.T, [self.height_index(r, c["t0"]), self.elevation_index(r, _dot(p, d), above, c["t1"])])

    def coordinates(self, p, d, l, above):
        c, r = self.case, p.norm(dim=-1)
        return [self.height_index(r, c["n0"]), self.elevation_index(r, _dot(p, d), above, c["n1"]),
                self.sun_index(_dot(p, l) / r, c["n2"]), (c["n3"] - 1) * (1 + _dot(d, l)) / 2]

    def look_in_scatter(self, p, d, l, above):
        at = self.coordinates(p, d, l, above)
        phase = self.phase(self.p["mie_g"], _dot(d, l))
        return _interp(self.Sc, at) + _interp(self.M, at) * phase[..., None]

    def look_track(self, p, q, l):
        """Transmittance and in-scatter between p and q; 1 and 0 where they are the same point."""
        d = q - p
        length = d.norm(dim=-1, keepdim=True)
        none = length == 0
        d = d / torch.where(none, torch.ones_like(length), length)
        above = self.above_horizon(p, d)
        t = self.look_transmittance(p, d, above) / self.look_transmittance(q, d, above)
        s = self.look_in_scatter(p, d, l, above) - t * self.look_in_scatter(q, d, l, above)
        return torch.where(none, torch.ones_like(t), t), torch.where(none, torch.zeros_like(s), s)

    def direct(self, x, v, l):
        """The rendered in-scatter by quadrature at the point."""
        c, out = self.case, []
        step = max(1, 6_000_000 // self.S)
        for lo in range(0, len(x), step):
            X, V, L = x[lo:lo + step], v[lo:lo + step], l[lo:lo + step]
            above = self.above_horizon(X, V)
            D = self.exit_point(X, V, above) - X
            s = ((self.range(self.S) + 0.5) / self.S)[None, :, None]
            p = X[:, None, :] + D[:, None, :] * s
            T = self.transmittance(X[:, None, :].expand_as(p), p)
            r = p.norm(dim=-1)
            q, b = (r - self.R) * (r + self.R), _dot(p, L[:, None, :])
            lit = (b >= 0) | (b * b <= q)
            far = (-b + torch.sqrt((b * b - q + self.Hh ** 2).clamp(min=0))).clamp(min=0)
            ray, mie = self.sums(q, b, far)
            sun = torch.exp(-(ray[..., None] * self.ray_base + mie[..., None] * self.mie_ext)) * lit[..., None]
            mu = _dot(V, L)
            at = [self.height_index(r, c["n0"]), self.elevation_index(r, _dot(p, V[:, None, :]), above[:, None], c["n1"]),
                  self.sun_index(b / r, c["n2"]), ((c["n3"] - 1) * (1 + mu) / 2)[:, None].expand_as(r)]
            h = r - self.R
            er = torch.exp(-h / self.p["ray_scale"])[..., None] * self.ray_base
            em = torch.exp(-h / self.p["mie_scale"])[..., None] * self.mie_base
            first = (er * self.phase(0.0, mu)[:, None, None] + em * self.phase(self.p["mie_g"], mu)[:, None, None])
            total = T * (first * sun * self.t(self.p["intensity"]) + _interp(self.Jsum, at))
            out.append(total.sum(1) * (D.norm(dim=-1) / self.S)[:, None])
        return torch.cat(out)


def _features(u):
    k = torch.arange(16, device=u.device)
    f = torch.where(k % 2 == 1, math.sqrt(2.0), 1.0).double() * 2.0 ** (k // 2)
    a = math.pi * u[:, :6, None] * f
    h = 2.0 * (torch.arange(8, device=u.device) + 1).double()
    b = math.pi * u[:, 6:, None] * h
    return torch.cat([torch.stack([torch.sin(z), torch.cos(z)], -1).reshape(len(u), -1) for z in (a, b)], 1)


def _layers(params, device):
    p, out, o = torch.as_tensor(params.astype(np.float64), device=device), [], 0
    for rows in (256, 256, 256, 256, 4):
        out.append((p[o:o + 256 * rows].reshape(rows, 256).clone(), p[o + 256 * rows:o + 257 * rows].clone()))
        o += 257 * rows
    return out


def _network(layers, u):
    h = _features(u)
    for w, b in layers[:-1]:
        h = torch.nn.functional.silu(h @ w.T + b)
    return h @ layers[-1][0].T + layers[-1][1]


def _exact_gradients(case, seed, device):
    coords, targets = (torch.as_tensor(v, device=device).double() for v in _training_batch(case, seed))
    layers = [(w.requires_grad_(), b.requires_grad_()) for w, b in _layers(_mlp_parameters(seed), device)]
    out = _network(layers, coords)
    m = ((out[:, :3] - targets) ** 2).mean(1)
    s = out[:, 3].clamp(-40, 20)
    (m.mean() + 0.01 * 0.5 * (m.detach() * torch.exp(-s) + s).mean()).backward()
    grads = torch.cat([t.grad.reshape(-1) for layer in layers for t in layer])
    return dict(loss=float(m.detach().mean()), grads=grads)


def _exact_noise(case, seed):
    grid, gradients, _ = _noise_inputs(case, seed)
    n, d = case["size"], case["divisions"]
    cs = n // d
    at = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1)  # [k][j][i]
    p = at + 0.5
    cell = at // cs
    best = np.full((n,) * 3, np.inf)
    for step in np.ndindex(3, 3, 3):
        c = cell[..., ::-1] + (np.array(step) - 1)  # grid[z][y][x] of the point (x, y, z) = p
        w = grid[tuple(np.moveaxis(c % d, -1, 0))] + (n * (c // d))[..., ::-1]
        best = np.minimum(best, ((w - p) ** 2).sum(-1))
    worley = np.sqrt(best)
    worley = 1 - worley / worley.max()
    table = np.array([(1, 1, 0), (-1, 1, 0), (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1),
                      (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1)], float)
    q = (at[..., ::-1] + 0.5) * d / n  # out[k][j][i] is the sample at (i, j, k)
    c = np.floor(q).astype(int)
    perlin = np.zeros((n,) * 3)
    for corner in np.ndindex(2, 2, 2):
        o = np.array(corner)
        g = table[gradients[tuple(np.moveaxis(((c + o) % d)[..., ::-1], -1, 0))]]
        v = q - (c + o)
        t = 1 - np.abs(v)
        perlin += (((6 * t - 15) * t + 10) * t ** 3).prod(-1) * (g * v).sum(-1)
    perlin = (perlin - perlin.min()) / (perlin.max() - perlin.min())
    return dict(worley=worley.reshape(-1), perlin=perlin.reshape(-1), blue=None)


def exact(case, seed):
    op, device = case["op"], "cuda" if torch.cuda.is_available() else "cpu"
    if op == "noise":
        return _exact_noise(case, seed)
    if op == "gradients":
        return _exact_gradients(case, seed, device)
    # sun-ray samples of the first order: the part that takes long
    samples = case["n0"] * case["n1"] * case["n2"] * case["n3"] * case["steps"] ** 2 * case.get("batch", 1)
    if samples > 5e10:
        return None
    if op == "build" and case["how"] == "batch":
        each = []
        for b in range(case["batch"]):
            a = Atmosphere64(case, _physics(case, 1000 * int(seed) + b), device)
            a.build()
            each.append(a.files())
        return {k: torch.stack([e[k] for e in each]) for k in TABLES}
    a = Atmosphere64(case, _physics(case, seed), device)
    a.build()
    if op == "build":
        return a.files()
    x, v, l, g = _query_points(case, seed, device)
    if op == "direct":
        return a.direct(x, v, l)
    if op in ("table", "attenuation"):
        x, v, l = x.float().double(), v.float().double(), l.float().double()
    up = torch.ones(len(x), dtype=torch.bool, device=device)
    if op == "table":
        if case["kind"] == 1:
            return a.look_transmittance(x, v, up)
        return a.look_in_scatter(x, v, l, up if case["kind"] == 3 else a.above_horizon(x, v))
    if op == "attenuation":
        segment = _segments(case, seed, x, v).double()
        inc = torch.rand((case["n"], 4), generator=g, device=device, dtype=torch.float32).double()
        if case["kind"] == 3:
            return torch.cat([a.look_transmittance(x, l, up), torch.ones_like(inc[:, 3:])], 1)
        if case["kind"] == 0:
            t, s = a.look_transmittance(x, v, up), a.look_in_scatter(x, v, l, up)
        else:
            t, s = a.look_track(x, x + v * segment[:, 1:], l)
        return torch.cat([inc[:, :3] * t + s * inc[:, 3:], inc[:, 3:]], 1)
    # the surrogate: the lookup at the 32-bit point corrected by the network
    x, v, l = x.float().double(), v.float().double(), l.float().double()
    above, out, layers = a.above_horizon(x, v), [], _layers(_mlp_parameters(seed), device)
    at = a.coordinates(x, v, l, above)
    sizes = (case["n0"], case["n1"], case["n2"], case["n3"])
    u = [c / (n - 1) for c, n in zip(at, sizes)]
    u += [(0.5 * (1 + _dot(x, l) / x.norm(dim=-1))).clamp(0, 1), (~above).double()] + [c - c.floor() for c in at]
    u, table = torch.stack(u, 1), a.look_in_scatter(x, v, l, above).clamp(min=0)
    for lo in range(0, len(x), 1 << 18):
        r = _network(layers, u[lo:lo + (1 << 18)])[:, :3]
        out.append(((table[lo:lo + (1 << 18)] + 1e-7) * torch.exp(r) - 1e-7).clamp(min=0))
    return torch.cat(out)
