"""The work that users of this framework have it do, as cases that can be timed.

A case is a simulation stepped through the package's public calls (GpuBubble, GpuBatch): a state is a bubble,
or a batch of them, with its initial fields; one pass steps it by some time steps at its present frame time and
streams the thickness, the surfactant and both velocity components to the caller's page-locked buffers, as a
program that shows or stores frames does.  After `span` steps the simulation starts again from its initial
fields (the upload belongs to that pass), so that any number of passes stays in the part of a run that the case
stands for: a soap film that is whole.  `request` cases make their bubble anew in every pass, as a serving
loop does for a request that it runs on its own.

Fields keep to the benchmark's recipes: thickness 1 + a * (smooth random field of a band of degrees),
surfactant 1 + noise of one percent (or a smooth field), a wind of largest speed 1 from a random stream
function, velocities from rest.  A random field of degree k is a sum of plane waves of wave number k in space,
read on the sphere.  All of them are rounded to FP32, so that every precision starts from the same numbers.
"""
import math

import numpy as np
import torch

STATE = ("eta", "gamma", "u_theta", "u_phi")


# -- the cases ----------------------------------------------------------------------------------------------


def _case(name, nThetas, steps, span, **more):
    """`nThetas`: the grid rows of the members, as text; one member is a single bubble."""
    c = {"name": name, "form": "single" if "," not in nThetas else "batch", "nThetas": nThetas, "steps": steps,
         "span": span, "dt": 0.005, "radius": 1.0, "t0": 0.0, "band": "1-4", "amplitude": 0.1, "surfactant": "noise",
         "thin": 1.0, "spread": 0.0, "storage": "fp32", "solver": "mixed", "bimocq": True, "rk2": True}
    c.update(more)
    return c


_C1 = dict(dt=0.002, band="8-32", amplitude=0.2)
_C2 = dict(dt=0.001, band="8-24", amplitude=0.2, surfactant="smooth")


def listed():
    return [
        # the smallest benchmark grid stepped one step at a time, as an interactive viewer does: latency and launches
        _case("c0_step", "64", 1, 100),
        # a frame of the shipped config.txt: 256 x 512, a bubble of 5 cm, four steps of 5 ms
        _case("config_frame", "256", 4, 200, radius=0.05, band="2-12"),
        # the headline benchmark, 512 x 1024: a frame of ten steps of a wind-blown film that drains
        _case("c1_frame", "512", 10, 200, **_C1),
        # the same with the plain FP32 solve and without the characteristic maps, the cheaper switches of a quick look
        _case("c1_plain", "512", 10, 200, solver="plain", bimocq=False, rk2=False, **_C1),
        # a film that has drained: thin at the top, where the surfactant system is stiff and takes many iterations
        _case("c1_drained", "512", 5, 60, thin=0.01, t0=0.4, **_C1),
        # the largest grid, 1024 x 2048
        _case("c2_frame", "1024", 5, 200, **_C2),
        # the largest grid with the thickness and surfactant stored in BF16
        _case("c2_bf16", "1024", 5, 200, storage="bf16", **_C2),
        # the batched ensemble: uneven grids, gravity, air viscosity and Marangoni coefficient +-50 % per member
        _case("ensemble", "512,64,256,128,512,64,128,256,64,512,128,64,256,512,128,64,256", 5, 50, spread=0.5),
        # serving many small requests at once, each at its own frame time
        _case("serving_small", ",".join(["64,64,128,64,64"] * 7), 10, 50, spread=0.5, t0=0.3),
        # a request that is run on its own: its bubble made, filled, stepped for three frames, each frame streamed
        _case("request", "128", 30, 30, form="request"),
    ]


def draw(rng):
    form = rng.choice(["single", "single", "single", "batch", "request"])
    nT = rng.choice([32, 64, 128, 256, 512, 1024])
    more = dict(rng.choice([dict(), _C1, _C2]))
    more["t0"] = rng.choice([0.0, round(rng.uniform(0.05, 2.5), 3)])
    more["storage"] = rng.choice(["fp32", "fp32", "bf16"])
    more["solver"] = rng.choice(["mixed", "mixed", "plain"])
    more["rk2"] = rng.random() < 0.8
    more["bimocq"] = rng.random() < 0.8
    more["amplitude"] = round(rng.uniform(0.05, 0.25), 3)
    if form == "batch":
        most, sizes = rng.choice([256, 512]), []
        for _ in range(rng.randint(2, 45)):
            n = rng.choice([32, 64, 128, 256, 512])
            if n <= most and sum(2 * m * m for m in sizes + [n]) <= 2_400_000:
                sizes.append(n)
        sizes = sizes if len(sizes) > 1 else [64, 32, 128]
        more["spread"] = round(rng.uniform(0.05, 0.5), 3)
        names, steps = ",".join(map(str, sizes)), rng.randint(1, 5)
    else:
        names = str(min(nT, 256) if form == "request" else nT)
        steps = rng.randint(5, 30) if form == "request" else rng.randint(1, {1024: 5, 512: 10}.get(nT, 16))
    if more["solver"] == "mixed" and form == "single" and rng.random() < 0.2:
        more["thin"] = 0.01
    c = _case("", names, steps, max(steps, 60), **more)
    c["form"] = form
    del c["name"]
    return c


def _sizes(case):
    return [int(n) for n in str(case["nThetas"]).split(",")]


def work(case):
    """One step reads the state and writes the next one: per cell the four state fields (thickness and
    surfactant in their storage), with the characteristic maps two displacements (three floats each) there and
    back, a third one read, the reference fields and accumulated changes of both scalars (all of the
    thickness's, two of the surfactant's) read and two accumulators written, and the wind (initial wind and
    corridor factor of both components) read.  About 3000 operations per cell and step with the maps
    (two great-circle traces, nine map samples and their positions, two velocity advections, the scalar samples,
    a few solver iterations), 1200 without."""
    s = 2 if case["storage"] == "bf16" else 4
    cell = 2 * (2 * s + 8) + 16
    if case["bimocq"]:
        cell += 2 * 24 + 12 + 3 * s + 3 * 4 + 8
    cells = sum(2 * n * n for n in _sizes(case)) * case["steps"]
    return {"bytes": cells * cell, "flops": cells * (3000 if case["bimocq"] else 1200)}


# -- inputs -------------------------------------------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Waves:
    """A random smooth function on the sphere: plane waves of wave numbers in [lo, hi]."""

    def __init__(self, lo, hi, gen, count=24):
        k = torch.randn(count, 3, generator=gen, dtype=torch.float64)
        size = lo + (hi - lo) * torch.rand(count, 1, generator=gen, dtype=torch.float64)
        self.k = k / k.norm(dim=1, keepdim=True) * size
        self.a = torch.randn(count, generator=gen, dtype=torch.float64)
        self.phase = 2 * math.pi * torch.rand(count, generator=gen, dtype=torch.float64)

    def value(self, x):
        v = 0
        for k, a, p in zip(self.k.tolist(), self.a.tolist(), self.phase.tolist()):
            v = v + a * torch.cos(k[0] * x[0] + k[1] * x[1] + k[2] * x[2] + p)
        return v

    def gradient(self, x):
        g = [0, 0, 0]
        for k, a, p in zip(self.k.tolist(), self.a.tolist(), self.phase.tolist()):
            s = -a * torch.sin(k[0] * x[0] + k[1] * x[1] + k[2] * x[2] + p)
            g = [g[c] + k[c] * s for c in range(3)]
        return g


def _fields(case, nT, seed):
    """Initial fields of one member, float64 tensors holding FP32 values."""
    gen = torch.Generator().manual_seed(seed)
    nP, h, dev = 2 * nT, math.pi / nT, _device()
    i = torch.arange(nT, dtype=torch.float64, device=dev)[:, None]
    j = torch.arange(nP, dtype=torch.float64, device=dev)[None, :]

    def point(th, ph):
        return [torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th) + 0 * ph]

    centre = point((i + 0.5) * h, j * h)
    lo, hi = (float(v) for v in case["band"].split("-"))
    f = _Waves(lo, hi, gen).value(centre)
    eta = 1 + case["amplitude"] * f / f.abs().max()
    if case["thin"] < 1:  # thickness falling off smoothly towards the top
        x = (((i + 0.5) * h - 0.3) / 0.9).clamp(0, 1)
        eta = eta * (case["thin"] + (1 - case["thin"]) * x * x * (3 - 2 * x))
    if case["surfactant"] == "smooth":
        f = _Waves(0, 16, gen).value(centre)
        gamma = 1 + 0.05 * f / f.abs().max()
    else:
        u = torch.rand(nT, nP, generator=gen, dtype=torch.float64).to(dev)
        gamma = 1 + 0.01 * (2 * u - 1)
    psi = _Waves(1, 8, gen)

    def wind(th, ph, component):
        x, g = point(th, ph), psi.gradient(point(th, ph))
        w = [x[1] * g[2] - x[2] * g[1], x[2] * g[0] - x[0] * g[2], x[0] * g[1] - x[1] * g[0]]
        if component == "phi":
            return -torch.sin(ph) * w[0] + torch.cos(ph) * w[1]
        return torch.cos(th) * (torch.cos(ph) * w[0] + torch.sin(ph) * w[1]) - torch.sin(th) * w[2]

    uair, vair = wind((i + 0.5) * h, (j - 0.5) * h, "phi"), wind((i[:-1] + 1) * h, j * h, "theta")
    top = max(float(uair.abs().max()), float(vair.abs().max()))
    out = {"eta": eta, "gamma": gamma, "u_theta": torch.zeros(nT - 1, nP, device=dev), "u_phi": torch.zeros(nT, nP, device=dev),
           "uair_init": uair / top, "vair_init": vair / top}
    return {k: v.float().double() for k, v in out.items()}


def _members(case, seed):
    """(rows, scales of gravity, air viscosity and Marangoni coefficient, frame time, seed) of every member."""
    rng = np.random.default_rng(seed)
    out = []
    for n, nT in enumerate(_sizes(case)):
        scales = [float(v) for v in 1 + case["spread"] * rng.uniform(-1, 1, 3)]
        t = case["t0"] if n == 0 else case["t0"] * float(rng.uniform(0, 2))
        out.append((nT, scales, t, int(rng.integers(1 << 40))))
    return out


# -- the passes ---------------------------------------------------------------------------------------------


def _params(case, nT, scales):
    from soapbubble_gb300.bubble import make_params
    return make_params(nT, case["dt"], radius=case["radius"], gs_scale=scales[0], nu_scale=scales[1], M_scale=scales[2],
                       storage=1 if case["storage"] == "bf16" else 0, solver_mode=1 if case["solver"] == "plain" else 0,
                       plain_advection=0 if case["bimocq"] else 1, single_step_velocity=0 if case["rk2"] else 1)


def prepare(case, seed):
    from soapbubble_gb300.bubble import GpuBatch, GpuBubble
    members = _members(case, seed)
    fields = [{k: v.cpu().numpy() for k, v in _fields(case, m[0], m[3]).items()} for m in members]
    state = {"case": case, "members": members, "fields": fields, "done": 0, "batch": None, "bubbles": []}
    if case["form"] != "request":
        for (nT, scales, _, _), f in zip(members, fields):
            g = GpuBubble(_params(case, nT, scales))
            g.upload_fields(**f)
            state["bubbles"].append(g)
        if case["form"] == "batch":
            state["batch"] = GpuBatch(state["bubbles"])
    # one page-locked buffer per field, the members one after the other
    count = {k: [f[k].size for f in fields] for k in STATE}
    host = {k: torch.empty(sum(n), dtype=torch.float32, pin_memory=torch.cuda.is_available()) for k, n in count.items()}
    state["out"] = {k: v.numpy() for k, v in host.items()}
    state["host"] = host
    state["parts"] = [{k: state["out"][k][sum(count[k][:m]):sum(count[k][:m + 1])] for k in STATE} for m in range(len(members))]
    return state


def _request(state):
    """A request's life: its bubble made and filled, frames of ten steps streamed, the final state read."""
    from soapbubble_gb300.bubble import GpuBubble
    case, (nT, scales, t0, _), out = state["case"], state["members"][0], state["parts"][0]
    with GpuBubble(_params(case, nT, scales)) as g:
        g.upload_fields(**state["fields"][0])
        for k in range(0, case["steps"], 10):
            n = min(10, case["steps"] - k)
            g.step(n, t0 + k * case["dt"], case["dt"])
            if k + n < case["steps"]:
                g.download_f32("eta", out["eta"])
                g.synchronize()
        for name in STATE:
            g.download_f32(name, out[name])
        g.synchronize()
    return state["out"]


def run(state):
    case = state["case"]
    if case["form"] == "request":
        return _request(state)
    if state["done"] + case["steps"] > case["span"]:
        for g, f in zip(state["bubbles"], state["fields"]):
            g.upload_fields(eta=f["eta"], gamma=f["gamma"], u_theta=f["u_theta"], u_phi=f["u_phi"])
        state["done"] = 0
    # time stands still within a frame of ten steps
    t = (state["done"] // 10) * 10 * case["dt"]
    state["done"] += case["steps"]
    if state["batch"] is None:
        g = state["bubbles"][0]
        g.step(case["steps"], case["t0"] + t, case["dt"])
        for name in STATE:
            g.stage_download_f32(name, state["parts"][0][name])
        return state["out"]
    state["batch"].step(case["steps"], [m[2] + t for m in state["members"]], case["dt"])
    state["batch"].synchronize()
    for g, part in zip(state["bubbles"], state["parts"]):
        for name in STATE:
            g.download_f32(name, part[name])
    for g in state["bubbles"]:
        g.synchronize()
    return state["out"]


# -- the same in 64 bits ------------------------------------------------------------------------------------


class _Film:
    """The time step in FP64, whole-array, for a film without holes.  Points are Cartesian unit vectors in one
    fixed frame; a characteristic map is an array of them."""

    def __init__(self, case, nT, scales, f):
        self.nT, self.nP, self.h = nT, 2 * nT, math.pi / nT
        self.bimocq, self.rk2 = case["bimocq"], case["rk2"]
        # air, water and film constants of the model; lengths in radii, speeds in m/s
        r, H, gas = case["radius"], 1e-6, 8.3144598 * 298.15
        self.M = 1e-6 * gas / (3 * 1e3 * H) * scales[2]
        self.Cr = 1.184 * math.sqrt(1.562e-5 * scales[1] * r) / (1e3 * H)
        self.gs = 9.8 * r * scales[0]
        self.evap = -3e-8 * r / H
        self.blend, self.radius = 0.5, r
        self.dt = case["dt"] / r
        d = f["eta"].device
        self.i = torch.arange(nT, dtype=torch.float64, device=d)[:, None].expand(nT, self.nP)
        self.j = torch.arange(self.nP, dtype=torch.float64, device=d)[None, :].expand(nT, self.nP)
        self.sin_c = torch.sin((self.i + 0.5) * self.h)
        edge = torch.sin(torch.arange(nT + 1, dtype=torch.float64, device=d) * self.h)
        edge[0] = edge[-1] = 0.0
        self.sin_n, self.sin_s = edge[:-1, None], edge[1:, None]
        self.eta, self.gam, self.uth, self.uph = f["eta"], f["gamma"], f["u_theta"], f["u_phi"]
        self.uair0, self.vair0 = f["uair_init"], f["vair_init"]
        self.corr_u = self.corridor((self.i + 0.5) * self.h, (self.j - 0.5) * self.h, "phi")
        self.corr_v = self.corridor((self.i[:-1] + 1) * self.h, self.j[:-1] * self.h, "theta")
        self.home = self.point(self.i + 0.5, self.j)
        self.fwd = self.bwd = self.prev = self.home
        zero = torch.zeros_like(self.eta)
        self.init, self.delta = [self.eta, self.gam], [zero, zero]
        self.initL, self.deltaL = [self.eta, self.gam], [zero, zero]

    def corridor(self, th, ph, component):
        """The wind corridor around the great circle through the poles and phi = 0."""
        st, ct, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
        x = [st * cp, st * sp, ct]
        n = [0.0, -1.0, math.cos(math.pi / 2)]  # normal of the corridor's plane
        dn = sum(a * b for a, b in zip(n, x))
        beta = torch.acos(dn.clamp(-1, 1))
        p = [b - dn * a for a, b in zip(n, x)]
        size = torch.sqrt(p[0] ** 2 + p[1] ** 2 + p[2] ** 2)
        p = [v / size for v in p]
        w = [n[1] * p[2] - n[2] * p[1], n[2] * p[0] - n[0] * p[2], n[0] * p[1] - n[1] * p[0]]
        s = (((beta - math.pi / 2).abs() - 0.2) / 0.2).clamp(0, 1)
        s = 0.5 * torch.sin(beta) * self.radius * (1 - s * s * (3 - 2 * s))
        if component == "phi":
            return s * (-sp * w[0] + cp * w[1])
        return s * (ct * cp * w[0] + ct * sp * w[1] - st * w[2])

    # positions in grid units: theta / h, phi / h
    def point(self, t, p):
        t, p = t * self.h, p * self.h
        return torch.stack([torch.sin(t) * torch.cos(p), torch.sin(t) * torch.sin(p), torch.cos(t)], -1)

    def position(self, x):
        return torch.atan2(torch.hypot(x[..., 0], x[..., 1]), x[..., 2]) / self.h, torch.atan2(x[..., 1], x[..., 0]) / self.h

    def stencil(self, t, p, shift=0.0):
        """Corner indices of a cell-centred bilinear sample, fractions, and which rows lie across a pole."""
        t, p = t - 0.5, p - shift
        lo, left = torch.floor(t), torch.floor(p)
        a, b = t - lo, p - left
        lo, left = lo.long().clamp(-1, self.nT - 1), left.long()
        over0, over1 = lo < 0, lo + 1 > self.nT - 1
        r0, r1 = lo.clamp(min=0), (lo + 1).clamp(max=self.nT - 1)
        col = [torch.remainder(left + c + over.long() * self.nT, self.nP) for over in (over0, over1) for c in (0, 1)]
        return [r0 * self.nP + col[0], r0 * self.nP + col[1], r1 * self.nP + col[2], r1 * self.nP + col[3]], a, b, over0, over1

    @staticmethod
    def scalar(f, s):
        (i00, i01, i10, i11), a, b, _, _ = s
        f = f.reshape(-1)
        return (1 - a) * ((1 - b) * f[i00] + b * f[i01]) + a * ((1 - b) * f[i10] + b * f[i11])

    def at_uphi(self, t, p):
        (i00, i01, i10, i11), a, b, o0, o1 = self.stencil(t, p, -0.5)
        f = self.uph.reshape(-1)
        low, up = (1 - b) * f[i00] + b * f[i01], (1 - b) * f[i10] + b * f[i11]
        return (1 - a) * torch.where(o0, -low, low) + a * torch.where(o1, -up, up)

    def at_utheta(self, t, p):
        """Rows at theta / h = 1 .. nT - 1; beside a pole the nearest row and its reflection two cells away."""
        nT, nP, f = self.nT, self.nP, self.uth.reshape(-1)
        s, left = t - 1, torch.floor(p)
        b, left = p - left, left.long()
        lo = torch.floor(s).long().clamp(-1, nT - 1)
        north, south = lo < 0, lo >= nT - 2
        r0 = torch.where(south, nT - 2, lo).clamp(min=0)
        r1 = torch.where(north, 0, torch.where(south, nT - 2, lo + 1))
        a = torch.where(north, 0.5 * (s + 2), torch.where(south, 0.5 * (s - (nT - 2)), s - lo))
        c = [torch.remainder(left + k + o.long() * nT, nP) for o in (north, south) for k in (0, 1)]
        low = (1 - b) * f[r0 * nP + c[0]] + b * f[r0 * nP + c[1]]
        up = (1 - b) * f[r1 * nP + c[2]] + b * f[r1 * nP + c[3]]
        return (1 - a) * torch.where(north, -low, low) + a * torch.where(south, -up, up)

    def trace(self, t, p, gt, gp, dt, rk2):
        """The great-circle departure point of (t, p): the point, the final direction, its normal and the arc."""
        th, ph = t * self.h, p * self.h
        w = self.point(t, p)
        e_t = torch.stack([torch.cos(th) * torch.cos(ph), torch.cos(th) * torch.sin(ph), -torch.sin(th)], -1)
        e_p = torch.stack([-torch.sin(ph), torch.cos(ph), 0 * ph], -1)

        def direction(u):
            n = u.norm(dim=-1, keepdim=True)
            u_ = torch.where(n > 0, u / torch.where(n > 0, n, torch.ones_like(n)), e_p)
            return n, u_, torch.cross(w, u_, dim=-1)

        n, u_, v_ = direction(gt[..., None] * e_t + gp[..., None] * e_p)
        moving = n > 0
        if rk2:
            s = -0.5 * n * dt
            mid, du = torch.cos(s) * w + torch.sin(s) * u_, torch.cos(s) * u_ - torch.sin(s) * w
            mu, dv = self.velocity(mid), torch.cross(mid, du, dim=-1)
            n, u_, v_ = direction((mu * du).sum(-1, keepdim=True) * u_ + (mu * dv).sum(-1, keepdim=True) * v_)
            moving = moving & (n > 0)
        s = -n * dt * moving
        return torch.cos(s) * w + torch.sin(s) * u_, u_, v_, s, moving, (w, e_t, e_p)

    def velocity(self, x):
        """The velocity at points, as vectors."""
        t, p = self.position(x)
        th, ph = t * self.h, p * self.h
        e_t = torch.stack([torch.cos(th) * torch.cos(ph), torch.cos(th) * torch.sin(ph), -torch.sin(th)], -1)
        e_p = torch.stack([-torch.sin(ph), torch.cos(ph), 0 * ph], -1)
        return self.at_utheta(t, p)[..., None] * e_t + self.at_uphi(t, p)[..., None] * e_p

    def carried(self, t, p, gt, gp, component):
        """A velocity component advected with parallel transport along the trace."""
        x, u_, v_, s, moving, (w, e_t, e_p) = self.trace(t, p, gt, gp, self.dt, self.rk2)
        v = self.velocity(x)
        du = torch.cos(s) * u_ - torch.sin(s) * w
        dv = torch.cross(x, du, dim=-1)
        back = (v * du).sum(-1, keepdim=True) * u_ + (v * dv).sum(-1, keepdim=True) * v_
        return torch.where(moving[..., 0], (back * (e_p if component == "phi" else e_t)).sum(-1), 0.0)

    @staticmethod
    def slerp(a, b, f):
        f = f[..., None]
        W = 2 * torch.asin((0.5 * (b - a).norm(dim=-1, keepdim=True)).clamp(max=1))
        near = W < 1e-9
        sw = torch.where(near, torch.ones_like(W), torch.sin(W))
        return torch.where(near, (1 - f) * a + f * b, (torch.sin((1 - f) * W) * a + torch.sin(f * W) * b) / sw)

    def at_map(self, m, s):
        (i00, i01, i10, i11), a, b, _, _ = s
        m = m.reshape(-1, 3)
        return self.slerp(self.slerp(m[i00], m[i01], b), self.slerp(m[i10], m[i11], b), a)

    def five(self, m):
        """The map at the five sample points of every cell, with their weights."""
        for w, dt, dp in ((0.125, -0.25, -0.25), (0.125, 0.25, -0.25), (0.125, -0.25, 0.25), (0.125, 0.25, 0.25), (0.5, 0.0, 0.0)):
            yield w, self.stencil(*self.position(self.at_map(m, self.stencil(self.i + 0.5 + dt, self.j + dp))))

    def solve(self, dmass, east, south, rhs):
        """A x = rhs by conjugate gradients, preconditioned by every row's mean coefficients (a circulant)."""
        north = torch.cat([torch.zeros_like(south[:1]), south[:-1]])
        west = torch.roll(east, 1, 1)

        def A(x):
            y = dmass * x + east * (x - torch.roll(x, -1, 1)) + west * (x - torch.roll(x, 1, 1))
            y[:-1] += south[:-1] * (x[:-1] - x[1:])
            y[1:] += north[1:] * (x[1:] - x[:-1])
            return y

        k = torch.arange(self.nP // 2 + 1, dtype=torch.float64, device=rhs.device)
        symbol = (dmass + south + north).mean(1, keepdim=True) + 2 * east.mean(1, keepdim=True) * (1 - torch.cos(2 * math.pi * k / self.nP))
        scale = torch.sqrt((dmass + south + north + east + west).mean(1, keepdim=True) / (dmass + south + north + east + west))

        def B(r):
            return scale * torch.fft.irfft(torch.fft.rfft(scale * r) / symbol, n=self.nP)

        x, r = torch.zeros_like(rhs), rhs
        z = B(r)
        p, rz, stop = z, (r * z).sum(), 1e-26 * (rhs * rhs).sum()
        for n in range(3000):
            q = A(p)
            alpha = rz / (p * q).sum()
            x, r = x + alpha * p, r - alpha * q
            z = B(r)
            new = (r * z).sum()
            p, rz = z + new / rz * p, new
            if n % 8 == 7 and bool((r * r).sum() <= stop):
                break
        return x

    def step(self, t):
        nT, h, dt = self.nT, self.h, self.dt
        i, j = self.i, self.j
        # advection of gamma, the maps and the velocities
        gt, gp = self.at_utheta(i + 0.5, j), self.at_uphi(i + 0.5, j)
        back = self.stencil(*self.position(self.trace(i + 0.5, j, gt, gp, dt, True)[0]))
        gam = self.scalar(self.gam, back)
        uph = self.carried(i + 0.5, j - 0.5, self.at_utheta(i + 0.5, j - 0.5), self.uph, "phi")
        uth = self.carried(i[:-1] + 1, j[:-1], self.uth, self.at_uphi(i[:-1] + 1, j[:-1]), "theta")
        if self.bimocq:
            ahead = self.stencil(*self.position(self.trace(i + 0.5, j, gt, gp, -dt, True)[0]))
            fwd, bwd = self.at_map(self.fwd, ahead), self.at_map(self.bwd, back)
            eta = 0
            for w, s1 in self.five(bwd):
                s2 = self.stencil(*self.position(self.at_map(self.prev, s1)))
                d = self.scalar(self.delta[0], s1)
                eta = eta + w * ((1 - self.blend) * (self.scalar(self.initL[0], s2) + d + self.scalar(self.deltaL[0], s2)) +
                                 self.blend * (self.scalar(self.init[0], s1) + d))
            eta = eta.clamp(min=0)
        else:
            eta = self.scalar(self.eta, back)
        wind = 3.0 - abs(t - 3.0)
        uair, vair = self.uair0 + wind * self.corr_u, self.vair0 + wind * self.corr_v
        # the implicit surfactant system, for the increment of gamma
        mA, mB = t / 12.0, 1.0 - t / 12.0

        def mirrored(f):  # entry nP - j of the flat row, the next row's first one at j = 0
            flat = torch.cat([f.reshape(-1), f.new_zeros(1)])
            at = (self.i[: f.shape[0]] * self.nP + self.nP - self.j[: f.shape[0]]).long()
            return flat[at]

        um, vm = 0.5 * (uair * mA + mirrored(uair) * mB), 0.5 * (vair * mA - mirrored(vair) * mB)
        none = torch.zeros_like(um[:1])
        vN, vS, aN, aS = torch.cat([none, uth]), torch.cat([uth, none]), torch.cat([none, vm]), torch.cat([vm, none])
        pole = [torch.roll(eta[k:k + 1], nT, 1) for k in (0, nT - 1)]
        eN, eS = torch.cat([pole[0], eta[:-1]]), torch.cat([eta[1:], pole[1]])
        eW, eE = torch.roll(eta, 1, 1), torch.roll(eta, -1, 1)
        fN, fS, fW, fE = ((v + eta) / 2 for v in (eN, eS, eW, eE))
        c = self.Cr * dt
        rN, rS, rW, rE = (1 / (v + c) for v in (fN, fS, fW, fE))
        south = (self.sin_s * self.M * dt * rS / h**2).clone()
        south[-1] = 0
        east = self.M * dt * rE / h**2 / self.sin_c
        uE, umE = torch.roll(uph, -1, 1), torch.roll(um, -1, 1)
        div = (uE * fE * rE - uph * fW * rW + vS * self.sin_s * fS * rS - vN * self.sin_n * fN * rN) / h
        div = div + c / h * (umE * rE - um * rW + aS * self.sin_s * rS - aN * self.sin_n * rN)
        div = div + self.gs * dt / h * (self.sin_s**2 * fS * rS - self.sin_n**2 * fN * rN)
        lap = east * (gam - torch.roll(gam, -1, 1)) + torch.roll(east, 1, 1) * (gam - torch.roll(gam, 1, 1))
        lap[:-1] += south[:-1] * (gam[:-1] - gam[1:])
        lap[1:] += south[:-1] * (gam[1:] - gam[:-1])
        dx = self.solve(self.sin_c / (dt * gam), east, south, -div - lap)
        # forces, thickness, increments
        new = gam + dx
        d_eta = eta * torch.where(new > 2 * gam, 1.0, dx / gam) + self.evap * dt
        d_eta = torch.maximum(d_eta, -eta)
        self.eta, self.gam = eta + d_eta, new
        self.uph = (uph / dt * fW - self.M * (new - torch.roll(new, 1, 1)) / h / self.sin_c + self.Cr * uair) / (fW / dt + self.Cr)
        f = fS[:-1]
        self.uth = ((uth / dt + self.gs * self.sin_s[:-1]) * f - self.M * (new[1:] - new[:-1]) / h + self.Cr * vair) / (f / dt + self.Cr)
        if self.bimocq:
            self.accumulate(fwd, bwd, [d_eta, dx])

    def accumulate(self, fwd, bwd, change):
        delta, there = list(self.delta), [0, 0]
        for w, s in self.five(fwd):
            for k, now in enumerate((self.eta, self.gam)):
                delta[k] = delta[k] + w * self.scalar(change[k], s)
                there[k] = there[k] + w * self.scalar(now, s)

        def apart(a, b):
            x = self.at_map(b, self.stencil(*self.position(a)))
            return float((2 * torch.asin((0.5 * (x - self.home).norm(dim=-1)).clamp(max=1))).max()) / self.h

        self.delta, self.fwd, self.bwd = delta, fwd, bwd
        if max(apart(fwd, bwd), apart(bwd, fwd)) <= 4:
            return
        # new maps from here on, the fields corrected by the round trip's error
        error = [(there[k] - delta[k] - self.init[k]) * 0.5 for k in (0, 1)]
        now = [self.eta, self.gam]
        right = list(now)
        for w, s in self.five(bwd):
            right = [right[k] - w * self.scalar(error[k], s) for k in (0, 1)]
        for k in (0, 1):
            f = now[k]
            rows = torch.cat([torch.roll(f[:1], self.nT, 1), f, torch.roll(f[-1:], self.nT, 1)])
            near = [torch.roll(rows[1 + a:1 + a + self.nT], b, 1) for a in (-1, 0, 1) for b in (-1, 0, 1)]
            low, high = near[0], near[0]
            for v in near[1:]:
                low, high = torch.minimum(low, v), torch.maximum(high, v)
            right[k] = torch.minimum(torch.maximum(right[k], low), high).clamp(min=0)
        self.eta, self.gam = right
        self.initL, self.deltaL, self.prev = self.init, self.delta, bwd
        self.init, self.delta = right, [torch.zeros_like(v) for v in right]
        self.fwd = self.bwd = self.home


def exact(case, seed):
    """The first pass of a new state in FP64."""
    parts = {k: [] for k in STATE}
    for nT, scales, t0, sub in _members(case, seed):
        film = _Film(case, nT, scales, _fields(case, nT, sub))
        for n in range(case["steps"]):
            film.step(t0 + ((n // 10) * 10 * case["dt"] if case["form"] == "request" else 0.0))
        for k, v in zip(STATE, (film.eta, film.gam, film.uth, film.uph)):
            parts[k].append(v.reshape(-1).cpu().numpy())
    return {k: np.concatenate(v) for k, v in parts.items()}
