"""The work that programs on this framework have it do, as cases that can be timed and checked.

A case is a dict of plain values; ``prepare`` builds what a program holds before the call (a
context with its scene, or device arrays), ``run`` is one pass through the public entry points,
``exact`` is the same pass restated in 64-bit torch without this package, and ``work`` counts
the bytes and operations that a pass cannot do without.

Kinds:
    wcsph    a few WCSPH steps from a given state (a restart or one env step of a rollout), the
             state given back by particle id; optionally with a floating cube coupled both ways
    pcisph   the same with the PCISPH predict-correct solver (static walls and cube)
    batch    independent WCSPH scenes of uneven size in one context
    adjoint  one optimisation step through the differentiable solver: forward, loss gradient,
             backward
    surface  one frame of the screen-space fluid surface of a context's particles
    sort     the stable (key, value) sort on device arrays
"""
import math

import numpy as np
import torch

from fluids_gb300 import capi, render, scenes, workloads

REST = 1000.0
GAMMA = 7.0
CELL_RATIO = 2.0     # support radius over spacing
CAP = 50             # neighbours kept per particle


def listed():
    return [
        # a tank of two thousand particles: an interactive toy or a unit of a parameter sweep,
        # where launches and latency are the time
        dict(name="wcsph_2k", kind="wcsph", nx=13, ny=15, nz=11, blocks=1, dx=0.015, steps=4, sigma=0.001, body=0),
        # the 65,536-particle dam break of the benchmark configurations
        dict(name="wcsph_65k", kind="wcsph", nx=32, ny=64, nz=32, blocks=1, dx=0.015, steps=4, sigma=0.001, body=0),
        # a mid-size scene with sizes that divide nothing
        dict(name="wcsph_1m", kind="wcsph", nx=79, ny=83, nz=81, blocks=2, dx=0.0077, steps=4, sigma=0.001, body=0),
        # the double dam break of the headline metric
        dict(name="wcsph_4m", kind="wcsph", nx=128, ny=128, nz=128, blocks=2, dx=0.005, steps=4, sigma=0.001, body=0),
        # a floating cube coupled both ways: its particles move, are binned and sorted every step
        dict(name="wcsph_body_41k", kind="wcsph", nx=27, ny=41, nz=37, blocks=1, dx=0.0155, steps=4, sigma=0.001,
             body=1),
        # a small PCISPH tank
        dict(name="pcisph_9k", kind="pcisph", nx=19, ny=23, nz=21, blocks=1, dx=0.0125, steps=3),
        # PCISPH at the size of the double block configuration
        dict(name="pcisph_358k", kind="pcisph", nx=40, ny=80, nz=56, blocks=2, dx=0.0125, steps=3),
        # PCISPH on the double dam break of the headline metric
        dict(name="pcisph_4m", kind="pcisph", nx=128, ny=128, nz=128, blocks=2, dx=0.005, steps=2),
        # a batch of uneven scenes, as data generation and parameter studies run them
        dict(name="batch_40", kind="batch", scenes=40, nmin=2048, nmax=65536, dx=0.015, steps=3),
        # the differentiable solver on its benchmark block of 32^3 particles
        dict(name="adjoint_32k", kind="adjoint", side=32, steps=16, every=8),
        # a full-HD frame of a million particles
        dict(name="surface_1080p", kind="surface", n=1062234, width=1920, height=1080, iterations=2),
        # the sort primitive on a million 24-bit cell keys
        dict(name="sort_1m", kind="sort", n=1062234, bits=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng, lo, hi, most):
    """Lattice sides of about 1 : a : b with lo to hi particles."""
    n = _log_int(rng, lo, hi)
    a, b = rng.uniform(0.7, 1.6), rng.uniform(0.7, 1.6)
    nx = max(3, int(round((n / (a * b)) ** (1.0 / 3.0))))
    return [min(most, max(3, int(v))) for v in (nx, round(a * nx), round(b * nx))]


def draw(rng):
    kind = rng.choices(["wcsph", "pcisph", "batch", "adjoint", "surface", "sort"], [8, 5, 2, 2, 2, 2])[0]
    if kind == "wcsph":
        blocks = rng.choice([1, 1, 2])
        nx, ny, nz = _block(rng, 1000, 2000000 // blocks, 160)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, blocks=blocks, dx=_spacing(rng, nx, ny, nz, blocks), steps=4,
                    sigma=rng.choice([0.0, 0.001, 0.001]), body=1 if blocks == 1 and rng.random() < 0.25 else 0)
    if kind == "pcisph":
        blocks = rng.choice([1, 2])
        nx, ny, nz = _block(rng, 1000, 600000 // blocks, 160)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, blocks=blocks, dx=_spacing(rng, nx, ny, nz, blocks),
                    steps=rng.choice([2, 3]))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 40), nmin=rng.choice([700, 2048]),
                    nmax=rng.choice([9000, 30000, 65536]), dx=0.015, steps=3)
    if kind == "adjoint":
        every = rng.randint(2, 9)
        return dict(kind=kind, side=rng.randint(7, 32), steps=rng.randint(every, 2 * every), every=every)
    if kind == "surface":
        w, h = rng.choice([(640, 480), (1280, 720), (1921, 1079), (1024, 1024), (333, 517)])
        return dict(kind=kind, n=_log_int(rng, 4000, 1000000), width=w, height=h, iterations=rng.choice([1, 2, 3]))
    return dict(kind=kind, n=_log_int(rng, 1000, 6000000), bits=rng.choice([16, 21, 24, 30, 32]))


def _spacing(rng, nx, ny, nz, blocks):
    """A spacing at which the blocks take up to three quarters of a 2 x 1 x 1 m tank."""
    fit = min(1.4 / (blocks * nx + 4), 0.72 / (ny + 4), 0.72 / (nz + 4))
    return round(min(0.03, fit * rng.uniform(0.8, 1.0)), 5)


# ---- scenes ---------------------------------------------------------------------------------

CONTAINER = (2.0, 1.0, 1.0)


def _dt(case):
    return (5e-4 * case["dx"] / 0.0125) if case["kind"] == "pcisph" else (2e-4 * case["dx"] / 0.015)


def _swirl(u, L):
    """A field without divergence on the box [0, L], zero with its normal part on the faces."""
    s = [torch.sin(math.pi * u[:, a] / L[a]) for a in range(3)]
    c = [torch.cos(math.pi * u[:, a] / L[a]) for a in range(3)]
    v = torch.zeros_like(u)
    for a, b, k in ((0, 1, 1.0), (1, 2, 0.7), (2, 0, 0.4)):
        v[:, a] += k * s[a] ** 2 * 2.0 * s[b] * c[b] / L[b]
        v[:, b] -= k * s[b] ** 2 * 2.0 * s[a] * c[a] / L[a]
    return v * min(L)


def _fluid(nx, ny, nz, dx, lo, gen, speed=3.0, hollow=None):
    """A block of nx x ny x nz particles that has begun to flow: the lattice carried along a
    swirl that keeps volume, jittered by 2 % of the spacing; positions and velocities (at most
    speed, as a collapsing column of a metre reaches).  hollow: a test of positions that stay empty."""
    dev = "cuda"
    ax = [torch.arange(k, dtype=torch.float64, device=dev) * dx for k in (nx, ny, nz)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    u = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
    L = [(k - 1) * dx for k in (nx, ny, nz)]
    far = min(2.0 * dx, 0.03 * min(L))
    for _ in range(8):
        v = _swirl(u, L)
        u = u + (far / 8) * _swirl(u + (far / 16) * v, L)
    vel = _swirl(u, L)
    vel = vel * (speed / vel.norm(dim=1).max())
    if hollow is not None:
        keep = ~hollow(u + torch.tensor(lo, dtype=torch.float64, device=dev))
        u, vel = u[keep], vel[keep]
    u = u + 0.02 * dx * (2.0 * torch.rand(u.shape, generator=gen, dtype=torch.float64, device=dev) - 1.0)
    return u + torch.tensor(lo, dtype=torch.float64, device=dev), vel


def _spread(a):
    a = a & 0x3ff
    a = (a | (a << 16)) & 0x30000ff
    a = (a | (a << 8)) & 0x300f00f
    a = (a | (a << 4)) & 0x30c30c3
    return (a | (a << 2)) & 0x9249249


def _in_order(p, v, container, h):
    """float32 (n, 4) positions and velocities in the cells' Morton order, as a running
    simulation holds them."""
    lo = torch.tensor([-c / 2 - 2.0 * h for c in container], dtype=torch.float64, device=p.device)
    c = ((p - lo) / h).floor().long()
    key = _spread(c[:, 0]) | (_spread(c[:, 1]) << 1) | (_spread(c[:, 2]) << 2)
    at = torch.sort(key, stable=True).indices
    pos = torch.ones((len(p), 4), dtype=torch.float32, device=p.device)
    vel = torch.zeros((len(p), 4), dtype=torch.float32, device=p.device)
    pos[:, :3], vel[:, :3] = p[at].float(), v[at].float()
    return pos, vel


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _inputs(case, seed):
    """Fluid positions and velocities of a wcsph or pcisph case."""
    gen, dx = _generator(seed), case["dx"]
    n = (case["nx"], case["ny"], case["nz"])
    W, H, _ = CONTAINER
    z0 = -(n[2] - 1) * dx / 2
    at = [(-W / 2 + dx, -H / 2 + dx, z0)]
    if case["blocks"] == 2:
        at.append((W / 2 - n[0] * dx, -H / 2 + dx, z0))
    hollow = None
    if case.get("body"):
        side, _, rot, _ = _cube(case)
        rot = torch.as_tensor(np.asarray(rot, np.float64).reshape(3, 4), device="cuda")

        def hollow(q):
            return (((q - rot[:, 3]) @ rot[:, :3]).abs() < 0.5 * side + 0.35 * dx).all(1)

    got = [_fluid(*n, dx, lo, gen, hollow=hollow) for lo in at]
    p, v = torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])
    return _in_order(p, v, CONTAINER, CELL_RATIO * dx)


def _cube(case):
    """The floating cube of a case with a body: side, points, pose, mass."""
    dx = case["dx"]
    side = 0.35 * dx * min(case["nx"], case["ny"], case["nz"])
    centre = (-1.0 + 0.5 * case["nx"] * dx, -0.5 + 0.6 * case["ny"] * dx, 0.0)
    cube = scenes.Cube(side, 0.0, centre, scenes.rotation_y(0.3))
    return side, cube.surface_sampling(dx), cube.rot3x4(), 0.4 * REST * side ** 3


def _params(case):
    if case["kind"] == "pcisph":
        return capi.make_params(capi.SPH_PCISPH, mode=capi.SPH_MODE_PHYSICS, time_step=_dt(case), max_vel=20.0,
                                particle_radius=case["dx"] / 2.0, support_radius=CELL_RATIO * case["dx"],
                                pcisph_min_iterations=3, pcisph_max_iterations=8, pcisph_error_ratio=0.01,
                                rest_density=REST, k_viscosity=1.7, gravity=9.81, surface_tension=1.0, relax_on_add=0)
    return workloads.wcsph_params(case["dx"], _dt(case), sigma=case.get("sigma", 0.001))


class _Span:
    """A context's device field for torch.as_tensor."""

    def __init__(self, ptr, shape, kind):
        self.__cuda_array_interface__ = dict(shape=shape, typestr=kind, data=(ptr, False), version=3)


def _field(ctx, name, n, width=4, kind="<f4"):
    return torch.as_tensor(_Span(ctx.device_ptr(name), (n, width) if width > 1 else (n,), kind), device="cuda")


_streams = []


def _stream():
    """The program's one work stream."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


class _Stepper:
    """A context with views of its state and the state that passes start from."""

    def __init__(self, ctx, pos, vel, steps):
        self.ctx, self.steps = ctx, steps
        self.stream = _stream()
        ctx.set_stream(self.stream.cuda_stream)
        n = len(pos)
        self.names = ["POS", "VEL"] + (["VEL_HALF"] if ctx.params.method == capi.SPH_WCSPH else [])
        self.state = [_field(ctx, f, n) for f in self.names]
        self.ids = _field(ctx, "ID", n, 1, "<i4")
        self.start = [pos, vel, vel][:len(self.names)]
        self.ids0 = torch.arange(n, dtype=torch.int32, device="cuda")
        self.pose = None
        torch.cuda.synchronize()

    def run(self):
        with torch.cuda.stream(self.stream):
            for a, b in zip(self.state, self.start):
                a.copy_(b)
            self.ids.copy_(self.ids0)
            if self.pose is not None:
                body, rot = self.pose
                self.ctx.set_body_transform(body, rot, (0.0, 0.0, 0.0, 0.0), (0.0, 0.0, 0.0, 0.0))
            self.ctx.simulate(self.steps)
            at = self.ids.long()
            out = {f.lower(): torch.empty_like(a).index_copy_(0, at, a) for f, a in zip(self.names, self.state)}
            if self.pose is not None:
                out["body_force"] = _field(self.ctx, "BODY_FORCE", 2)[1].clone()
        return out


def _prepare_steps(case, seed):
    pos, vel = _inputs(case, seed)
    ctx = capi.Context(_params(case))
    ctx.set_rect_limits(*CONTAINER)
    ctx.add_boundary(scenes.FishTank(*CONTAINER).surface_sampling(case["dx"]))
    pose = None
    if case.get("body"):
        side, pts, rot, mass = _cube(case)
        ctx.add_boundary(pts, can_move=True, rot3x4=rot, mass=mass)
        ctx.set_body_dynamics(1, True, [6.0 / (mass * side * side)] * 3, 0.0)
        pose = (1, rot)
    ctx.add_volume(pos.cpu().numpy(), vel.cpu().numpy())
    s = _Stepper(ctx, pos, vel, case["steps"])
    s.pose = pose
    return s


def _batch_scenes(case, seed):
    """Containers, parameters and fluid of each scene of a batch."""
    rng, gen, dx = np.random.default_rng(1000 + case["scenes"]), _generator(seed), case["dx"]
    got = []
    for _ in range(case["scenes"]):
        n = math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        box = (float(np.float32(rng.uniform(1.0, 3.0))), 1.0, 1.0)
        mu, c0 = math.exp(rng.uniform(math.log(1e-3), math.log(1e-1))), rng.uniform(10.0, 40.0)
        nx = max(3, round((n / 2.0) ** (1.0 / 3.0)))
        ny = max(3, min(60, round(n / (nx * nx))))
        p, v = _fluid(nx, ny, nx, dx, (box[0] / 2 - nx * dx, -0.5 + dx, -(nx - 1) * dx / 2), gen)
        pos, vel = _in_order(p, v, box, CELL_RATIO * dx)
        got.append(dict(container=box, mu=mu, kgas=REST * c0 * c0 / GAMMA, fluid=pos, vel=vel))
    return got


def _prepare_batch(case, seed):
    got = _batch_scenes(case, seed)
    descs = [dict(container=s["container"], mu=s["mu"], kgas=s["kgas"], fluid=s["fluid"].cpu().numpy(),
                  vel=s["vel"].cpu().numpy(),
                  boundary=scenes.FishTank(*s["container"]).surface_sampling(case["dx"])) for s in got]
    ctx = capi.BatchContext(workloads.wcsph_params(case["dx"], _dt(case)), descs)
    return _Stepper(ctx, torch.cat([s["fluid"] for s in got]), torch.cat([s["vel"] for s in got]), case["steps"])


ADJ_DX, ADJ_BOX, ADJ_MU, ADJ_C0 = 0.015, (2.0, 2.0, 2.0), 0.01, 20.0


def _adjoint_inputs(case, seed):
    gen, k = _generator(seed), case["side"]
    lo = -(k - 1) * ADJ_DX / 2
    p, v = _fluid(k, k, k, ADJ_DX, (lo, lo, lo), gen, speed=0.5)
    x0 = torch.ones((len(p), 4), dtype=torch.float32, device="cuda")
    v0 = torch.zeros_like(x0)
    x0[:, :3], v0[:, :3] = p.float(), v.float()
    y = x0.clone()
    y[:, :3] += 0.01 * torch.randn((len(p), 3), generator=gen, device="cuda")
    y[:, 0] += 0.01
    return x0, v0, y


class _Optimise:
    def __init__(self, case, seed):
        self.x0, self.v0, self.y = _adjoint_inputs(case, seed)
        p = workloads.wcsph_params(ADJ_DX, 2e-4, c0=ADJ_C0, mu=ADJ_MU, sigma=0.0)
        self.ctx = capi.Context(p)
        self.ctx.set_rect_limits(*ADJ_BOX)
        self.ctx.add_volume(self.x0.cpu().numpy(), self.v0.cpu().numpy())
        self.stream = _stream()
        self.ctx.set_stream(self.stream.cuda_stream)
        self.adj = capi.Adjoint(self.ctx, case["steps"], case["every"])
        torch.cuda.synchronize()

    def run(self):
        with torch.cuda.stream(self.stream):
            xT, vT, gx0, gv0 = (torch.empty_like(self.x0) for _ in range(4))
            self.adj.forward(self.x0.data_ptr(), self.v0.data_ptr(), ADJ_MU, REST * ADJ_C0 * ADJ_C0 / GAMMA,
                             out_x=xT.data_ptr(), out_v=vT.data_ptr())
            seed = (xT - self.y) * (2.0 / len(xT))
            g = self.adj.backward(seed.data_ptr(), None, out_gx0=gx0.data_ptr(), out_gv0=gv0.data_ptr())
        return dict(xT=xT[:, :3], vT=vT[:, :3], gx0=gx0[:, :3], gv0=gv0[:, :3], g_mu=g["g_mu"], g_k=g["g_k"])


class _Frame:
    def __init__(self, case, seed):
        k = round(case["n"] ** (1.0 / 3.0))
        ny = max(3, round(case["n"] / (k * k)))
        dx = min(0.9 / (max(k, ny) + 2), 0.03)
        gen = _generator(seed)
        lo = (-(k - 1) * dx / 2, -0.5 + dx, -(k - 1) * dx / 2)
        p, v = _fluid(k, ny, k, dx, lo, gen)
        pos, vel = _in_order(p, v, CONTAINER, CELL_RATIO * dx)
        self.ctx = capi.Context(workloads.wcsph_params(dx, 2e-4 * dx / 0.015))
        self.ctx.set_rect_limits(*CONTAINER)
        self.ctx.add_volume(pos.cpu().numpy(), vel.cpu().numpy())
        self.stream = _stream()
        self.ctx.set_stream(self.stream.cuda_stream)
        w, h = case["width"], case["height"]
        self.camera = render.Camera(w, h)
        self.renderer = render.SSpaceFluidRenderer(w, h, filter_iterations=case["iterations"])
        self.background = torch.rand((h, w, 4), generator=gen, device="cuda")
        self.cube = torch.rand((6, 64, 64, 4), generator=gen, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        with torch.cuda.stream(self.stream):
            s = self.stream.cuda_stream
            depth, normals = self.renderer.render(self.ctx, self.camera, self.camera.transformation(), s)
            color = self.renderer.shade(self.camera, self.background, self.cube, s)
        return dict(depth=depth, normals=normals, color=color)


class _Sort:
    def __init__(self, case, seed):
        gen = _generator(seed)
        n, bits = case["n"], case["bits"]
        # cell keys: about eight particles share one
        top = min(1 << bits, max(2, n // 8) * 4)
        self.keys0 = (torch.randint(0, top, (n,), generator=gen, device="cuda") * ((1 << bits) // top)).to(torch.int32)
        self.vals0 = torch.randint(0, 1 << 30, (n,), generator=gen, device="cuda", dtype=torch.int32)
        self.keys, self.vals = torch.empty_like(self.keys0), torch.empty_like(self.vals0)
        self.bits = bits

    def run(self):
        with torch.cuda.stream(_stream()):
            self.keys.copy_(self.keys0)
            self.vals.copy_(self.vals0)
            capi.sort_pairs_device(self.keys.data_ptr(), self.vals.data_ptr(), len(self.keys), self.bits,
                                   _stream().cuda_stream)
        return dict(keys=self.keys, vals=self.vals)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("wcsph", "pcisph"):
        return _prepare_steps(case, seed)
    return dict(batch=_prepare_batch, adjoint=_Optimise, surface=_Frame, sort=_Sort)[kind](case, seed)


def run(state):
    return state.run()


def _batch_count(case):
    rng, total = np.random.default_rng(1000 + case["scenes"]), 0
    for _ in range(case["scenes"]):
        n = math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"])))
        rng.uniform(), rng.uniform(), rng.uniform()
        nx = max(3, round((n / 2.0) ** (1.0 / 3.0)))
        total += nx * nx * max(3, min(60, round(n / (nx * nx))))
    return total


def work(case):
    """Bytes: the state in and out once a pass.  Operations: about 29 neighbours a particle, 8
    for a density pair, 12 for a normal pair, 60 for a force pair; a PCISPH step has at least
    three iterations of a density and a 20-operation force pair."""
    kind = case["kind"]
    if kind in ("wcsph", "pcisph"):
        n = case["nx"] * case["ny"] * case["nz"] * case["blocks"]
        if kind == "wcsph":
            return dict(bytes=96.0 * n, flops=29.0 * (80 if case["sigma"] else 55) * n * case["steps"])
        return dict(bytes=64.0 * n, flops=29.0 * (80 + 3 * 28) * n * case["steps"])
    if kind == "batch":
        n = _batch_count(case)
        return dict(bytes=96.0 * n, flops=29.0 * 80 * n * case["steps"])
    if kind == "adjoint":
        n = case["side"] ** 3
        return dict(bytes=32.0 * n + 80.0 * n, flops=29.0 * (2 * 48 + 110) * n * case["steps"])
    if kind == "surface":
        px = case["width"] * case["height"]
        return dict(bytes=16.0 * case["n"] + px * (4 + 16 + 16 + 16.0), flops=60.0 * case["n"] + 200.0 * px)
    return dict(bytes=16.0 * case["n"], flops=0.0)


# ---- the same in 64 bits --------------------------------------------------------------------

def _r6(x):
    """Kernel constants reach the kernels printed with six decimals."""
    return float("%.6f" % float(np.float32(x)))


class _K:
    """Kernel constants from a case's float32 parameters."""

    def __init__(self, dx, dt, pcisph=False):
        f = lambda v: float(np.float32(v))   # noqa: E731
        self.h, self.dt = f(CELL_RATIO * dx), f(dt)
        r = f(dx / 2.0)
        self.H = _r6(self.h)
        self.m = REST * (2.0 * r) ** 3
        self.M = _r6(self.m)
        h, pi = self.h, math.pi
        self.poly6 = 315.0 / (64.0 * pi * h ** 9)
        self.poly6_grad = -945.0 / (32.0 * pi * h ** 9)
        self.spiky = -45.0 / (pi * h ** 6)
        self.lapl = 45.0 / (pi * h ** 6)
        self.st_main, self.st_term = 32.0 / (pi * h ** 9), h ** 6 / 64.0
        self.g, self.vmax = -f(9.81), 20.0 if pcisph else 10.0
        if pcisph:
            self.delta = self._delta(r)

    def _delta(self, r):
        h = self.h
        x = np.arange(-h - r, h + r * 1.01, 2.0 * r)
        p = np.stack(np.meshgrid(x, x, x, indexing="ij"), -1).reshape(-1, 3)
        r2 = (p * p).sum(1)
        p, r2 = p[r2 < h * h], r2[r2 < h * h]
        rn = np.sqrt(r2)
        s = (self.spiky * (h - rn) ** 2 / rn)[:, None] * p
        v = (self.poly6_grad * (h * h - r2) ** 2)[:, None] * p
        beta = 2.0 * (self.dt * self.m / REST) ** 2
        return -1.0 / (beta * (-(s.sum(0) @ v.sum(0)) - (v * s).sum()))


@torch.no_grad()
def _pairs(a, b, h):
    """(i, j) with |a_i - b_j| < h."""
    lo = torch.minimum(a.amin(0), b.amin(0)) - 2.0 * h
    ca, cb = ((a - lo) / h).floor().long(), ((b - lo) / h).floor().long()
    dims = torch.maximum(ca.amax(0), cb.amax(0)) + 3
    ny, nz = int(dims[1]), int(dims[2])
    lin = lambda c: (c[:, 0] * ny + c[:, 1]) * nz + c[:, 2]   # noqa: E731
    kb, order = torch.sort(lin(cb))
    bs = b[order]
    ka = lin(ca)
    ii, jj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = ka + (dx * ny + dy) * nz + dz
                s = torch.searchsorted(kb, k)
                e = torch.searchsorted(kb, k, right=True)
                i = (e > s).nonzero().squeeze(1)
                s, e = s[i], e[i]
                while len(i):
                    hit = ((a[i] - bs[s]) ** 2).sum(1) < h * h
                    ii.append(i[hit])
                    jj.append(order[s[hit]])
                    s = s + 1
                    go = s < e
                    i, s, e = i[go], s[go], e[go]
    none = torch.zeros(0, dtype=torch.long, device=a.device)
    return torch.cat(ii + [none]), torch.cat(jj + [none])


def _sum(n, i, v):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, i, v)


def _within(n, i):
    """Whether no neighbour list reaches its cap (a truncated list has no 64-bit value)."""
    return not len(i) or int(torch.bincount(i, minlength=n).max()) < CAP


def _psi(pts, k):
    i, j = _pairs(pts, pts, k.H)
    t = k.H ** 2 - ((pts[i] - pts[j]) ** 2).sum(1)
    return REST / (_sum(len(pts), i, t ** 3) * k.poly6)


def _st(r, h, term):
    t = (h - r) ** 3 * r ** 3
    return torch.where(r <= 0.5 * h, 2.0 * t - term, torch.where(r <= h, t, torch.zeros_like(t)))


def _clamp(x, v):
    return x.clamp(-v, v)


def _walls(x, v, box, dt):
    """The container's clamp and reflection: (position, velocity)."""
    half = box / 2
    top = half.clone()
    top[..., 1] = 10.0
    c = torch.minimum(torch.maximum(x, -half), top)
    e = c - x
    d, vn = e.norm(dim=1), v.norm(dim=1)
    hit = (d > 0) & (vn > 0)
    s = torch.sign(e)
    s = s / s.norm(dim=1, keepdim=True).clamp_min(1e-300)
    rest = d / (dt * vn.clamp_min(1e-300))
    w = v - ((1.0 + rest) * (v * s).sum(1))[:, None] * s
    return torch.where(hit[:, None], c, x), torch.where(hit[:, None], w, v)


def _wcsph_step(k, x, v, u, kgas, mu, sigma, wall, psi, box, body=None, off=0.0):
    """One WCSPH step; kgas and mu are numbers or one value a particle, wall the boundary
    particles with their psi, box the container (None: no wall is near) around the point off,
    body a dict that the step advances.  None when a list is full."""
    n = len(x)
    i, j = _pairs(x, x, k.H)
    pts, ph = wall, psi
    if body is not None:
        bx = body["pts"] @ body["rot"].T + body["c"]
        pts, ph = torch.cat([wall, bx]), torch.cat([psi, body["psi"]])
    bi, bj = _pairs(x, pts, k.H) if len(pts) else (i[:0], j[:0])
    if not (_within(n, i) and _within(n, bi)):
        return None
    d = x[i] - x[j]
    r2 = (d * d).sum(1)
    db = x[bi] - pts[bj]
    rb2 = (db * db).sum(1)
    h, hh = k.h, k.h * k.h
    rho = k.poly6 * k.m * _sum(n, i, (hh - r2) ** 3) + k.poly6 * _sum(n, bi, (hh - rb2) ** 3 * ph[bj])
    p = kgas * ((rho / REST) ** 7 - 1.0)
    p = torch.where(p > 0, p, torch.zeros_like(p))
    C = p / rho ** 2
    if body is not None:
        qi, qj = _pairs(bx, x, k.H)
        e = x[qj] - bx[qi]
        rn = e.norm(dim=1)
        f = _sum(len(bx), qi, e * (k.spiky / rn * (k.H - rn) ** 2 * 2.0 * C[qj])[:, None])
        f = f * (k.m * body["psi"])[:, None]
        body["force"], tau = f.sum(0), torch.linalg.cross(bx - body["c"], f).sum(0)
        _move_body(body, tau, k)
    far = r2 > 1e-10
    i, j, d, r2 = i[far], j[far], d[far], r2[far]
    r = r2.sqrt()
    w = h - r
    acc = -k.m * _sum(n, i, d * (k.spiky / r * w * w * (C[i] + C[j]))[:, None])
    vs = (k.lapl * mu) * (k.m / rho)
    acc = acc + vs[:, None] * _sum(n, i, (v[j] - v[i]) * (w / rho[j])[:, None])
    if sigma:
        nrm = k.poly6_grad * k.M * k.H * _sum(n, i, d * ((k.H ** 2 - r2) ** 2 / rho[j])[:, None])
        q = 2.0 * REST / (rho[i] + rho[j])
        cu = _sum(n, i, (nrm[i] - nrm[j]) * q[:, None])
        co = _sum(n, i, d * (_st(r, h, k.st_term) * q / r)[:, None])
        acc = acc - sigma * (cu + co * (k.st_main * k.m))
    if len(bi):
        rb = rb2.sqrt()
        acc = acc + _sum(n, bi, db * (-ph[bj] * (h - rb) ** 2 / rb * 2.0 * C[bi] * k.spiky)[:, None])
    acc = acc + torch.tensor([0.0, k.g, 0.0], dtype=x.dtype, device=x.device)
    dt, vm = k.dt, k.vmax
    un = u + dt * acc
    xn = x + dt * _clamp(un + dt * acc, vm)
    if box is not None:
        xn, un = _walls(xn - off, un, box, dt)
        xn = xn + off
    return xn, _clamp(un + dt * acc * 0.5, vm), _clamp(un, vm)


def _move_body(b, tau, k):
    b["lin"] = b["lin"] + k.dt * (b["force"] / b["mass"] + torch.tensor([0.0, k.g, 0.0], dtype=tau.dtype,
                                                                        device=tau.device))
    b["c"] = b["c"] + k.dt * b["lin"]
    R = b["rot"]
    b["ang"] = b["ang"] + k.dt * (R @ (b["inv"] * (R.T @ tau)))
    wn = b["ang"].norm()
    if float(wn) > 0:
        a, th = b["ang"] / wn, wn * k.dt
        A = torch.zeros((3, 3), dtype=tau.dtype, device=tau.device)
        A[0, 1], A[0, 2], A[1, 2] = -a[2], a[1], -a[0]
        A = A - A.T
        q = torch.eye(3, dtype=tau.dtype, device=tau.device) + torch.sin(th) * A + (1 - torch.cos(th)) * (A @ A)
        b["rot"] = torch.linalg.svd(q @ R)[0] @ torch.linalg.svd(q @ R)[2]


def _pcisph_step(k, x, v, mu, sigma, wall, psi, box):
    n = len(x)
    i, j = _pairs(x, x, k.H)
    bi, bj = _pairs(x, wall, k.H)
    if not (_within(n, i) and _within(n, bi)):
        return None
    H, HH, M = k.H, k.H * k.H, k.M
    d = x[i] - x[j]
    r2 = (d * d).sum(1)
    db = x[bi] - wall[bj]
    rb2 = (db * db).sum(1)
    rho = k.poly6 * (M * _sum(n, i, (HH - r2) ** 3) + _sum(n, bi, (HH - rb2) ** 3 * psi[bj]))
    nrm = k.poly6_grad * M * H * _sum(n, i, d * ((HH - r2) ** 2 / rho[j])[:, None])
    off = r2 > 0
    fi, fj, fd, fr = i[off], j[off], d[off], r2[off].sqrt()
    q = 2.0 * REST / (rho[fi] + rho[fj])
    vis = _sum(n, fi, (v[fj] - v[fi]) * ((H - fr) / rho[fj])[:, None])
    cu = _sum(n, fi, (nrm[fi] - nrm[fj]) * q[:, None])
    co = _sum(n, fi, fd * (_st(fr, H, k.st_term) * q / fr)[:, None])
    fo = vis * (mu * M * M * k.lapl / rho)[:, None] - sigma * M * (cu + co * (M * k.st_main))
    g = torch.tensor([0.0, k.g, 0.0], dtype=x.dtype, device=x.device)
    half = box / 2
    top = half.clone()
    top[..., 1] = 10.0
    p, fp = torch.zeros_like(rho), torch.zeros_like(x)
    rb = rb2.sqrt()

    def advance():
        vv = v + _clamp((g + (fp + fo) / M) * k.dt, k.vmax)
        return x + vv * k.dt, vv

    for it in range(1, 9):
        xs = torch.minimum(torch.maximum(advance()[0], -half), top)
        r2s = ((xs[i] - xs[j]) ** 2).sum(1)
        rbs = ((xs[bi] - wall[bj]) ** 2).sum(1)
        err = k.poly6 * (M * _sum(n, i, (HH - r2s).clamp_min(0.0) ** 3) +
                         _sum(n, bi, (HH - rbs).clamp_min(0.0) ** 3 * psi[bj])) - REST
        err = err.clamp_min(0.0)
        p = p + err * k.delta
        C = p / rho ** 2
        fp = -M * M * k.spiky * _sum(n, fi, fd * ((C[fi] + C[fj]) / fr * (H - fr) ** 2)[:, None])
        fp = fp - M * k.spiky * _sum(n, bi, db * (psi[bj] * 2.0 * C[bi] / rb * (H - rb) ** 2)[:, None])
        if it >= 3 and float(err.max()) / REST < 0.01:
            break
    xn, vn = advance()
    return _walls(xn, vn, box, k.dt)


def _d(a):
    return (a if torch.is_tensor(a) else torch.as_tensor(np.asarray(a), device="cuda")).to("cuda")[..., :3].double()


def _with_w(a, w):
    return torch.cat([a, torch.full((len(a), 1), w, dtype=a.dtype, device=a.device)], 1)


def _exact_steps(case, seed):
    pos, vel = _inputs(case, seed)
    pc = case["kind"] == "pcisph"
    k = _K(case["dx"], _dt(case), pc)
    box = torch.tensor([CONTAINER], dtype=torch.float64, device="cuda")
    wall = _d(scenes.FishTank(*CONTAINER).surface_sampling(case["dx"]))
    psi = _psi(wall, k)
    x, v = _d(pos), _d(vel)
    u, body = v, None
    if case.get("body"):
        side, pts, rot, mass = _cube(case)
        rot = torch.as_tensor(np.asarray(rot, np.float32).reshape(3, 4), device="cuda").double()
        body = dict(pts=_d(pts), rot=rot[:, :3], c=rot[:, 3], mass=float(np.float32(mass)),
                    inv=float(np.float32(6.0 / (mass * side * side))), lin=torch.zeros(3, device="cuda").double(),
                    ang=torch.zeros(3, device="cuda").double())
        body["psi"] = _psi(body["pts"] @ body["rot"].T + body["c"], k)
    kgas, mu = float(np.float32(REST * 400.0 / GAMMA)), float(np.float32(0.01))
    for _ in range(case["steps"]):
        if pc:
            got = _pcisph_step(k, x, v, float(np.float32(1.7)), 1.0, wall, psi, box)
        else:
            got = _wcsph_step(k, x, v, u, kgas, mu, float(np.float32(case["sigma"])), wall, psi, box, body)
        if got is None:
            return None
        x, v, u = got if len(got) == 3 else got + (None,)
    out = dict(pos=_with_w(x, 1.0), vel=_with_w(v, 0.0))
    if not pc:
        out["vel_half"] = _with_w(u, 0.0)
    if body is not None:
        out["body_force"] = torch.cat([body["force"], torch.zeros(1, dtype=torch.float64, device="cuda")])
    return out


def _exact_batch(case, seed):
    """All scenes at once, set so far apart that no pair spans two of them."""
    got = _batch_scenes(case, seed)
    k = _K(case["dx"], _dt(case))
    row = lambda v, n: torch.full((n,), float(np.float32(v)), dtype=torch.float64, device="cuda")   # noqa: E731
    xs, vs, walls, kg, mu, box, off = [], [], [], [], [], [], []
    for s, sc in enumerate(got):
        n, shift = len(sc["fluid"]), torch.tensor([8.0 * s, 0.0, 0.0], dtype=torch.float64, device="cuda")
        xs.append(_d(sc["fluid"]))
        vs.append(_d(sc["vel"]))
        walls.append(_d(scenes.FishTank(*sc["container"]).surface_sampling(case["dx"])) + shift)
        kg.append(row(sc["kgas"], n))
        mu.append(row(sc["mu"], n))
        box.append(torch.tensor([sc["container"]], dtype=torch.float64, device="cuda").expand(n, 3))
        off.append(shift.expand(n, 3))
    x, v, wall, box, off = torch.cat(xs), torch.cat(vs), torch.cat(walls), torch.cat(box), torch.cat(off)
    kg, mu, psi, u = torch.cat(kg), torch.cat(mu), _psi(wall, k), v
    x = x + off
    for _ in range(case["steps"]):
        got = _wcsph_step(k, x, v, u, kg, mu, float(np.float32(0.001)), wall, psi, box, off=off)
        if got is None:
            return None
        x, v, u = got
    return dict(pos=_with_w(x - off, 1.0), vel=_with_w(v, 0.0), vel_half=_with_w(u, 0.0))


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint
    x0, v0, y = (_d(a) for a in _adjoint_inputs(case, seed))
    k = _K(ADJ_DX, 2e-4)
    none, no = torch.zeros((0, 3), dtype=torch.float64, device="cuda"), torch.zeros(0, device="cuda").double()
    kg = torch.tensor(float(np.float32(REST * ADJ_C0 * ADJ_C0 / GAMMA)), dtype=torch.float64, device="cuda")
    mu = torch.tensor(float(np.float32(ADJ_MU)), dtype=torch.float64, device="cuda")
    for t in (x0, v0, kg, mu):
        t.requires_grad_(True)
    x, v, u = x0, v0, v0

    def step(x, v, u, kg, mu):
        got = _wcsph_step(k, x, v, u, kg, mu, 0.0, none, no, None)
        if got is None:
            raise ValueError("a full list")
        return got

    try:
        for _ in range(case["steps"]):
            x, v, u = checkpoint(step, x, v, u, kg, mu, use_reentrant=False)
    except ValueError:
        return None
    seed_grad = 2.0 * (x.detach() - y) / len(x)
    gx, gv, gk, gm = torch.autograd.grad(x, (x0, v0, kg, mu), seed_grad)
    return dict(xT=x.detach(), vT=v.detach(), gx0=gx, gv0=gv, g_mu=float(gm), g_k=float(gk))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("wcsph", "pcisph"):
        return _exact_steps(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return None   # an image's silhouettes and a sort have no value between two others
