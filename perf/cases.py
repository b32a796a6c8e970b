"""Timed cases of the step engine: what a DEM user has it do, through its public entry points.

A simulation program holds an :class:`Engine`, advances it by the steps of one output interval and takes
the state back to the host (the reference's main loop: ``device_dem_verlet_verlet`` per step, then
``copyFromDevice``).  So most passes are ``step(K)`` followed by ``export``, in both precisions, both contact
laws, dense and sparse, still and flowing, closed and periodic, one scene and many.  One more stands for
a host that hands a state over with its contact history and takes it back.

Every scene is made here from its seed: a random close packing of spheres (a relaxed periodic tile, repeated
and relaxed against the walls of its box) for the beds, a jittered lattice for the sparse ones.
"""
import math
import types

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
YOUNG, POISSON, DENSITY = 5e6, 0.3, 2500.0


# --------------------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: a hundred spheres in a 12-triangle box, the reference's own mode (FP64,
        # linear law) with its short skin; launches and latency are all there is
        dict(name="box-100-fp64-linear", kind="bed", n=100, r0=1e-2, precision="fp64", model="linear", steps=100,
             dt=1e-5, faces=1, skin=0.1, flow=0.05),
        # a small validation run: a few thousand polydisperse spheres in FP64
        dict(name="bed-3k-fp64-hertz", kind="bed", n=3001, r0=2e-3, precision="fp64", model="hertz_mindlin", steps=50,
             dt=2e-6, faces=4, skin=0.0, flow=0.2),
        # the reference's mode at the size of an ordinary production bed
        dict(name="bed-40k-fp64-linear", kind="bed", n=40_000, r0=2e-3, precision="fp64", model="linear", steps=50,
             dt=2e-6, faces=13, skin=0.0, flow=0.02),
        # the largest FP64 bed: reference-exact runs of a dense bed
        dict(name="bed-300k-fp64-hertz", kind="bed", n=300_000, r0=1e-3, precision="fp64", model="hertz_mindlin",
             steps=20, dt=1e-6, faces=24, skin=0.0, flow=0.02),
        # a small mixed-precision bed, as parameter studies run by the thousand
        dict(name="bed-2k-mixed-hertz", kind="bed", n=2000, r0=2e-3, precision="mixed", model="hertz_mindlin",
             steps=100, dt=2e-6, faces=4, skin=0.0, flow=0.02),
        # ordinary mixed-precision beds with each law
        dict(name="bed-30k-mixed-hertz", kind="bed", n=30_011, r0=2e-3, precision="mixed", model="hertz_mindlin",
             steps=100, dt=2e-6, faces=13, skin=0.0, flow=0.02),
        dict(name="bed-250k-mixed-linear", kind="bed", n=250_000, r0=1e-3, precision="mixed", model="linear",
             steps=100, dt=1e-6, faces=24, skin=0.0, flow=0.05),
        # the production bed: a million spheres on some 36,000 triangles that may move, so the mesh
        # tree is rebuilt in every step
        dict(name="bed-1M-mixed-hertz", kind="bed", n=1_000_000, r0=1e-3, precision="mixed", model="hertz_mindlin",
             steps=100, dt=1e-6, faces=55, skin=0.0, flow=0.02, tree=True),
        # a pour: spheres raining in at the large time step of a filling run, with list rebuilds on the way
        dict(name="pour-300k-mixed-hertz", kind="pour", n=300_007, r0=1e-3, precision="mixed", model="hertz_mindlin",
             steps=200, dt=2e-5, faces=24, skin=0.0, flow=0.3),
        # a dilute channel, periodic in x, with rolling friction
        dict(name="channel-1M-mixed-hertz", kind="channel", n=1_000_000, r0=1e-3, precision="mixed",
             model="hertz_mindlin", steps=100, dt=1e-6, faces=110, skin=0.0, flow=0.5),
        # an ensemble of independent boxes with materials of their own, packed into one engine
        dict(name="ensemble-48-mixed-hertz", kind="ensemble", n=96_000, r0=1e-3, precision="mixed",
             model="hertz_mindlin", steps=100, dt=1e-6, faces=4, skin=0.0, flow=0.05, scenes=48),
        # the host hands the state over with its contact history, steps and takes it back with it (a host
        # program that couples every output interval)
        dict(name="handover-20k-mixed-linear", kind="handover", n=20_000, r0=2e-3, precision="mixed", model="linear",
             steps=20, dt=2e-6, faces=8, skin=0.0, flow=0.02),
    ]


# spheres times steps of the dearest listed case: a drawn one stays below
_SPHERE_STEPS = {"fp64": 6.0e6, "mixed": 1.0e8}


def draw(rng):
    kind = rng.choice(["bed", "bed", "bed", "bed", "pour", "channel", "ensemble", "handover"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    precision = rng.choice(["fp64", "mixed"]) if kind in ("bed", "pour", "handover") else "mixed"
    model = rng.choice(["linear", "hertz_mindlin"]) if kind != "ensemble" else "hertz_mindlin"
    top = {"bed": 300_000 if precision == "fp64" else 1_000_000, "pour": 100_000 if precision == "fp64" else 300_000,
           "channel": 1_000_000, "ensemble": 200_000, "handover": 20_000}[kind]
    low = {"bed": 100, "pour": 2000, "channel": 50_000, "ensemble": 20_000, "handover": 1000}[kind]
    n = log(low, top)
    r0 = rng.choice([1e-3, 2e-3])
    steps = min(rng.choice([20, 37, 50, 64, 100]), max(1, int(_SPHERE_STEPS[precision] / n)))
    c = dict(kind=kind, n=n, r0=r0, precision=precision, model=model, steps=steps,
             dt=(1e-5 if kind == "pour" else 1e-6) * r0 / 1e-3, faces=rng.randint(1, 1 + int(0.45 * n ** (1 / 3))),
             skin=rng.choice([0.0, 0.0, 0.4]), flow=rng.choice([0.02, 0.05, 0.2]))
    if kind == "bed":
        c["tree"] = rng.random() < 0.25
    if kind == "channel":
        c["faces"] = int(rng.uniform(0.4, 0.85) * _channel_sites(n)[2])
    if kind == "ensemble":
        c.update(scenes=rng.randint(5, 64), faces=rng.randint(1, 6))
    return c


# --------------------------------------------------------------------------- scenes

def _join(start, count, want):
    """For each entry of `want` (indices into start/count), every position of its run: (entry, position)."""
    c = count[want]
    e = torch.repeat_interleave(torch.arange(want.numel(), device=want.device), c)
    first = torch.cumsum(c, 0) - c
    return e, start[want][e] + torch.arange(e.numel(), device=want.device) - first[e]


class _Cells:
    """Positions sorted into cells of side >= `side`; with `period`, x wraps."""

    def __init__(self, x, side, period=None):
        lo = x.amin(0) - 1e-9
        self.lo, self.wrap = lo, period is not None
        ext = x.amax(0) + 1e-9 - lo
        self.side = torch.full((3,), side, dtype=F64, device=x.device)
        self.dim = [max(1, int(math.floor(float(e) / side)) + 1) for e in ext]
        if period is not None:
            self.lo = torch.stack([torch.tensor(period[0], dtype=F64, device=x.device), lo[1], lo[2]])
            self.dim[0] = int(math.floor((period[1] - period[0]) / side))
            self.side[0] = (period[1] - period[0]) / self.dim[0]
        self.c = torch.minimum(((x - self.lo) / self.side).floor().long().clamp_(min=0),
                               torch.tensor(self.dim, device=x.device) - 1)
        ident = self.id(self.c[:, 0], self.c[:, 1], self.c[:, 2])
        self.order = torch.sort(ident, stable=True).indices
        self.count = torch.bincount(ident, minlength=self.dim[0] * self.dim[1] * self.dim[2])
        self.start = torch.cumsum(self.count, 0) - self.count

    def id(self, a, b, c):
        return (a * self.dim[1] + b) * self.dim[2] + c

    def pairs(self, keep):
        """Directed pairs (i, j), j != i, within neighbouring cells for which keep(i, j) holds, sorted by (i, j)."""
        n, out = self.c.shape[0], []
        everyone = torch.arange(n, device=self.c.device)
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                for d in (-1, 0, 1):
                    t = self.c + torch.tensor([a, b, d], device=self.c.device)
                    ok = (t[:, 1] >= 0) & (t[:, 1] < self.dim[1]) & (t[:, 2] >= 0) & (t[:, 2] < self.dim[2])
                    if self.wrap:
                        t[:, 0] %= self.dim[0]
                    else:
                        ok &= (t[:, 0] >= 0) & (t[:, 0] < self.dim[0])
                    who = everyone[ok]
                    e, p = _join(self.start, self.count, self.id(t[ok, 0], t[ok, 1], t[ok, 2]))
                    i, j = who[e], self.order[p]
                    k = (i != j) & keep(i, j)
                    out.append(i[k] * n + j[k])
        key = torch.cat(out).sort().values
        return key // n, key % n


def _rows(i, j, n, width):
    """Partners of each i (pairs sorted by i) as an (n, width) table, n where there is none."""
    count = torch.bincount(i, minlength=n)
    rank = torch.arange(i.numel(), device=i.device) - (torch.cumsum(count, 0) - count)[i]
    t = torch.full((n, width), n, device=i.device)
    k = rank < width
    t[i[k], rank[k]] = j[k]
    return t


def _relax(x, r, table, sweeps, clamp, period=None):
    """Overlaps pushed apart, half of each by either sphere, sweep by sweep."""
    n = x.shape[0]
    far = torch.full((1, 3), 1e9, dtype=F64, device=x.device)
    rr = torch.cat([r, r.new_zeros(1)])
    reach = r[:, None] + rr[table]
    for _ in range(sweeps):
        d = x[:, None, :] - torch.cat([x, far])[table]
        if period is not None:
            d -= torch.where(d.abs() < 1e8, period * torch.round(d / period), torch.zeros_like(d))
        dist = d.square().sum(-1).sqrt()
        push = (reach - dist).clamp_(min=0.0)
        push = torch.where(table < n, push, torch.zeros_like(push))
        x = x + 0.3 * (d * (push / dist.clamp(min=1e-12))[:, :, None]).sum(1)
        x = clamp(x)
    return x


def _tile(m, radii, fill, rng):
    """m spheres closely packed in a periodic cube: (positions, radii, side)."""
    r = torch.as_tensor(radii, dtype=F64, device=DEV)
    side = float((4.0 / 3.0 * math.pi * (r ** 3).sum() / fill) ** (1.0 / 3.0))
    x = torch.as_tensor(rng.random((m, 3)) * side, device=DEV)
    for sweeps in (8, 12, 20, 30, 50, 80, 120):
        gap = torch.zeros((m, m), dtype=F64, device=DEV)
        for a in range(3):
            d = x[:, None, a] - x[None, :, a]
            gap += (d - side * torch.round(d / side)).square_()
        gap = gap.sqrt_() - r[:, None] - r[None, :]
        gap.fill_diagonal_(1e9)
        table = torch.topk(gap, min(24, m - 1), largest=False).indices
        x = _relax(x, r, table, sweeps, lambda y: y % side, side)
    return x, r, side


def _box(lo, hi, k):
    """Closed box, each face k x k quads of two triangles: (12 k^2, 3, 3)."""
    axis = [np.linspace(lo[a], hi[a], k + 1) for a in range(3)]
    out = []
    for a in range(3):
        b, c = (a + 1) % 3, (a + 2) % 3
        for end, flip in ((0, True), (k, False)):
            g = np.zeros((k + 1, k + 1, 3))
            g[..., a] = axis[a][end]
            g[..., b] = axis[b][:, None]
            g[..., c] = axis[c][None, :]
            p, q, s, t = g[:-1, :-1], g[1:, :-1], g[1:, 1:], g[:-1, 1:]
            for tri in ((p, q, s), (p, s, t)):
                tri = np.stack([v.reshape(-1, 3) for v in tri], 1)
                out.append(tri[:, ::-1] if flip else tri)
    return np.ascontiguousarray(np.concatenate(out))


def _radii(n, r0, rng):
    """Log-normal sizes, sigma 0.15, cut at 0.6 and 1.6 of the median."""
    return r0 * np.clip(np.exp(0.15 * rng.standard_normal(n)), 0.6, 1.6)


def _bed(n, r0, faces, rng):
    """n closely packed spheres in a closed box with room above them: (x, r, triangles)."""
    m = int(min(max(n, 400), 3000))
    x, r, side = _tile(m, _radii(m, r0, rng), 0.60, rng)
    x = (x + torch.as_tensor(rng.random(3) * side, device=DEV)) % side
    volume = float((4.0 / 3.0 * math.pi * r ** 3).mean()) * n / 0.60
    w = volume ** (1.0 / 3.0)
    reps = [math.ceil(w / side) + 1, math.ceil(1.5 * w / side) + 1, math.ceil(w / side) + 1]
    shift = torch.cartesian_prod(*[torch.arange(k, dtype=F64, device=DEV) for k in reps]) * side
    x = (x[None] + shift[:, None]).reshape(-1, 3)
    r = r.repeat(shift.shape[0])
    inside = (x >= 0.8 * r[:, None]).all(1) & (x[:, 0] <= w - 0.8 * r) & (x[:, 2] <= w - 0.8 * r)
    x, r = x[inside], r[inside]
    low = torch.sort(x[:, 1], stable=True).indices[:n]
    assert low.numel() == n
    perm = torch.as_tensor(rng.permutation(n), device=DEV)  # ids say nothing about places
    x, r = x[low][perm], r[low][perm]
    top = float((x[:, 1] + r).max()) + 4.0 * r0
    # against the walls: into the box, the neighbours pushed on
    cells = _Cells(x, 2.0 * 1.6 * r0 + 0.4 * r0)
    i, j = cells.pairs(lambda a, b: (x[a] - x[b]).square().sum(1) < (r[a] + r[b] + 0.3 * r0) ** 2)
    table = _rows(i, j, n, 20)
    lo = 0.9995 * r[:, None]
    hi = torch.stack([w - 0.9995 * r, top - r, w - 0.9995 * r], 1)
    x = _relax(x, r, table, 80, lambda y: torch.minimum(torch.maximum(y, lo), hi))
    tris = _box((0.0, 0.0, 0.0), (w, top, w), faces)
    return x.cpu().numpy(), r.cpu().numpy(), tris


def _lattice(n, lo, step, dims, jitter, rng):
    """n of the lattice's sites in a random order, jittered."""
    s = rng.permutation(dims[0] * dims[1] * dims[2])[:n]
    x = np.stack([s % dims[0], s // (dims[0] * dims[2]), (s // dims[0]) % dims[2]], 1) * np.asarray(step) + np.asarray(lo)
    return x + (rng.random((n, 3)) - 0.5) * jitter


def _pour(n, r0, faces, rng):
    """n spheres falling through a tall closed box."""
    r = _radii(n, r0, rng)
    a = 2.0 * 1.6 * r0 * 1.03
    k = math.ceil(n ** (1.0 / 3.0))
    layers = math.ceil(n / (k * k))
    w = (k + 1) * a
    x = _lattice(n, [a, 1.7 * r0, a], [a, a, a], (k, layers, k), 0.05 * r0, rng)
    return x, r, _box((0.0, 0.0, 0.0), (w, (layers + 3) * a, w), faces)


def _channel_sites(n):
    """Lattice sites of the channel along x, y and z: twice as long as wide, and low."""
    ny = max(4, round(0.32 * n ** (1.0 / 3.0)))
    nz = max(6, math.ceil(math.sqrt(n / (2.0 * ny))))
    return 2 * nz, ny, nz


def _channel(n, r0, faces, rng):
    """Dilute spheres over a corrugated floor between side walls, periodic in x: (x, r, triangles, box)."""
    r = np.where(rng.random(n) < 0.7, r0, 1.5 * r0)
    a = 3.0 * r0 * 1.05
    nx, ny, nz = _channel_sites(n)
    length, width, amp = nx * a, (nz + 1) * a, r0
    gx, gz = np.linspace(0.0, length, 2 * faces + 1), np.linspace(0.0, width, faces + 1)
    X, Z = np.meshgrid(gx, gz, indexing="ij")
    Y = amp * np.sin(2 * math.pi * 5 * X / length) * np.cos(2 * math.pi * 3 * Z / width)
    p = np.stack([X, Y, Z], -1)
    c = [p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]]
    c = [v.reshape(-1, 3) for v in c]
    tris = [np.stack([c[0], c[1], c[2]], 1), np.stack([c[0], c[2], c[3]], 1)]
    top = 2.0 * amp + 2.0 * r0 + ny * a + 4.0 * r0
    for z in (0.0, width):
        xs = np.linspace(0.0, length, 9)
        for u, v in zip(xs[:-1], xs[1:]):
            q = [np.array([u, -2 * amp, z]), np.array([v, -2 * amp, z]), np.array([v, top, z]), np.array([u, top, z])]
            tris.append(np.array([[q[0], q[1], q[2]], [q[0], q[2], q[3]]]))
    x = _lattice(n, [0.5 * a, amp + 1.6 * r0, a], [a, a, a], (nx, ny, nz), 0.14 * r0, rng)
    lo, hi = np.array([0.0, -3 * amp, -4 * r0]), np.array([length, top + 20 * r0, width + 4 * r0])
    return x, r, np.concatenate(tris), (lo, hi)


def _stiffness(r0):
    return 4.0 / 3.0 * (YOUNG * 0.5) * math.sqrt(r0 * 0.5) * math.sqrt(0.05 * r0)


def _eta(k, e):
    le = math.log(e)
    return -2.0 * le * np.sqrt(k / (math.pi ** 2 + le * le))


def _contacts(x, r, per=None):
    """Touching pairs (i, j), both directions, by (i, j)."""
    xt, rt = torch.as_tensor(x, device=DEV), torch.as_tensor(r, device=DEV)
    cells = _Cells(xt, 2.0 * float(rt.max()) * 1.001)
    return cells.pairs(lambda a, b: (xt[a] - xt[b]).square().sum(1) < (rt[a] + rt[b]) ** 2)


def _scene(case, seed):
    """The inputs of a case, as plain arrays."""
    rng = np.random.default_rng([int(seed), 77])
    n, r0, kind = case["n"], case["r0"], case["kind"]
    s = types.SimpleNamespace(mu=0.5, e=0.5, mu_roll=0.0, box=None, mu_p=None, e_p=None, history=None, stride=0)
    if kind in ("bed", "handover"):
        s.x, s.r, s.tris = _bed(n, r0, case["faces"], rng)
    elif kind == "pour":
        s.x, s.r, s.tris = _pour(n, r0, case["faces"], rng)
        s.e = 0.3
    elif kind == "channel":
        s.x, s.r, s.tris, s.box = _channel(n, r0, case["faces"], rng)
        s.mu_roll = 0.05 if case["model"] == "hertz_mindlin" else 0.0
    else:
        # boxes of uneven sizes on a square grid, far enough apart never to meet
        k = case["scenes"]
        share = np.exp(rng.uniform(0.0, math.log(8.0), k))
        sizes = np.maximum(20, np.floor(n * share / share.sum())).astype(int)
        sizes[0] += max(0, n - int(sizes.sum()))
        parts, pitch = [_bed(int(q), r0, case["faces"], rng) for q in sizes], 0.0
        pitch = max(float(t.max()) for _, _, t in parts) + 16.0 * r0
        side = math.ceil(k ** (1.0 / 3.0))
        at = [pitch * np.array([q % side, (q // side) % side, q // (side * side)], float) for q in range(k)]
        s.x = np.concatenate([x + o for (x, _, _), o in zip(parts, at)])
        s.r = np.concatenate([r for _, r, _ in parts])
        s.tris = np.concatenate([t + o for (_, _, t), o in zip(parts, at)])
        s.mu_p = np.repeat(rng.uniform(0.2, 0.7, k), sizes)
        s.e_p = np.repeat(rng.uniform(0.3, 0.9, k), sizes)
    n = s.n = s.x.shape[0]
    s.m = DENSITY * 4.0 / 3.0 * math.pi * s.r ** 3
    s.k = np.full(n, _stiffness(r0))
    s.eta = _eta(s.k, s.e)
    s.v = rng.normal(0.0, case["flow"], (n, 3))
    if kind == "pour":
        s.v[:, 1] -= 0.5
    s.w = rng.normal(0.0, case["flow"] / r0, (n, 3))
    s.g = np.array([0.0, -9.81, 0.0])
    rmax = float(s.r.max())
    s.skin = case["skin"] * rmax if case["skin"] > 0 else -1.0
    if kind == "handover":
        # the history of every touching pair, with small springs
        i, j = (a.cpu().numpy() for a in _contacts(s.x, s.r))
        s.stride = 32
        cnt = np.bincount(i, minlength=n)
        rank = np.arange(i.size) - (np.cumsum(cnt) - cnt)[i]
        h = dict(numCont=cnt.astype(np.int32), numContWall=np.zeros(n, np.int32))
        ind = np.full((n, s.stride), -1, np.int32)
        ind[i, rank] = j
        h["indHis"] = ind.reshape(-1)
        h["indHisWall"] = np.full(n * s.stride, -1, np.int32)
        for c in "xyz":
            d = np.zeros((n, s.stride))
            d[i, rank] = rng.normal(0.0, 1e-4 * r0, i.size)
            h["deltHis" + c] = d.reshape(-1)
            h["deltHis%sWall" % c] = np.zeros(n * s.stride)
        s.history = h
    return s


# --------------------------------------------------------------------------- what a program does

def prepare(case, seed):
    from gpudem_gb300.engine import Engine
    from gpudem_gb300.scenes import Scene
    s = _scene(case, seed)
    v = s.tris.reshape(-1, 3)
    scene = Scene(x=s.x, r=s.r, m=s.m, k=s.k, eta=s.eta, mu=s.mu, dt=case["dt"], tris=s.tris, inlet_lo=v.min(0) - 0.01,
                  inlet_hi=v.max(0) + 0.01, g=s.g, v=s.v, w=s.w, skin=s.skin, E=YOUNG, nu=POISSON, e=s.e,
                  mu_roll=s.mu_roll, history=s.history, hist_stride=s.stride, mu_p=s.mu_p, e_p=s.e_p, box=s.box,
                  periodic_x=s.box is not None)
    engine = Engine(scene, precision=case["precision"], model=case["model"], bvh_every_step=bool(case.get("tree")))
    return types.SimpleNamespace(engine=engine, scene=scene, steps=case["steps"], handover=case["kind"] == "handover")


def run(state):
    e = state.engine
    if state.handover:
        e.import_particles(state.scene, history=state.scene.history, hist_stride=state.scene.hist_stride)
        e.step(state.steps)
        return e.export(history=True, hist_stride=state.scene.hist_stride)
    e.step(state.steps)
    return e.export(history=False)


# mean contacts of a sphere (each pair counted for both), by kind
_TOUCHING = {"bed": 5.0, "handover": 5.0, "ensemble": 4.5, "pour": 0.2, "channel": 0.2}


def work(case):
    n, k, c = case["n"], case["steps"], _TOUCHING[case["kind"]]
    # a step reads position, velocity, spin, radius and mass and writes the first three, and reads and
    # writes each contact's spring and partner; positions and velocities are FP64 or float pairs alike,
    # the springs FP64 or (mixed) FP32 with their compensation terms
    step = n * 8 * (11 + 9) + n * c * 2 * (3 * 8 + 4)
    if case["kind"] == "handover":
        state = n * (8 * 13 + 4) + n * 2 * (4 + 32 * (4 + 3 * 8))
        return {"bytes": k * step + 2 * state, "flops": n * k * (60 + 150 * c)}
    return {"bytes": k * step + n * (8 * 13 + 4), "flops": n * k * (60 + 150 * c)}


# --------------------------------------------------------------------------- the same in plain 64 bits

def _dot(a, b):
    return (a * b).sum(-1)


class _Springs:
    """Tangential springs of the contacts, row by row in the order of encounter; a row ends at its first lost
    contact, as the reference's bookkeeping leaves it."""

    def __init__(self, n, m):
        self.n, self.m = n, m
        self.key = torch.zeros(0, dtype=torch.long, device=DEV)
        self.slot = self.key.clone()
        self.d = torch.zeros((0, 3), dtype=F64, device=DEV)
        self.rows = torch.zeros(n, dtype=torch.long, device=DEV)

    def find(self, i, j):
        """Slots and springs of this step's contacts (i, j), sorted by i and in the order they are met."""
        key = i * self.m + j
        at = torch.searchsorted(self.key, key).clamp_(max=max(0, self.key.numel() - 1))
        old = self.key[at] == key if self.key.numel() else torch.zeros_like(key, dtype=torch.bool)
        fresh = (~old).long()
        before = torch.cumsum(fresh, 0) - fresh
        first = torch.searchsorted(i, i)
        slot = self.rows[i] + before - before[first] if i.numel() else i
        d = torch.zeros((i.numel(), 3), dtype=F64, device=DEV)
        if self.key.numel():
            slot = torch.where(old, self.slot[at], slot)
            d = torch.where(old[:, None], self.d[at], d)
        self.rows = self.rows + torch.zeros_like(self.rows).scatter_add_(0, i, fresh)
        return slot, d

    def keep(self, i, j, slot, d):
        """The rows after the step: every slot before the first untouched one."""
        width = int(self.rows.max()) + 1 if self.n else 1
        touched = torch.zeros((self.n, width + 1), dtype=torch.bool, device=DEV)
        touched[i, slot] = True
        self.rows = torch.minimum((~touched).long().argmax(1), self.rows)
        k = slot < self.rows[i]
        key, order = torch.sort(i[k] * self.m + j[k])
        self.key, self.slot, self.d = key, slot[k][order], d[k][order]


class _Exact:
    """The step in 64 bits, vectorised over the contacts."""

    def __init__(self, case, s):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=DEV)
        self.x, self.v, self.w = t(s.x).clone(), t(s.v).clone(), t(s.w).clone()
        self.r, self.m, self.k, self.eta, self.g = t(s.r), t(s.m), t(s.k), t(s.eta), t(s.g)
        self.n, self.dt, self.hertz, self.roll = s.n, case["dt"], case["model"] == "hertz_mindlin", s.mu_roll
        self.rmax = float(s.r.max())
        self.inv_m = 1.0 / self.m
        self.inv_i = 1.0 / (0.4 * self.m * self.r * self.r)
        es, gs = YOUNG / (2 * (1 - POISSON ** 2)), YOUNG / (4 * (1 + POISSON) * (2 - POISSON))
        self.kn, self.sn, self.kt = 4.0 / 3.0 * es, 2.0 * es, 8.0 * gs
        e = t(s.e_p) if s.e_p is not None else torch.full((s.n,), s.e, dtype=F64, device=DEV)
        self.mu = t(s.mu_p) if s.mu_p is not None else torch.full((s.n,), s.mu, dtype=F64, device=DEV)
        le = torch.log(e)
        self.damp = -2.0 * math.sqrt(5.0 / 6.0) * le / torch.sqrt(le * le + math.pi ** 2)
        self.period = None if s.box is None else (float(s.box[0][0]), float(s.box[1][0]))
        tri = t(s.tris)
        self.a = tri[:, 0]
        self.ab, self.ac, self.bc = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0], tri[:, 2] - tri[:, 1]
        nrm = torch.linalg.cross(self.ab, self.ac)
        self.nrm = nrm / nrm.norm(dim=1, keepdim=True)
        self.tlo, self.thi = tri.amin(1), tri.amax(1)
        corner = np.unique(np.round(s.tris.reshape(-1, 3) / 1e-9).astype(np.int64), axis=0, return_inverse=True)[1]
        corner = corner.reshape(-1, 3)
        edge = np.concatenate([corner[:, [1, 2]], corner[:, [0, 2]], corner[:, [0, 1]]])
        edge = np.unique(np.sort(edge, 1), axis=0, return_inverse=True)[1].reshape(3, -1).T + corner.max() + 1
        self.feature = torch.as_tensor(np.concatenate([corner, edge], 1), device=DEV)
        self.features = int(self.feature.max()) + 1
        self.spring, self.wall = _Springs(s.n, s.n), _Springs(s.n, len(s.tris))
        if s.history is not None:
            cnt = torch.as_tensor(s.history["numCont"], device=DEV).long()
            i = torch.repeat_interleave(torch.arange(s.n, device=DEV), cnt)
            q = torch.arange(i.numel(), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[i]
            j = torch.as_tensor(s.history["indHis"], device=DEV).long().reshape(s.n, -1)[i, q]
            d = torch.stack([t(s.history["deltHis" + c]).reshape(s.n, -1)[i, q] for c in "xyz"], 1)
            self.spring.rows = cnt
            self.spring.key, order = torch.sort(i * s.n + j)
            self.spring.slot, self.spring.d = q[order], d[order]
        self.lists()

    def image(self, d):
        if self.period is not None:
            span = self.period[1] - self.period[0]
            d = d.clone()
            d[:, 0] -= span * torch.round(d[:, 0] / span)
        return d

    def lists(self):
        """Candidate pairs and candidate triangles for a while: those within half a radius of touching."""
        self.margin, self.at = 0.5 * self.rmax, self.x.clone()
        cells = _Cells(self.x, 2.0 * self.rmax + self.margin, self.period)
        near = lambda a, b: self.image(self.x[a] - self.x[b]).square().sum(1) < (self.r[a] + self.r[b] + self.margin) ** 2
        self.i, self.j = cells.pairs(near)
        # triangles: the cells that each one's box, grown by the reach, covers
        reach = self.rmax + self.margin
        c0 = ((self.tlo - reach - cells.lo) / cells.side).floor().long()
        c1 = ((self.thi + reach - cells.lo) / cells.side).floor().long()
        top = torch.tensor(cells.dim, device=DEV) - 1
        axes = (1, 2) if self.period is not None else (0, 1, 2)
        for a in axes:
            c0[:, a].clamp_(min=0)
            c1[:, a] = torch.minimum(c1[:, a], top[a])
        if self.period is not None:
            c1[:, 0] = torch.minimum(c1[:, 0], c0[:, 0] + top[0])
        span = (c1 - c0 + 1).clamp_(min=0)
        total = span.prod(1)
        t = torch.repeat_interleave(torch.arange(total.numel(), device=DEV), total)
        q = torch.arange(t.numel(), device=DEV) - (torch.cumsum(total, 0) - total)[t]
        cz = c0[t, 2] + q % span[t, 2]
        cy = c0[t, 1] + (q // span[t, 2]) % span[t, 1]
        cx = c0[t, 0] + q // (span[t, 2] * span[t, 1])
        if self.period is not None:
            cx = cx % cells.dim[0]
        e, p = _join(cells.start, cells.count, cells.id(cx, cy, cz))
        i, t = cells.order[p], t[e]
        x = self.near(i, t)
        d = torch.maximum(self.tlo[t] - x, x - self.thi[t]).clamp_(min=0)
        k = d.square().sum(1) < (self.r[i] + self.margin) ** 2
        key = (i[k] * self.nrm.shape[0] + t[k]).sort().values
        self.wi, self.wt = key // self.nrm.shape[0], key % self.nrm.shape[0]

    def near(self, i, t):
        """Centre i at its image nearest triangle t."""
        return self.a[t] + self.image(self.x[i] - self.a[t])

    def tangential(self, nrm, fn2, vt, gt, kt, mu, d):
        d = d + vt * self.dt
        d = d - _dot(d, nrm)[:, None] * nrm
        f = -kt[:, None] * d
        f2 = _dot(f, f)
        slip = f2 > mu * mu * fn2
        cap = f * (mu * torch.sqrt(fn2) / (torch.sqrt(f2) + 1e-15))[:, None]
        return torch.where(slip[:, None], cap, f - gt[:, None] * vt), torch.where(slip[:, None], -cap / kt[:, None], d)

    def law(self, i, nrm, lap, rstar, mstar, vr, spin, d, rel):
        """Force and torque on i of contacts with normal `nrm`, overlap `lap`; the springs after it."""
        vn = _dot(vr, nrm)
        if self.hertz:
            root = torch.sqrt(rstar * lap)
            gn = self.damp[i] * torch.sqrt(self.sn * root * mstar)
            fn = (self.kn * root * lap - gn * vn)[:, None] * nrm
            kt = self.kt * root
            gt = self.damp[i] * torch.sqrt(kt * mstar)
        else:
            kt = self.k[i]
            gt = self.eta[i] * torch.sqrt(mstar)
            fn = (kt * lap - gt * vn)[:, None] * nrm
        vt = (vr - vn[:, None] * nrm) + torch.linalg.cross(spin, nrm)
        fn2 = _dot(fn, fn)
        ft, d = self.tangential(nrm, fn2, vt, gt, kt, self.mu[i], d)
        tq = self.r[i][:, None] * torch.linalg.cross(nrm, ft)
        if self.roll > 0:
            size = rel.norm(dim=1, keepdim=True)
            tq = tq - torch.where(size > 0, (self.roll * rstar * torch.sqrt(fn2))[:, None] * rel / size.clamp(min=1e-300), torch.zeros_like(rel))
        return fn + ft, tq, d

    def closest(self, i, t):
        """Centre of i minus the feature of triangle t that the reference's classification picks: (vector, feature or -1)."""
        p = self.near(i, t) - self.a[t]
        ab, ac, bc = self.ab[t], self.ac[t], self.bc[t]
        d00, d01, d11 = _dot(ab, ab), _dot(ab, ac), _dot(ac, ac)
        d20, d21 = _dot(p, ab), _dot(p, ac)
        den = d00 * d11 - d01 * d01
        v, w = (d11 * d20 - d01 * d21) / den, (d00 * d21 - d01 * d20) / den
        u = 1.0 - v - w
        part = lambda q, e: q - (_dot(q, e) / _dot(e, e)).clamp(0, 1)[:, None] * e
        nrm = self.nrm[t]
        choice = [(u > 0) & (v > 0) & (w > 0), (v <= 0) & (w <= 0), (u <= 0) & (w <= 0), (u <= 0) & (v <= 0), u <= 0, v <= 0]
        vec = [_dot(p, nrm)[:, None] * nrm, p, p - ab, p - ac, part(p - ab, bc), part(p, ac), part(p, ab)]
        f = self.feature[t]
        ids = [torch.full_like(t, -1), f[:, 0], f[:, 1], f[:, 2], f[:, 3], f[:, 4], f[:, 5]]
        out, hit = vec[6], ids[6]
        for c, a, b in list(zip(choice, vec, ids))[::-1]:
            out, hit = torch.where(c[:, None], a, out), torch.where(c, b, hit)
        plane = _dot(p, nrm).abs()
        return out, hit, plane <= self.r[i]

    def step(self):
        if bool((self.image(self.x - self.at).square().sum(1) > (0.45 * self.margin) ** 2).any()):
            self.lists()
        force, torque = torch.zeros_like(self.x), torch.zeros_like(self.x)
        # sphere on sphere
        d = self.image(self.x[self.i] - self.x[self.j])
        d2, reach = _dot(d, d), self.r[self.i] + self.r[self.j]
        k = d2 < reach * reach
        i, j, d, reach = self.i[k], self.j[k], d[k], reach[k]
        dist = torch.sqrt(d2[k])
        slot, s = self.spring.find(i, j)
        ri, rj = self.r[i], self.r[j]
        f, q, s = self.law(i, d / dist[:, None], reach - dist, ri * rj / reach, 1.0 / (self.inv_m[i] + self.inv_m[j]),
                           self.v[i] - self.v[j], ri[:, None] * self.w[i] + rj[:, None] * self.w[j], s, self.w[i] - self.w[j])
        self.spring.keep(i, j, slot, s)
        force.index_add_(0, i, f)
        torque.index_add_(0, i, q)
        # sphere on wall; an edge or corner of several triangles acts once
        u, hit, close = self.closest(self.wi, self.wt)
        dist = u.norm(dim=1)
        k = close & (dist < self.r[self.wi])
        i, t, u, hit, dist = self.wi[k], self.wt[k], u[k], hit[k], dist[k]
        key = torch.where(hit >= 0, i * self.features + hit, self.n * self.features + torch.arange(i.numel(), device=DEV))
        order = torch.sort(key, stable=True).indices
        first = torch.ones_like(order, dtype=torch.bool)
        first[1:] = key[order][1:] != key[order][:-1]
        k = torch.sort(order[first]).values
        i, t, u, dist = i[k], t[k], u[k], dist[k]
        slot, s = self.wall.find(i, t)
        ri = self.r[i]
        f, q, s = self.law(i, u / dist[:, None], ri - dist, ri, self.m[i], self.v[i], ri[:, None] * self.w[i], s, self.w[i])
        self.wall.keep(i, t, slot, s)
        force.index_add_(0, i, f)
        torque.index_add_(0, i, q)
        self.v = self.v + (force * self.inv_m[:, None] + self.g) * self.dt
        self.x = self.x + self.v * self.dt
        if self.period is not None:
            span = self.period[1] - self.period[0]
            self.x[:, 0] -= torch.where(self.x[:, 0] >= self.period[1], span, 0.0)
            self.x[:, 0] += torch.where(self.x[:, 0] < self.period[0], span, 0.0)
        self.w = self.w + torque * self.inv_i[:, None] * self.dt


def exact(case, seed):
    s = _scene(case, seed)
    sim = _Exact(case, s)
    for _ in range(case["steps"]):
        sim.step()
    if s.mu_p is not None:  # the records that held them hold the materials now
        k = eta = None
    else:
        k, eta = sim.k, sim.eta
    out = {"x": sim.x.reshape(-1), "v": sim.v.reshape(-1), "angv": sim.w.reshape(-1),
           "isActive": torch.ones(s.n, dtype=torch.int32, device=DEV), "r": sim.r, "m": sim.m, "k": k, "etaconst": eta}
    if s.history is not None:
        for nm, h, wall in (("", sim.spring, ""), ("Wall", sim.wall, "Wall")):
            out["numCont" + nm] = h.rows.int()
            i = h.key // h.m
            out["indHis" + nm] = torch.full((s.n, s.stride), -1, dtype=torch.int32, device=DEV)
            out["indHis" + nm][i, h.slot] = (h.key % h.m).int()
            out["indHis" + nm] = out["indHis" + nm].reshape(-1)
            for a, c in enumerate("xyz"):
                d = torch.zeros((s.n, s.stride), dtype=F64, device=DEV)
                d[i, h.slot] = h.d[:, a]
                out["deltHis%s%s" % (c, wall)] = d.reshape(-1)
    return out
