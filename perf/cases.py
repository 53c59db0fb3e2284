"""The work a user of the framework gives it, as cases that can be timed and compared.

Every case is a shallow-water run on a rectangular-cross mesh whose interior
nodes are moved off the lattice, with a sloping bed under Gaussian bumps, waves
and currents on the water and about a third of the land dry:

* plain FP64 through ``Domain``: ``evolve`` with yieldsteps, ``advance_steps``,
  and the host-driven step a boundary given as a Python function needs;
* the mixed-precision form through ``Batch`` and its ``Pool``: single domains
  and many scenarios together, their results as the single-precision output
  frames (node and cell values of stage, xmomentum, ymomentum) that a run
  stores.

``exact`` restates the flow algorithm in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

CELL = 10.0                 # side of a mesh square, metres
RAIN = 50.0e-3 / 3600.0     # 50 mm/h
HMIN_FRAME = 1.0e-5         # minimum storable height of the frames, metres
G, EPS = 9.8, 1.0e-12

# CFL, stages, minimum depth, beta (the limiter's, on stage and momenta alike; 0 where dry)
ALGORITHMS = {"DE0": (0.9, 1, 1.0e-12, 0.5), "DE1": (1.0, 2, 1.0e-5, 1.0), "DE2": (1.0, 3, 1.0e-5, 1.0)}


def _case(name, form, call, algorithm, scene, nx, ny, steps, count=1):
    return {"name": name, "form": form, "call": call, "algorithm": algorithm, "scene": scene, "nx": nx, "ny": ny,
            "steps": steps, "count": count}


def listed():
    return [
        # a tutorial-sized dam break: a few hundred triangles, the step's launches are what it waits for
        _case("plain-dam-tiny", "plain", "evolve", "DE0", "dam", 11, 9, 20),
        # the dam break of the parity tests: 40,000 triangles, one yieldstep of about 40 steps
        _case("plain-dam-40k", "plain", "evolve", "DE0", "dam", 100, 100, 40),
        # a tide gauge given as a Python function: the host drives the phases of every step
        _case("plain-tide-python", "plain", "evolve", "DE1", "tide", 61, 47, 8),
        # a town-sized model in the second-order scheme, between two outputs
        _case("plain-inflow-250k", "plain", "steps", "DE1", "inflow", 251, 249, 10),
        # the third-order scheme on an odd size
        _case("plain-rk3-400k", "plain", "steps", "DE2", "inflow", 333, 301, 4),
        # the benchmark's mesh: 4.0M triangles, FP64
        _case("plain-inflow-4m", "plain", "steps", "DE1", "inflow", 1000, 1000, 2),
        # a small mixed-precision run between two frames
        _case("mixed-small", "mixed", "steps", "DE1", "inflow", 25, 27, 50),
        # rain over a quarter of a catchment, mixed precision, between two frames
        _case("mixed-rain-300k", "mixed", "steps", "DE1", "rain", 271, 277, 80),
        # the benchmark's mesh: 4.0M triangles, mixed precision
        _case("mixed-inflow-4m", "mixed", "steps", "DE1", "inflow", 1000, 1000, 60),
        # a model coupled to a host program: new state in, one step, a frame out
        _case("mixed-coupled-1m", "mixed", "coupled", "DE1", "inflow", 501, 497, 1),
        # an ensemble: many scenarios of very different sizes in one pool
        _case("batch-ensemble", "mixed", "steps", "DE1", "mix", 20, 200, 20, 48),
        # the serving loop's chunk: running scenarios, 64 more steps, their statistics and frames
        _case("serve-chunk", "mixed", "chunk", "DE1", "mix", 50, 180, 64, 12),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(("evolve", "steps", "mixed", "coupled", "ensemble", "chunk"))
    if family == "evolve":
        scene = rng.choice(("dam", "inflow", "tide"))
        top = 80 if scene == "tide" else 220
        return _case("", "plain", "evolve", rng.choice(("DE0", "DE1")), scene, log_int(5, top), log_int(5, top),
                     rng.randint(4, 8) if scene == "tide" else rng.randint(10, 40))
    if family == "steps":
        nx, ny = log_int(20, 960), log_int(20, 960)
        return _case("", "plain", "steps", rng.choice(("DE0", "DE1", "DE2")), rng.choice(("dam", "inflow")), nx, ny,
                     max(1, min(20, 2000000 // (nx * ny))))
    if family == "mixed":
        nx, ny = log_int(8, 960), log_int(8, 960)
        return _case("", "mixed", "steps", rng.choice(("DE0", "DE1", "DE2")), rng.choice(("dam", "inflow", "rain")),
                     nx, ny, max(20, min(120, 55000000 // (nx * ny))))
    if family == "coupled":
        return _case("", "mixed", "coupled", "DE1", rng.choice(("dam", "inflow")), log_int(20, 700), log_int(20, 700),
                     rng.randint(1, 4))
    if family == "ensemble":
        return _case("", "mixed", "steps", "DE1", "mix", rng.randint(12, 40), rng.randint(60, 210),
                     rng.randint(8, 24), rng.randint(8, 60))
    return _case("", "mixed", "chunk", "DE1", "mix", rng.randint(20, 60), rng.randint(80, 200), 64, rng.randint(3, 14))


# ---------------------------------------------------------------------------
# meshes and fields


def _runs(case):
    """(nx, ny, scene) of every scenario of a case: one, or `count` of them
    with sides log-uniform between nx and ny, dam breaks and inflows in turn."""
    if case["count"] == 1:
        return [(case["nx"], case["ny"], case["scene"])]
    r = np.random.default_rng([case["nx"], case["ny"], case["count"]])
    s = np.round(np.exp(r.uniform(math.log(case["nx"]), math.log(case["ny"]), case["count"]))).astype(int)
    return [(int(m), int(m), "dam" if i % 2 == 0 else "inflow") for i, m in enumerate(s)]


def _cells(case):
    return sum(4 * nx * ny for nx, ny, _ in _runs(case))


def _triangles(nx, ny):
    """Nodes, triangles and the side (0 west, 1 south, 2 east, 3 north, -1
    none) each triangle's edge 1 lies on: nx x ny squares cut by their
    diagonals, the nodes inside moved by up to 0.12 of a square."""
    vid = np.arange((nx + 1) * (ny + 1)).reshape(nx + 1, ny + 1)
    xi, yi = np.meshgrid(np.arange(nx + 1.0), np.arange(ny + 1.0), indexing="ij")
    xc, yc = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny) + 0.5, indexing="ij")
    P = np.concatenate([np.stack([xi.ravel(), yi.ravel()], 1), np.stack([xc.ravel(), yc.ravel()], 1)])
    r = np.random.default_rng([nx, ny])
    move = r.uniform(-0.12, 0.12, P.shape)
    inside = (P[:, 0] > 0) & (P[:, 0] < nx) & (P[:, 1] > 0) & (P[:, 1] < ny)
    P = (P + np.where(inside[:, None], move, 0.0)) * CELL
    a, b = vid[:-1, :-1].ravel(), vid[1:, :-1].ravel()
    c, d = vid[1:, 1:].ravel(), vid[:-1, 1:].ravel()
    m = (nx + 1) * (ny + 1) + np.arange(nx * ny)
    T = np.empty((4 * nx * ny, 3), np.int64)
    T[0::4] = np.stack([a, m, d], 1)
    T[1::4] = np.stack([b, m, a], 1)
    T[2::4] = np.stack([c, m, b], 1)
    T[3::4] = np.stack([d, m, c], 1)
    side = np.full(4 * nx * ny, -1)
    i, j = np.divmod(np.arange(nx * ny), ny)
    side[0::4] = np.where(i == 0, 0, -1)
    side[1::4] = np.where(j == 0, 1, -1)
    side[2::4] = np.where(i == nx - 1, 2, -1)
    side[3::4] = np.where(j == ny - 1, 3, -1)
    return P, T, side


def _fields(P, T, scene, seed):
    """Vertex bed [N, 3] and centroid stage, momenta and friction [N]."""
    r = np.random.default_rng([seed, len(T)])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    xy = torch.from_numpy(P).to(dev)
    x, y = xy[:, 0], xy[:, 1]
    Lx, Ly = float(P[:, 0].max()), float(P[:, 1].max())
    z = (-7.0 + 10.0 * x / Lx) if scene != "dam" else -2.0 * x / Lx
    for _ in range(10):
        s = r.uniform(0.03, 0.12) * max(Lx, Ly)
        z = z + (r.uniform(-2.0, 2.0) if scene != "dam" else r.uniform(-0.4, 0.4)) * torch.exp(
            -((x - r.uniform(0, Lx)) ** 2 + (y - r.uniform(0, Ly)) ** 2) / (2.0 * s * s))
    t = torch.from_numpy(T).to(dev)
    zv = z[t]
    zc = (zv[:, 0] + zv[:, 1] + zv[:, 2]) / 3.0
    cx, cy = x[t].mean(1) / Lx, y[t].mean(1) / Ly
    k = [r.uniform(2.0, 6.0) for _ in range(4)]
    ph = [r.uniform(0.0, 6.28) for _ in range(4)]
    if scene == "dam":
        w = zc + torch.where(cx < 0.5, 1.0, 0.1) + 0.02 * torch.sin(6.28 * k[0] * cy + ph[0])
    else:
        w = torch.maximum(zc, 0.15 * torch.sin(6.28 * k[0] * cx + ph[0]) * torch.cos(6.28 * k[1] * cy + ph[1]))
    h = w - zc
    uh = h * (0.4 * torch.sin(6.28 * k[2] * cy + ph[2]) + 0.1)
    vh = h * 0.4 * torch.cos(6.28 * k[3] * cx + ph[3])
    eta = r.uniform(0.02, 0.06, len(T))
    return [q.cpu().numpy() for q in (zv, w, uh, vh)] + [eta]


def _rain_cells(P, T):
    c = P[T].mean(1) / P.max(0)
    return np.nonzero((np.abs(c - 0.5) < 0.25).all(1))[0]


def _tide(t):
    return (0.4 + 0.5 * math.sin(0.05 * t), 0.0, 0.0)


def _walls(scene):
    """Boundary kinds of the west, south, east and north sides."""
    if scene == "dam":
        return ("wall", "wall", "wall", "wall")
    return ("tide" if scene == "tide" else "stage", "wall", "open", "wall")


STAGE = (0.6, 0.0, 0.0)     # what a "stage" side is held at


def _yieldstep(case):
    """Simulated seconds of about `steps` timesteps (depths of about 8 m, or of 1 m behind the dam)."""
    c = 3.6 if case["scene"] == "dam" else 9.0
    return case["steps"] * 0.09 * CELL / c


# ---------------------------------------------------------------------------
# the framework's side

_MESHES = {}


def _mesh(nx, ny, form):
    """A program's meshes and their packed tables are made once and shared by its runs."""
    from anuga_core_gb300 import Mesh
    from anuga_core_gb300.tables import pack_mixed
    key = (nx, ny)
    if key not in _MESHES:
        while len(_MESHES) > 64:
            _MESHES.pop(next(iter(_MESHES)))
        P, T, side = _triangles(nx, ny)
        names = ("west", "south", "east", "north")
        B = {(int(k), 1): names[side[k]] for k in np.nonzero(side >= 0)[0]}
        _MESHES[key] = [Mesh(P, T, B), None]
    entry = _MESHES[key]
    if form == "mixed" and entry[1] is None:
        entry[1] = pack_mixed(entry[0])
    return entry


def _domain(mesh, case, scene, seed):
    import anuga_core_gb300 as anuga
    zv, w, uh, vh, eta = _fields(mesh.nodes, mesh.triangles, scene, seed)
    d = anuga.Domain(mesh=mesh)
    d.set_flow_algorithm(case["algorithm"])
    d.set_gpu_options(precision="fp64" if case["form"] == "plain" else "mixed")
    d.set_store(False)
    d.set_quantity("elevation", zv)
    for q, v in (("stage", w), ("xmomentum", uh), ("ymomentum", vh), ("friction", eta)):
        d.set_quantity(q, v, location="centroids")
    kinds = {"wall": lambda: anuga.Reflective_boundary(d), "open": lambda: anuga.Transmissive_boundary(d),
             "stage": lambda: anuga.Dirichlet_boundary(list(STAGE)),
             "tide": lambda: anuga.Time_boundary(d, function=_tide)}
    d.set_boundary({t: kinds[k]() for t, k in zip(("west", "south", "east", "north"), _walls(scene))})
    if scene == "rain":
        anuga.Rate_operator(d, rate=RAIN, indices=_rain_cells(mesh.nodes, mesh.triangles))
    return d


def prepare(case, seed):
    runs = _runs(case)
    meshes = [_mesh(nx, ny, case["form"]) for nx, ny, _ in runs]
    doms = [_domain(m[0], case, scene, seed + 1000 * i) for i, (m, (_, _, scene)) in enumerate(zip(meshes, runs))]
    state = {"case": case}
    if case["form"] == "plain":
        d = state["domain"] = doms[0]
        if case["call"] == "steps":
            state["views"] = [d.device_tensor(q) for q in ("stage", "xmomentum", "ymomentum")]
        return state
    from anuga_core_gb300.batch import Batch
    batch = state["batch"] = Batch(doms, tables=[m[1] for m in meshes])
    state["nodes"] = []
    for sid, (m, _) in zip(batch.sids, meshes):
        flat = m.triangles.ravel()
        off = np.zeros(m.number_of_nodes + 1, np.int64)
        off[1:] = np.cumsum(np.bincount(flat, minlength=m.number_of_nodes))
        batch.pool.sww_bind(sid, off, np.argsort(flat, kind="stable"))
        state["nodes"].append(m.number_of_nodes)
        if case["call"] == "chunk":
            batch.pool.set_clock(sid, 0.0, 1.0e300, 1.0e9, 0)
    if case["call"] == "coupled":
        d = doms[0]
        pinned = [torch.empty(len(d), dtype=torch.float64, pin_memory=torch.cuda.is_available()) for _ in range(3)]
        for p, q in zip(pinned, ("stage", "xmomentum", "ymomentum")):
            p.numpy()[:] = d.quantities[q].centroid_values
        state["incoming"] = [p.numpy() for p in pinned]
        state["pinned"] = pinned
    if len(doms) > 1:
        batch.domains = doms
    return state


def _frames(state):
    pool, sids = state["batch"].pool, state["batch"].sids
    for sid in sids:
        pool.sww_frame_async(sid, HMIN_FRAME)
    got = [pool.sww_frame_wait(sid, n) for sid, n in zip(sids, state["nodes"])]
    if len(got) == 1:
        return [got[0][0], got[0][1]]
    return [np.concatenate([v for v, _ in got], 1), np.concatenate([c for _, c in got], 1)]


def run(state):
    case = state["case"]
    if case["form"] == "plain":
        d = state["domain"]
        if case["call"] == "evolve":
            ys = _yieldstep(case)
            for _ in d.evolve(yieldstep=ys, duration=ys):
                pass
            return [d.quantities[q].centroid_values for q in ("stage", "xmomentum", "ymomentum")] + [d.get_time()]
        st = d.advance_steps(case["steps"])
        return state["views"] + [st.time]
    batch = state["batch"]
    if case["call"] == "coupled":
        batch.pool.set_state(batch.sids[0], *state["incoming"])
    if case["call"] == "chunk":
        batch.pool.launch_chunk(case["steps"])
        batch.pool.wait()
        stats, _ = batch.pool.stats_all(batch.sids)
    else:
        stats = batch.advance_steps(case["steps"])
    times = np.array([s.time for s in stats], np.float32) if case["call"] != "coupled" else np.zeros(1, np.float32)
    return _frames(state) + [times]


def work(case):
    """Per step the state, the neighbours' states and the mesh tables are read
    and the new state is written, once a stage: 232 (one FP64 stage), 244 (each
    of several) or 176 (mixed) bytes a cell and stage; a frame reads the state
    and writes 24 + 12 bytes a cell."""
    n, stages = _cells(case), ALGORITHMS[case["algorithm"]][1]
    per = 176 if case["form"] == "mixed" else (232 if stages == 1 else 244)
    b = n * case["steps"] * stages * per
    if case["form"] == "mixed":
        b += n * 36
    if case["call"] == "coupled":
        b += n * 24
    return {"bytes": float(b), "flops": float(n * case["steps"] * stages * 330)}


# ---------------------------------------------------------------------------
# the same in 64 bits


class _Flow:
    """The discontinuous-elevation scheme on one mesh: torch, float64."""

    def __init__(self, P, T, side, scene, algorithm, zc, w, uh, vh, eta, rain):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
        self.cfl, self.stages, self.hmin, self.beta = ALGORITHMS[algorithm]
        self.kinds = [{"wall": 1, "open": 2, "stage": 3, "tide": 3}[k] for k in _walls(scene)]
        self.held = _tide if scene == "tide" else (lambda time: STAGE)
        N = len(T)
        T = t(T)
        V = t(P)[T]
        a, b = T[:, [1, 2, 0]].reshape(-1), T[:, [2, 0, 1]].reshape(-1)
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        order = torch.sort(lo * len(P) + hi, stable=True)
        key, pos = order.values, order.indices
        self.opp = torch.arange(3 * N, device=dev)
        two = torch.nonzero(key[1:] == key[:-1]).reshape(-1)
        self.opp[pos[two]] = pos[two + 1]
        self.opp[pos[two + 1]] = pos[two]
        self.inner = (self.opp != torch.arange(3 * N, device=dev)).reshape(N, 3)
        self.nb = (self.opp // 3).reshape(N, 3)
        self.side = torch.where(self.inner, -1, t(side)[:, None].expand(N, 3))
        nxt, aft = V[:, [1, 2, 0]], V[:, [2, 0, 1]]
        e = aft - nxt
        self.len = e.square().sum(2).sqrt()
        self.n1, self.n2 = e[..., 1] / self.len, -e[..., 0] / self.len
        self.area = 0.5 * (e[:, 2, 0] * -e[:, 1, 1] + e[:, 2, 1] * e[:, 1, 0]).abs()
        C = V.mean(1)
        self.d = 0.5 * (nxt + aft) - C[:, None]
        self.radius = self.d.square().sum(2).sqrt().amin(1)
        S = C[self.nb]
        p, q = S[:, 1] - S[:, 0], S[:, 2] - S[:, 0]
        self.p, self.q, self.det = p, q, q[:, 1] * p[:, 0] - p[:, 1] * q[:, 0]
        self.z, self.w, self.uh, self.vh, self.eta = (t(v).clone() for v in (zc, w, uh, vh, eta))
        self.rain = None if rain is None else t(rain)
        self.time = 0.0

    def protect(self):
        h = self.w - self.z
        self.w = torch.where(h < 0, self.z, self.w)
        dry = torch.clamp(self.w - self.z, min=0) <= self.hmin
        self.uh = torch.where(dry, 0.0, self.uh)
        self.vh = torch.where(dry, 0.0, self.vh)

    def surrounded(self, h):
        s = ((h[self.nb] < self.hmin) | ~self.inner).all(1)
        self.uh = torch.where(s, 0.0, self.uh)
        self.vh = torch.where(s, 0.0, self.vh)
        return s

    def limited(self, c, n, beta):
        d0, d1, d2 = n[:, 0] - c, n[:, 1] - n[:, 0], n[:, 2] - n[:, 0]
        gx = (self.q[:, 1] * d1 - self.p[:, 1] * d2) / self.det
        gy = (self.p[:, 0] * d2 - self.q[:, 0] * d1) / self.det
        J = gx[:, None] * self.d[..., 0] + gy[:, None] * self.d[..., 1]
        D = torch.stack([d0, d0 + d1, d0 + d2, torch.zeros_like(d0)], 1)
        hi, lo = D.amax(1), D.amin(1)
        r, cand = torch.full_like(c, 1000.0), torch.ones_like(c)
        for i in range(3):
            j = J[:, i]
            cand = torch.where(j < -1e-100, lo / j, cand)
            cand = torch.where(j > 1e-100, hi / j, cand)
            r = torch.minimum(cand, r)
        phi = torch.clamp(r * beta, max=1.0)
        return c[:, None] + J * phi[:, None]

    def edges(self):
        self.protect()
        h = torch.clamp(self.w - self.z, min=0)
        wet = h > self.hmin
        u, v = torch.where(wet, self.uh / h, 0.0), torch.where(wet, self.vh / h, 0.0)
        s = self.surrounded(h)
        own = lambda q, qs: torch.where(self.inner, q[self.nb], qs[:, None])  # noqa: E731
        us, vs = torch.where(s, 0.0, u), torch.where(s, 0.0, v)
        hn = own(h, h)
        hlo, hhi = torch.minimum(hn.amin(1), h), torch.maximum(hn.amax(1), h)
        c = 1.0 / (0.3 - 0.1)
        e = 1.0 - c * 0.3
        f = torch.clamp(c * h / torch.clamp(hhi, min=1e-6) + e, max=1.0)
        f = torch.clamp(torch.minimum(c * hlo / torch.clamp(h, min=1e-6) + e, f), min=0.0)
        f = torch.minimum(1.2 * torch.clamp(hlo - self.hmin, min=0) / (hlo + self.hmin), f)
        beta = self.beta * f
        we = self.limited(self.w, own(self.w, self.w), beta)
        he = self.limited(h, hn, beta)
        ue = self.limited(us, own(u, us), beta)
        ve = self.limited(vs, own(v, vs), beta)
        return h, we, he, ue * he, ve * he

    def slope(self, time):
        """Explicit updates and each cell's largest wave speed at the present state."""
        hc, we, he, ue, ve = self.edges()
        ze = we - he
        n1, n2 = self.n1, self.n2
        far = lambda q: q.reshape(-1)[self.opp].reshape(q.shape)  # noqa: E731
        wr, zr, hr, ur, vr = far(we), far(ze), far(he), far(ue), far(ve)
        qn, qt = ue * n1 + ve * n2, -ue * n2 + ve * n1
        for k, kind in enumerate(self.kinds):
            at = self.side == k
            if kind == 1:
                ur = torch.where(at, -n1 * qn - n2 * qt, ur)
                vr = torch.where(at, -n2 * qn + n1 * qt, vr)
            elif kind == 3:
                val = self.held(time)
                wr = torch.where(at, val[0], wr)
                ur = torch.where(at, val[1], ur)
                vr = torch.where(at, val[2], vr)
        hr = torch.where(self.inner, hr, torch.clamp(wr - ze, min=0))
        zh = torch.maximum(ze, zr)
        Hl, Hr = torch.clamp(he + ze - zh, min=0), torch.clamp(hr + zr - zh, min=0)
        il, ir = torch.where(he > 0, 1.0 / he, 0.0), torch.where(hr > 0, 1.0 / hr, 0.0)
        ul, vl = qn * il, qt * il
        unr, utr = (ur * n1 + vr * n2) * ir, (-ur * n2 + vr * n1) * ir
        cl, cr = (G * Hl).sqrt(), (G * Hr).sqrt()
        smax = torch.clamp(torch.maximum(ul + cl, unr + cr), min=0)
        smin = torch.clamp(torch.minimum(ul - cl, unr - cr), max=0)
        span = smax - smin
        live = ((Hl != 0) | (Hr != 0)) & (span >= EPS)
        inv = torch.where(live, 1.0 / span, 0.0)
        ss = smax * smin
        F0 = (smax * ul * Hl - smin * unr * Hr + ss * (torch.maximum(wr, zh) - torch.maximum(we, zh))) * inv
        F1 = (smax * ul * ul * Hl - smin * unr * unr * Hr + ss * (unr * Hr - ul * Hl)) * inv
        F2 = (smax * ul * vl * Hl - smin * unr * utr * Hr + ss * (utr * Hr - vl * Hl)) * inv
        pf = torch.where(live, 0.5 * G * (smax * Hl * Hl - smin * Hr * Hr) * inv,
                         torch.where((Hl != 0) | (Hr != 0), 0.25 * G * (Hl * Hl + Hr * Hr), 0.0))
        pg = -0.5 * G * (Hl * Hl - he * he - (he + hc[:, None]) * (ze - self.z[:, None])) + pf
        speed = torch.where(live, torch.maximum(smax, -smin), 0.0).amax(1)
        X = [(-(F0) * self.len).sum(1) / self.area,
             (-(n1 * F1 - n2 * F2 + n1 * pg) * self.len).sum(1) / self.area,
             (-(n2 * F1 + n1 * F2 + n2 * pg) * self.len).sum(1) / self.area]
        return X, speed

    def update(self, X, dt):
        h = self.w - self.z
        ok = (h >= self.hmin) & (self.eta > self.hmin)
        S = torch.where(ok, G * self.eta ** 2 * (self.uh ** 2 + self.vh ** 2).sqrt()
                        / torch.where(ok, h, 1.0) ** (7.0 / 3.0), 0.0)
        den = 1.0 + dt * S
        self.w = self.w + dt * X[0]
        self.uh = torch.where(self.uh != 0, (self.uh + dt * X[1]) / den, self.uh + dt * X[1])
        self.vh = torch.where(self.vh != 0, (self.vh + dt * X[2]) / den, self.vh + dt * X[2])
        neg = self.w - self.z < 0
        self.w = torch.where(neg, self.z, self.w)
        self.uh = torch.where(neg, 0.0, self.uh)
        self.vh = torch.where(neg, 0.0, self.vh)

    def step(self, stop=math.inf):
        old = [self.w, self.uh, self.vh]

        def mix(a, b, over=1.0):
            self.w, self.uh, self.vh = ((a * q + b * o) / over for q, o in zip((self.w, self.uh, self.vh), old))

        X, speed = self.slope(self.time)
        dt = min(self.cfl * float((self.radius / speed).min()), 1000.0)
        dt = min(dt, stop - self.time)
        self.update(X, dt)
        if self.stages > 1:
            self.update(self.slope(self.time + dt)[0], dt)
            if self.stages == 2:
                mix(0.5, 0.5)
            else:
                mix(0.25, 0.75)
                self.update(self.slope(self.time + 0.5 * dt)[0], dt)
                mix(2.0, 1.0, 3.0)
        if self.rain is not None:
            self.w[self.rain] += dt * RAIN
        self.time += dt

    def settle(self):
        """What a yield does to the state: dry and surrounded-dry cells lose their momenta."""
        self.protect()
        self.surrounded(torch.clamp(self.w - self.z, min=0))


def exact(case, seed):
    nodes, cells, times = [], [], []
    for i, (nx, ny, scene) in enumerate(_runs(case)):
        P, T, side = _triangles(nx, ny)
        zv, w, uh, vh, eta = _fields(P, T, scene, seed + 1000 * i)
        zc = (zv[:, 0] + zv[:, 1] + zv[:, 2]) / 3.0
        F = _Flow(P, T, side, scene, case["algorithm"], zc, w, uh, vh, eta,
                  _rain_cells(P, T) if scene == "rain" else None)
        if case["call"] == "evolve":
            stop = _yieldstep(case)
            F.settle()
            while F.time < stop - EPS:
                F.step(stop)
            F.settle()
        else:
            for _ in range(case["steps"]):
                F.step()
        if case["form"] == "plain":
            return [F.w, F.uh, F.vh, float(F.time)]
        flat = torch.as_tensor(T.ravel(), device=F.w.device)
        count = torch.bincount(flat, minlength=len(P)).double()
        mean = lambda q: torch.zeros_like(count).index_add_(0, flat, q.repeat_interleave(3)) / count  # noqa: E731
        aw, az, au, av = (mean(q) for q in (F.w, F.z, F.uh, F.vh))
        keep = aw - az >= HMIN_FRAME
        nodes.append(torch.stack([torch.where(keep, aw, az), torch.where(keep, au, 0.0), torch.where(keep, av, 0.0)]))
        cells.append(torch.stack([F.w, F.uh, F.vh]))
        times.append(F.time if case["call"] != "coupled" else 0.0)
    return [torch.cat(nodes, 1), torch.cat(cells, 1), torch.tensor(times, dtype=torch.float64)]
