"""The workloads whose speed this library is held to, through its public entry points.

Kinds (the key "kind" of a case):

  run       what the host driver does with one configuration: upload of the
            host state, pre-loop, a number of main-loop iterations (each with its
            step header, or without), download of the whole state.  Scenes: the
            reference's example lattice, dam breaks, periodic Taylor-Green
            vortices, and batches of dam breaks in one handle.
  adaptive  the same with a CFL time step computed and applied every iteration.
  serve     simulations submitted to the continuous-batching server, ticked
            until all are done, their results fetched.
  lists     export of the CSR neighbour lists of a computed state, plain or
            delta-coded.
  index     cell keys and stable key sort of positions already on the device.

Sizes are those of the library's own workloads and of its example configuration,
and odd ones between them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sph-simulations_gb300"))
import sphg  # noqa: E402
import workloads  # noqa: E402

FIELDS = ("x", "y", "vx", "vy", "rho", "fx", "fy")
PRECISION = {"plain": 0, "split": 1}


def listed():
    return [
        # a job of the size the serving workload's smallest requests have: launches and latency only
        dict(name="request_1k", kind="run", scene="dam", nx=33, ny=31, order="morton", precision="split",
             compute="sorted", vel=0.0, steps=100, headers=False),
        # the example configuration as it ships: 78 x 78 particles, row-major, a step header per iteration
        dict(name="example_6k", kind="run", scene="example", nx=78, ny=78, order="rowmajor", precision="plain",
             compute="sorted", vel=0.0, steps=49, headers=True),
        # the 12,800-particle dam break between two checkpoints
        dict(name="dam_12k", kind="run", scene="dam", nx=80, ny=160, order="morton", precision="plain",
             compute="sorted", vel=0.0, steps=100, headers=True),
        # a late dam-break state, the fluid moving: too many particles change cell to be merged, full sorts
        dict(name="dam_moving_423k", kind="run", scene="dam", nx=797, ny=531, order="morton", precision="split",
             compute="sorted", vel=3.0, steps=30, headers=True),
        # the periodic Taylor-Green vortex, 512 x 512
        dict(name="vortex_262k", kind="run", scene="vortex", nx=512, ny=512, order="morton", precision="plain",
             compute="sorted", vel=1.0, steps=50, headers=True),
        # the 1,000,000-particle dam break
        dict(name="dam_1m", kind="run", scene="dam", nx=1000, ny=1000, order="morton", precision="split",
             compute="sorted", vel=0.0, steps=40, headers=True),
        # 256 independent dam breaks of 2,000-65,536 particles in one handle
        dict(name="batch_256", kind="run", scene="batch", count=256, nmin=2000, nmax=65536, precision="split",
             compute="sorted", steps=20, headers=True),
        # the lists compute mode (compute_type=lists), row-major cells, odd size
        dict(name="lists_mode_93k", kind="run", scene="dam", nx=251, ny=373, order="rowmajor", precision="split",
             compute="lists", vel=0.0, steps=30, headers=True),
        # a time step from the CFL condition every iteration
        dict(name="adaptive_20k", kind="adaptive", scene="dam", nx=101, ny=203, order="morton", precision="split",
             compute="sorted", vel=1.0, steps=10),
        # a dozen served simulations of mixed sizes, dam breaks and vortices
        dict(name="serve_12", kind="serve", count=12, nmin=1000, nmax=60000, steps=50, precision="split"),
        # the neighbour lists of a state, delta-coded (the encoder's form)
        dict(name="lists_export_90k", kind="lists", scene="dam", nx=301, ny=299, order="morton", precision="plain",
             compute="sorted", vel=0.0, encoded=True),
        # cell keys and key sort of a million positions on the device
        dict(name="index_1m", kind="index", n=1000003, cells=1000, order="morton"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "batch", "adaptive", "serve", "lists", "index"])
    order = rng.choice(["morton", "morton", "rowmajor"])
    precision = rng.choice(["plain", "split"])
    if kind == "batch":
        return dict(kind="run", scene="batch", count=_log(rng, 3, 200), nmin=2000, nmax=65536, precision=precision,
                    compute="sorted", steps=rng.randint(5, 20), headers=rng.random() < 0.7)
    if kind == "serve":
        return dict(kind="serve", count=rng.randint(3, 12), nmin=1000, nmax=60000, steps=rng.randint(10, 50),
                    precision=precision)
    if kind == "index":
        return dict(kind="index", n=_log(rng, 1000, 2000000), cells=_log(rng, 20, 4000), order=order)
    n = _log(rng, 900, 900000 if kind == "run" else 200000)
    nx = max(20, int(round(math.sqrt(n * rng.uniform(0.5, 2.0)))))
    ny = max(20, n // nx)
    if kind == "lists":
        return dict(kind="lists", scene="dam", nx=nx, ny=ny, order=order, precision=precision, compute="sorted",
                    vel=rng.choice([0.0, 1.0]), encoded=rng.random() < 0.5)
    if kind == "adaptive":
        return dict(kind="adaptive", scene="dam", nx=nx, ny=ny, order=order, precision=precision, compute="sorted",
                    vel=rng.uniform(0.5, 2.0), steps=rng.randint(5, 15))
    scene = rng.choice(["dam", "dam", "vortex"])
    if scene == "vortex":
        nx = ny = max(20, int(round(math.sqrt(min(n, 300000)))))
    return dict(kind="run", scene=scene, nx=nx, ny=ny, order=order, precision=precision,
                compute=rng.choice(["sorted", "sorted", "sorted", "lists"]), vel=rng.choice([0.0, 0.0, 1.0, 3.0]),
                steps=rng.randint(20, 50), headers=rng.random() < 0.7)


# ---------------------------------------------------------------- inputs
def _scene(case, seed):
    """(list of parameter dicts, counts, x, y, vx, vy) of a case's initial state."""
    prms, counts, state = _initial(case, seed)
    if case["precision"] == "plain":
        # a single-precision state: the values the library holds are the values it is given
        state = [a.astype(np.float32).astype(np.float64) for a in state]
    return (prms, counts, *state)


def _initial(case, seed):
    scene = case["scene"]
    if scene == "batch":
        # the boxes are the case's, the jitter of the particles in them the seed's
        shapes, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed)
        prms, xs, ys = [], [], []
        for _ in range(case["count"]):
            n = int(round(math.exp(shapes.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
            aspect, alpha = shapes.uniform(0.3, 2.0), shapes.uniform(0.05, 0.2)
            p, x, y = workloads.dam_break_sized(n, aspect, 0.005, rng, alpha)
            prms.append(p)
            xs.append(x)
            ys.append(y)
        counts = np.array([len(x) for x in xs], np.int64)
        z = np.zeros(int(counts.sum()))
        return prms, counts, (np.concatenate(xs), np.concatenate(ys), z, z.copy())
    nx, ny, order = case["nx"], case["ny"], case["order"]
    if scene == "vortex":
        p, x, y, vx, vy, _ = workloads.taylor_green(nx, seed=seed, order=order)
        return [p], np.array([len(x)], np.int64), (x, y, vx, vy)
    if scene == "example":
        # config/example.txt: spacing 0.5, H = 1, rest density 25, walls 96 x 48; a small jitter from the seed
        rng = np.random.default_rng(seed)
        gx, gy = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
        x = 0.5 * (gx.ravel() + 1.0) + rng.uniform(-0.005, 0.005, nx * ny)
        y = 0.5 * (gy.ravel() + 1.0) + rng.uniform(-0.005, 0.005, nx * ny)
        p = dict(order=order, h=1.0, dt=0.005, k=30.0, rho0=25.0, mu=0.01, gx=0.0, gy=-10.0, mass=1.0, alpha=0.0,
                 c0=math.sqrt(30.0), lo=(0.0, 0.0), hi=(96.0, 48.0), periodic=0)
        z = np.zeros(x.size)
        return [p], np.array([x.size], np.int64), (x, y, z, z.copy())
    # a dam break in a box of 2.5 x its width and 1.25 x its height; vel: a swirl of that speed in the column
    dx = 0.4 / nx
    p, x, y, vx, vy = workloads.dam_break(nx, ny, dx, seed=seed, order=order, box=(2.5 * nx * dx, 1.25 * ny * dx))
    if case["vel"]:
        u, v = np.pi * x / (nx * dx), np.pi * y / (ny * dx)
        vx = case["vel"] * np.sin(u) * np.cos(v)
        vy = -case["vel"] * np.cos(u) * np.sin(v)
    return [p], np.array([len(x)], np.int64), (x, y, vx, vy)


def _requests(case, seed):
    """The served simulations: (parameters, x, y, vx, vy) each, dam breaks and vortices in turn."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["count"]):
        # sizes spread over the whole range, each with a little of the seed
        f = (k + 0.5) / case["count"]
        n = int(math.exp(math.log(case["nmin"]) * (1 - f) + math.log(case["nmax"]) * f))
        if k % 2 == 0:
            p, x, y = workloads.dam_break_sized(n, 0.8 + 0.1 * (k % 5), 0.005, rng, alpha=0.1)
            vx, vy = np.zeros(len(x)), np.zeros(len(x))
        else:
            p, x, y, vx, vy, _ = workloads.taylor_green(int(math.sqrt(n)), seed=int(rng.integers(1 << 30)))
        out.append((p, x, y, vx, vy))
    return out


def _sim(case, prms, counts):
    opts = sphg.options(precision=PRECISION[case["precision"]], compute=case["compute"])
    if case["scene"] == "batch":
        return sphg.Sim([sphg.params(**p) for p in prms], counts, opts)
    return sphg.Sim(sphg.params(**prms[0]), int(counts[0]), opts)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "index":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        xy = torch.rand(2, n, generator=g, device="cuda", dtype=torch.float32)
        cells = case["cells"]
        prm = sphg.params(order=case["order"], h=1.0 / cells, lo=(0.0, 0.0), hi=(1.0, 1.0))
        side = cells if case["order"] == "rowmajor" else 1 << (cells - 1).bit_length()
        return dict(case=case, prm=prm, x=xy[0], y=xy[1], bits=max(1, (side * side - 1).bit_length()),
                    keys=torch.empty(n, dtype=torch.int32, device="cuda"),
                    sorted=torch.empty(n, dtype=torch.int32, device="cuda"),
                    slots=torch.empty(n, dtype=torch.int32, device="cuda"))
    if kind == "serve":
        reqs = [(sphg.params(**p), x, y, vx, vy) for p, x, y, vx, vy in _requests(case, seed)]
        server = sphg.Server(1.0e9, max_instances=64, opts=sphg.options(precision=PRECISION[case["precision"]]))
        return dict(case=case, server=server, reqs=reqs)
    prms, counts, x, y, vx, vy = _scene(case, seed)
    sim = _sim(case, prms, counts)
    state = dict(case=case, sim=sim, x=x, y=y, vx=vx, vy=vy, dt0=prms[0]["dt"])
    if kind == "lists":
        sim.upload(x, y, vx, vy)
        sim.preloop()
        return state
    # the buffers a program keeps for its results; headers arrive in pinned memory
    n = len(x)
    out = {k: np.zeros(n, np.float64) for k in FIELDS}
    out["ids"] = np.zeros(n, np.int32)
    state["out"] = out
    if case.get("headers"):
        state["headers"] = torch.zeros(case["steps"], len(prms), 6, dtype=torch.float64, pin_memory=True)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "index":
        stream = torch.cuda.current_stream()
        n = case["n"]
        sphg.cell_keys(state["prm"], state["x"].data_ptr(), state["y"].data_ptr(), n, state["keys"].data_ptr(),
                       stream=stream)
        sphg.sort_pairs(state["keys"].data_ptr(), None, state["sorted"].data_ptr(), state["slots"].data_ptr(), n,
                        state["bits"], stream=stream)
        return dict(keys=state["keys"], sorted=state["sorted"], slots=state["slots"])
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(*r, case["steps"]) for r in state["reqs"]]
        live = 1
        while live:
            live, _ = server.tick()
        out = []
        for i in ids:
            r = server.result(i)
            out.append({k: r[k] for k in ("x", "y", "vx", "vy", "rho")})
        return out
    sim = state["sim"]
    if kind == "lists":
        offs, idx = sim.neighbor_lists_encoded() if case["encoded"] else sim.neighbor_lists()
        return dict(offs=offs, idx=idx)
    if kind == "adaptive":
        sim.set_dt(state["dt0"])
        sim.upload(state["x"], state["y"], state["vx"], state["vy"])
        sim.preloop()
        dts = []
        for _ in range(case["steps"]):
            dt = float(sim.cfl_dt(0.05, 0.05).min())
            sim.set_dt(dt)
            sim.step(1)
            dts.append(dt)
        return dict(sim.download(out=state["out"]), dts=np.array(dts))
    sim.upload(state["x"], state["y"], state["vx"], state["vy"])
    sim.preloop()
    if case["headers"]:
        sim.step_headers(case["steps"], out=state["headers"].data_ptr())
        return dict(sim.download(out=state["out"]), headers=state["headers"])
    sim.step(case["steps"])
    return sim.download(out=state["out"])


# ---------------------------------------------------------------- work
def work(case):
    """A particle-step: its state (x, y, vx, vy) read and written twice (sort, then
    integration), key, slot and density -- 80 bytes; about 15 candidate distances
    and 5 interacting pairs.  A run also reads the host state (32 bytes a
    particle) and writes the result (60)."""
    kind = case["kind"]
    if kind == "index":
        return dict(bytes=case["n"] * (8 + 4 + 8), flops=case["n"] * 6)
    if kind == "serve":
        n = sum(int(math.exp(math.log(case["nmin"]) * (1 - f) + math.log(case["nmax"]) * f))
                for f in ((k + 0.5) / case["count"] for k in range(case["count"])))
        return dict(bytes=n * (80 * case["steps"] + 32 + 44), flops=n * 350 * case["steps"])
    if kind == "lists":
        n = case["nx"] * case["ny"]
        return dict(bytes=n * (12 + 8 + 5 * 4), flops=n * 75)
    if case["scene"] == "batch":
        n = int(case["count"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"]))
    else:
        n = case["nx"] * case["ny"]
    return dict(bytes=n * (80 * (case["steps"] + 1) + 32 + 60), flops=n * 350 * (case["steps"] + 1))


# ---------------------------------------------------------------- 64-bit values
def _dilate(v):
    v = v & 0xFFFF
    for s, m in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << s)) & m
    return v


class _Exact:
    """The step in 64 bits on plain torch tensors: several instances at once, the
    constants of each looked up by the particle's instance."""

    def __init__(self, prms, counts, x, y, vx, vy):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(np.asarray(a), device=dev)  # noqa: E731
        self.inst = torch.repeat_interleave(torch.arange(len(prms), device=dev), t(counts))
        self.ninst = len(prms)
        self.x, self.y, self.vx, self.vy = (t(a).double().clone() for a in (x, y, vx, vy))
        starts = np.repeat(np.concatenate([[0], np.cumsum(counts)[:-1]]), counts)
        self.ids = torch.arange(len(x), device=dev) if len(prms) == 1 else t(np.arange(len(x)) - starts)
        self.order = prms[0]["order"]
        self.periodic = bool(prms[0]["periodic"])
        c = {}
        for k in ("h", "dt", "k", "rho0", "mu", "gx", "gy", "mass", "alpha", "c0"):
            c[k] = t([float(p[k]) for p in prms])
        for a in (0, 1):
            lo, hi = np.array([p["lo"][a] for p in prms], float), np.array([p["hi"][a] for p in prms], float)
            h = np.array([p["h"] for p in prms], float)
            n = np.floor((hi - lo) / h) if self.periodic else np.ceil((hi - lo) / h)
            c["lo%d" % a], c["hi%d" % a] = t(lo), t(hi)
            c["cs%d" % a] = t((hi - lo) / n if self.periodic else h)
            c["n%d" % a] = t(n.astype(np.int64))
        self.c = c
        side = 1 << max(int(max(c["n0"].max(), c["n1"].max())) - 1, 1).bit_length()
        self.span = side * side
        self.dt = c["dt"]
        self.headers = []

    def _key(self, cx, cy, inst):
        code = (_dilate(cy) << 1) | _dilate(cx) if self.order == "morton" else cx + cy * self.c["n0"][inst]
        return code + inst * self.span

    def _cells(self):
        i, c = self.inst, self.c
        cx = torch.floor((self.x - c["lo0"][i]) / c["cs0"][i]).long().clamp_min(0).minimum(c["n0"][i] - 1)
        cy = torch.floor((self.y - c["lo1"][i]) / c["cs1"][i]).long().clamp_min(0).minimum(c["n1"][i] - 1)
        return cx, cy

    def sort(self):
        cx, cy = self._cells()
        key = self._key(cx, cy, self.inst)
        key, perm = torch.sort(key, stable=True)
        for f in ("x", "y", "vx", "vy", "ids", "inst"):
            setattr(self, f, getattr(self, f)[perm])
        self.key, self.cx, self.cy = key, cx[perm], cy[perm]

    def _pairs(self):
        """The pairs (i, j, dx, dy, r2) within h, the particle itself included, one stencil cell at a time."""
        c = self.c
        for k in range(9):
            jx, jy = self.cx + k // 3 - 1, self.cy + k % 3 - 1
            nx, ny = c["n0"][self.inst], c["n1"][self.inst]
            if self.periodic:
                jx, jy = jx % nx, jy % ny
                ok = torch.ones_like(jx, dtype=torch.bool)
            else:
                ok = (jx >= 0) & (jx < nx) & (jy >= 0) & (jy < ny)
            key = self._key(jx.clamp_min(0), jy.clamp_min(0), self.inst)
            s = torch.searchsorted(self.key, key)
            m = torch.where(ok, torch.searchsorted(self.key, key, right=True) - s, 0)
            i = torch.repeat_interleave(torch.arange(len(key), device=key.device), m)
            j = s[i] + torch.arange(len(i), device=key.device) - (torch.cumsum(m, 0) - m)[i]
            dx, dy = self.x[i] - self.x[j], self.y[i] - self.y[j]
            if self.periodic:
                Lx, Ly = (c["hi0"] - c["lo0"])[self.inst[i]], (c["hi1"] - c["lo1"])[self.inst[i]]
                dx, dy = dx - Lx * torch.round(dx / Lx), dy - Ly * torch.round(dy / Ly)
            r2 = dx * dx + dy * dy
            near = r2 <= (c["h"] ** 2)[self.inst[i]]
            yield i[near], j[near], dx[near], dy[near], r2[near]

    def forces(self):
        c, ii = self.c, self.inst
        S = torch.zeros_like(self.x)
        for i, _, _, _, r2 in self._pairs():
            S.index_add_(0, i, (1.0 - r2 / (c["h"] ** 2)[ii[i]]) ** 3)
        h6 = c["h"] ** 6
        self.rho = (c["mass"] * 315.0 / (64.0 * math.pi * c["h"] ** 3))[ii] * S
        P = c["k"][ii] * (self.rho - c["rho0"][ii]) / self.rho ** 2
        kp = (c["mass"] * 1.5 * 15.0 / (math.pi * h6))
        kv = (c["mass"] * 45.0 * c["mu"] / (math.pi * h6))
        self.fx, self.fy = c["gx"][ii].clone(), c["gy"][ii].clone()
        for i, j, dx, dy, r2 in self._pairs():
            other = i != j
            i, j, dx, dy, r2 = i[other], j[other], dx[other], dy[other], r2[other]
            q = ii[i]
            r = torch.sqrt(r2)
            hr = c["h"][q] - r
            dvx, dvy = self.vx[j] - self.vx[i], self.vy[j] - self.vy[i]
            s = kp[q] * (P[i] + P[j])
            # artificial viscosity of approaching pairs: -2 alpha c0 h (v.r) / ((r^2 + 0.01 h^2) (rho_i + rho_j))
            vr = -(dvx * dx + dvy * dy)
            pij = -2.0 * (c["alpha"] * c["c0"] * c["h"])[q] * vr / ((r2 + 0.01 * c["h"][q] ** 2) * (self.rho[i] + self.rho[j]))
            s = s + torch.where(vr < 0, 2.0 * kp[q] * pij, 0.0)
            s = s * hr * hr / r
            vis = kv[q] / self.rho[j] * hr
            self.fx.index_add_(0, i, s * dx + vis * dvx)
            self.fy.index_add_(0, i, s * dy + vis * dvy)

    def integrate(self):
        c, ii = self.c, self.inst
        dt = self.dt[ii]
        for f, v, p, a in ((self.fx, "vx", "x", 0), (self.fy, "vy", "y", 1)):
            vel = getattr(self, v) + dt * f
            pos = getattr(self, p) + dt * vel
            lo, hi = c["lo%d" % a][ii], c["hi%d" % a][ii]
            if self.periodic:
                pos = torch.where(pos >= hi, pos - (hi - lo), pos)
                pos = torch.where(pos < lo, pos + (hi - lo), pos)
            else:
                out = (pos > hi) | (pos < lo)
                pos, vel = pos.minimum(hi).maximum(lo), torch.where(out, -vel, vel)
            setattr(self, v, vel)
            setattr(self, p, pos)

    def header(self):
        c, ii = self.c, self.inst
        h = torch.zeros(self.ninst, 6, dtype=torch.float64, device=self.x.device)
        v2 = self.vx ** 2 + self.vy ** 2
        h[:, 0].index_add_(0, ii, 0.5 * c["mass"][ii] * v2)
        h[:, 1] = torch.zeros_like(h[:, 1]).scatter_reduce(0, ii, v2, "amax")
        inside = (self.x >= c["lo0"][ii]) & (self.x <= c["hi0"][ii]) & (self.y >= c["lo1"][ii]) & (self.y <= c["hi1"][ii])
        h[:, 2].index_add_(0, ii, inside.double())
        h[:, 3].index_add_(0, ii, c["mass"][ii] * self.vx)
        h[:, 4].index_add_(0, ii, c["mass"][ii] * self.vy)
        self.headers.append(h)

    def begin(self):
        self.sort()
        self.forces()

    def step(self):
        self.integrate()
        self.sort()
        self.forces()

    def out(self, fields):
        return {k: getattr(self, k) for k in fields}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("index", "lists"):
        return None  # whole numbers only
    # The particles come out in slot order (sorted by cell).  Single-precision
    # positions round across a cell's edge an iteration earlier or later than
    # 64-bit ones, which moves particles to other slots: such a state has no 64-bit
    # value slot by slot, its headers and time steps do.
    slots = case["precision"] == "split"
    if not slots and (kind == "serve" or (kind == "run" and not case["headers"])):
        return None
    if kind == "serve":
        out = []
        for p, x, y, vx, vy in _requests(case, seed):
            e = _Exact([p], [len(x)], x, y, vx, vy)
            e.begin()
            for _ in range(case["steps"] - 1):
                e.step()
            out.append(e.out(("x", "y", "vx", "vy", "rho")))
        return out
    prms, counts, x, y, vx, vy = _scene(case, seed)
    e = _Exact(prms, counts, x, y, vx, vy)
    e.begin()
    if kind == "adaptive":
        dts, nxt = [], e.dt
        for _ in range(case["steps"]):
            # a time step applies from the next iteration's update on
            vmax = float(torch.sqrt((e.vx ** 2 + e.vy ** 2).max()))
            amax = float(torch.sqrt((e.fx ** 2 + e.fy ** 2).max()))
            h, c0 = prms[0]["h"], prms[0]["c0"]
            dt = min(0.05 * h / (c0 + vmax), 0.05 * math.sqrt(h / amax))
            dts.append(dt)
            e.dt = nxt
            e.step()
            nxt = torch.full_like(e.dt, dt)
        return dict(e.out(FIELDS) if slots else dict.fromkeys(FIELDS), ids=None, dts=np.array(dts))
    for _ in range(case["steps"]):
        e.step()
        if case["headers"]:
            e.header()
    out = dict(e.out(FIELDS) if slots else dict.fromkeys(FIELDS), ids=None)
    if case["headers"]:
        out["headers"] = torch.stack(e.headers)
    return out
