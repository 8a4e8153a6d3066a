"""The workloads whose speed is measured, as a user's program runs them.

Every case is a simulation under way: ``prepare`` builds the solver from a
config (``LBMD3``), hands it the initial field and the bodies, and takes the
first step, which moves the state into the solver's own buffers; ``run`` takes
the next stretch of steps through ``LBMD3.run_step`` / ``run_steps`` and reads
what such a program reads -- velocity, density, particle state, step
statistics.  The served case hands a batch of requests to ``LBMServer``.
``exact`` is the same simulation in float64 with plain torch.
"""
import math
import os

os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")   # the server's stream pool

import numpy as np
import torch

FACES = ("input", "output", "back", "forward", "bottom", "top")
# boundary layouts: one letter per face (P periodic, W wall, S moving wall,
# N non-equilibrium inlet / outlet)
LAYOUTS = {"periodic": "PPPPPP", "closed": "WWWWWW", "channel": "WWWWPP", "lid": "WWWWWS",
           "duct": "NNWWWW", "slab": "PPWWPP", "tube": "PPWWWW", "couette": "PPPPSS"}
CODES = {"P": "PERIODICAL", "W": "WALL", "S": "WALL_WITH_SPEED", "N": "NON_EQUILIBRIUM"}
STORED = {"fp32": 4, "fp16s": 2, "bf16s": 2, "fp64": 8}


def _case(name, q, shape, storage, layout, mu, steps, how="run_steps", bodies="", force=0.0,
          flow=0.02, gl=0.0):
    return {"name": name, "kind": "solve", "q": q, "x": shape[0], "y": shape[1], "z": shape[2],
            "storage": storage, "layout": layout, "mu": mu, "steps": steps, "how": how,
            "bodies": bodies, "force": force, "flow": flow, "gl": gl}


def listed():
    return [
        # Poiseuille channel of the accuracy tests: the smallest lattice anyone
        # times; latency of the step and of reading the fields back
        _case("poiseuille_channel", 19, (33, 33, 65), "fp32", "channel", 0.1, 16, force=1e-6),
        # single-sphere free fall, stepped one run_step at a time as the
        # reference's own loop does: the particle kernels' latency
        _case("sphere_fall", 19, (161, 65, 65), "fp32", "closed", 0.0666667, 8, how="run_step",
              bodies="sphere:8:1.5:1", gl=2e-5, flow=1e-3),
        # multi-ellipsoid sedimentation: thousands of markers, rows of odd length
        _case("ellipsoids_q27", 27, (257, 129, 129), "fp32", "closed", 0.05, 8,
              bodies="ellipsoid:6:4:4:1.2:32", gl=1e-5, flow=1e-3),
        # the same coupling in 16-bit storage on a partly periodic lattice, as
        # served requests mix them
        _case("bodies_tube_fp16s", 19, (177, 113, 97), "fp16s", "tube", 0.05, 8,
              bodies="sphere:6:1.2:4", gl=1e-5, flow=1e-3),
        # the headline: periodic Taylor-Green vortex, 512 nodes per axis
        _case("sweep_512_q19_fp32", 19, (512, 512, 512), "fp32", "periodic", 0.0333333, 8,
              flow=0.05),
        # the same in half the bytes
        _case("sweep_512_q19_fp16s", 19, (512, 512, 512), "fp16s", "periodic", 0.0333333, 8,
              flow=0.05),
        # the sweep's other velocity sets and sizes, in both 16-bit forms
        _case("sweep_256_q27_fp16s", 27, (256, 256, 256), "fp16s", "periodic", 0.0333333, 8,
              flow=0.05),
        _case("sweep_256_q13_bf16s", 13, (256, 256, 256), "bf16s", "periodic", 0.0333333, 8,
              flow=0.05),
        # lid-driven cavity: moving wall, the reference's size + 1 = odd rows
        _case("lid_129_q15", 15, (129, 129, 129), "fp32", "lid", 0.05, 16),
        # duct with non-equilibrium inlet and outlet: the reference's call
        # sequence, one kernel per method
        _case("duct_129x49x49", 19, (129, 49, 49), "fp32", "duct", 0.1, 8),
        # every step logged, the reference's default cadence: step, then the
        # statistics of f, u and rho
        _case("logged_193x161x129", 19, (193, 161, 129), "fp32", "slab", 0.05, 4, how="logged"),
        # served stream: small mixed requests, continuous batching
        {"name": "served_8", "kind": "serve", "requests": 8, "low": 32, "high": 96, "steps": 96},
    ]


def draw(rng):
    """One more case of the same ranges; never dearer than the 512^3 ones."""
    kind = rng.choice(("sweep", "sweep", "bodies", "bodies", "walls", "duct", "logged", "serve"))
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(4, 8), "low": 32, "high": 96,
                "steps": rng.randint(48, 96)}
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    q = rng.choice((13, 15, 19, 27))
    storage = rng.choice(("fp32", "fp32", "fp16s", "bf16s"))
    how = rng.choice(("run_steps", "run_step"))
    steps = rng.randint(4, 12)
    if kind == "sweep":
        n = size(32, 320)
        shape = tuple(max(24, int(n * rng.uniform(0.8, 1.25))) for _ in range(3))
        if max(shape) < 160 and rng.random() < 0.25:
            storage = "fp64"
        c = _case("", q, shape, storage, "periodic", 0.0333333, steps, how=how, flow=0.05)
    elif kind == "bodies":
        shape = tuple(rng.randint(48, 192) for _ in range(3))
        r = rng.randint(4, 8)
        few = rng.randint(1, 8)
        body = rng.choice(("sphere:%d:1.2:%d" % (r, few),
                           "ellipsoid:%d:%d:%d:1.2:%d" % (r, max(2, r - 2), max(2, r - 2), few)))
        c = _case("", rng.choice((19, 27)), shape, storage,
                  rng.choice(("closed", "tube", "slab", "periodic")), 0.05, steps, how=how,
                  bodies=body, gl=1e-5, flow=1e-3)
    elif kind == "walls":
        shape = tuple(size(32, 224) for _ in range(3))
        c = _case("", q, shape, storage, rng.choice(("lid", "couette", "channel", "closed")), 0.06,
                  steps, how=how, force=rng.choice((0.0, 1e-6)))
    elif kind == "duct":
        shape = (size(48, 192), size(24, 80), size(24, 80))
        c = _case("", rng.choice((15, 19, 27)), shape, "fp32", "duct", 0.1, steps, how="run_step")
    else:
        shape = tuple(size(48, 224) for _ in range(3))
        c = _case("", q, shape, storage, rng.choice(("slab", "closed", "periodic")), 0.05,
                  rng.randint(3, 6), how="logged")
    c.pop("name")
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
# directions in the order of the reference's tables (the layout of ``flow.f``),
# one letter per component: - 0 +
_E13 = "000 ++0 +-0 +0+ +0- 0++ 0+- --0 -+0 -0- -0+ 0-- 0-+"
_E15 = "000 +00 -00 0+0 0-0 00+ 00- +++ -++ +-+ --+ ++- -+- +-- ---"
_E19 = "000 +00 -00 0+0 0-0 00+ 00- ++0 -+0 +-0 --0 0++ 0-+ 0+- 0-- +0+ -0+ +0- -0-"
_E27 = _E19 + " +++ ++- +-+ +-- -++ -+- --+ ---"
_DIRS = {13: _E13, 15: _E15, 19: _E19, 27: _E27}
# weights by number of non-zero components
_WEIGHTS = {13: (1 / 2, 0, 1 / 24, 0), 15: (2 / 9, 1 / 9, 0, 1 / 72),
            19: (1 / 3, 1 / 18, 1 / 36, 0), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}


def _velocities(q):
    e = [["-0+".index(s) - 1 for s in d] for d in _DIRS[q].split()]
    return e, [_WEIGHTS[q][sum(map(abs, v))] for v in e]


def _shape(c):
    return (c["x"], c["y"], c["z"])


def _initial(c, seed, e, w, device):
    """Initial populations, one float32 [x, y, z] plane set per direction:
    equilibrium of a Taylor-Green-like field of amplitude c["flow"] with the
    seed's phases and a slight density variation."""
    rng = np.random.default_rng(seed)
    ph = rng.uniform(0, 2 * np.pi, 4)
    amp = c["flow"] * rng.uniform(0.8, 1.0)
    ax = [2 * np.pi / s * torch.arange(s, device=device, dtype=torch.float32) for s in _shape(c)]
    x, y, z = ax[0][:, None, None] + float(ph[0]), ax[1][None, :, None] + float(ph[1]), \
        ax[2][None, None, :] + float(ph[2])
    u = [(amp * torch.sin(x)) * (torch.cos(y) * torch.cos(z)),
         (-amp * torch.cos(x)) * (torch.sin(y) * torch.cos(z)),
         (0.3 * amp * torch.cos(x)) * (torch.cos(y) * torch.sin(z + float(ph[3])))]
    rho = 1 + (0.05 * amp * torch.cos(x)) * (torch.cos(y) * torch.cos(z))
    usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    for i, (v, wi) in enumerate(zip(e, w)):
        eu = sum((s * 3.0) * u[k] for k, s in enumerate(v) if s)
        yield i, (wi * rho) * (1 - usq + ((1 + eu / 2) * eu if any(v) else 0.0))


def _bodies(text, shape, seed):
    """Configs of the bodies "sphere:r:density:count" or
    "ellipsoid:a:b:c:density:count", apart from each other and the walls,
    with the seed's positions and orientations."""
    if not text:
        return []
    parts = text.split(":")
    axes, rou, count = [int(v) for v in parts[1:-2]], float(parts[-2]), int(parts[-1])
    rng = np.random.default_rng(seed + 1)
    reach = max(axes) + 3.0
    centres, out = [], []
    for _ in range(20000):
        if len(centres) == count:
            break
        c = [float(rng.uniform(reach, s - 1 - reach)) for s in shape]
        if all(np.linalg.norm(np.subtract(c, d)) >= 2 * reach for d in centres):
            centres.append(c)
    for c in centres:
        rot = rng.uniform(-np.pi / 2, np.pi / 2, 3)
        coord = {"center": c, "alpha": float(rot[0]), "beta": float(rot[1]), "gamma": float(rot[2])}
        if parts[0] == "sphere":
            out.append({"type": "sphere", "r": axes[0], "rou": rou, "coord": coord})
        else:
            out.append({"type": "ellipsoid", "a": axes[0], "b": axes[1], "c": axes[2], "rou": rou,
                        "coord": coord})
    return out


def _config(c, seed):
    boundary = {f: {"code": CODES[k]} for f, k in zip(FACES, LAYOUTS[c["layout"]])}
    for f, k in zip(FACES, LAYOUTS[c["layout"]]):
        if k == "S":
            boundary[f]["uw"] = [0.0, 0.03, 0.0]
    flow = {"size": [s - 1 for s in _shape(c)], "param_type": "D3Q%d" % c["q"],
            "param": {"mu": c["mu"], "Re": 10.0, "gl": c["gl"]}, "boundary": boundary,
            "precision": {"storage": c["storage"]}}
    if c["force"]:
        flow["body_force"] = [0.0, 0.0, c["force"]]
    return {"device": "cuda", "log_per_steps": 10 ** 9, "file": {"per_steps": 10 ** 9},
            "flow": flow, "particles": _bodies(c["bodies"], _shape(c), seed)}


def _requests(c, seed):
    """Configs and step counts of a served batch: sizes, velocity sets,
    storages, faces and bodies mixed as in the benchmark's stream."""
    rng = np.random.default_rng(seed)
    sizes = np.arange(c["low"], c["high"] + 1, 16)
    out = []
    for j in range(c["requests"]):
        # the mix is the case's, the fields and positions are the seed's
        mix = np.random.default_rng(1000 * c["requests"] + c["steps"] + j)
        dims = [int(v) for v in mix.choice(sizes, 3)]
        boundary = {k: {"code": str(mix.choice(["WALL", "PERIODICAL"]))} for k in FACES}
        bodies = "sphere:%d:1.2:%d" % (mix.integers(4, 7), mix.integers(1, 4)) if j % 2 else ""
        out.append(({"device": "cuda",
                     "flow": {"size": dims, "param_type": "D3Q%d" % mix.choice([19, 27]),
                              "param": {"mu": 0.05, "gl": 1e-5}, "boundary": boundary,
                              "precision": {"storage": str(mix.choice(["fp32", "fp16s"]))},
                              "init_field": {"type": "taylor_green",
                                             "u0": float(rng.uniform(0.02, 0.05))}},
                     "particles": _bodies(bodies, [d + 1 for d in dims],
                                          int(rng.integers(1 << 30)))},
                    int(mix.integers(c["steps"] // 2, c["steps"] + 1))))
    return out


def prepare(case, seed):
    if case["kind"] == "serve":
        from funlbm_b200.serve import LBMServer, Request

        reqs = _requests(case, seed)
        server = LBMServer(budget_bytes=8e9, reserve=False)
        server.prepare([Request(cfg, steps) for cfg, steps in reqs])
        return {"case": case, "server": server, "requests": reqs}
    from funlbm_b200.lbm import LBMD3, Config

    e, w = _velocities(case["q"])
    lbm = LBMD3(config=Config().from_json(_config(case, seed)))
    f0 = torch.empty((case["q"],) + _shape(case), device="cuda",
                     dtype=torch.float64 if case["storage"] == "fp64" else torch.float32)
    for i, plane in _initial(case, seed, e, w, "cuda"):
        f0[i] = plane
    lbm.flow.init()
    lbm.flow.f = f0.permute(1, 2, 3, 0)
    lbm.flow.update_u_rou()
    lbm.flow.cul_equ()
    lbm.particle_swarm.init()
    lbm.run_steps(1)
    return {"case": case, "lbm": lbm}


def run(state):
    case = state["case"]
    if case["kind"] == "serve":
        from funlbm_b200.serve import Request

        reqs = [Request(cfg, steps) for cfg, steps in state["requests"]]
        state["server"].run(reqs, realtime=False)
        state["server"].done.clear()
        return [{k: v for k, v in r.result.items() if torch.is_tensor(v)} for r in reqs]
    lbm = state["lbm"]
    out = {}
    if case["how"] == "run_steps":
        lbm.run_steps(case["steps"])
    else:
        for _ in range(case["steps"]):
            lbm.run_step(step=lbm.step)
            lbm.step += 1
            if case["how"] == "logged":
                out["stats"] = lbm.flow.step_stats()
    out["u"] = lbm.flow.u
    out["rho"] = lbm.flow.rou
    sw = lbm.particle_swarm
    if sw.particles:
        out.update(cx=sw.cx, cu=sw.cu, cw=sw.cw, lx=sw.lx, lF=sw.lF)
    return out


def work(case):
    """Every step reads and writes each population once; the fields that are
    read back are written once more."""
    if case["kind"] == "serve":
        total = {"bytes": 0, "flops": 0}
        for cfg, steps in _requests(case, 0):
            dims = [d + 1 for d in cfg["flow"]["size"]]
            c = {"kind": "solve", "q": int(cfg["flow"]["param_type"][3:]), "x": dims[0],
                 "y": dims[1], "z": dims[2], "storage": cfg["flow"]["precision"]["storage"],
                 "steps": steps}
            for k, v in work(c).items():
                total[k] += v
        return total
    n = case["x"] * case["y"] * case["z"]
    field = 16 if case["storage"] != "fp64" else 32
    return {"bytes": n * (2 * case["q"] * STORED[case["storage"]] * case["steps"] + field),
            "flops": n * case["steps"] * (10 * case["q"] + 20)}


# ---------------------------------------------------------------------------
# The same simulations in float64, plain torch
# ---------------------------------------------------------------------------
def _duct_profile(a, b):
    y, z = (np.linspace(-(s - 1) / 2, (s - 1) / 2, s) for s in (a, b))
    ha, hb = a / 2.0, b / 2.0
    val = np.broadcast_to(1 - (y[:, None] / ha) ** 2, (a, b)).copy()
    for k in range(100):
        m = (2 * k + 1) * np.pi
        val += (32 * (-1.0) ** (k + 1) / m ** 3 * np.cos(m * y[:, None] / (2 * ha))
                * np.cosh(m * z[None] / (2 * ha)) / np.cosh(m * hb / (2 * ha)))
    return np.round(val, 6)


class _Flow64:
    """Populations, density, velocity and force of one lattice."""

    def __init__(self, q, shape, letters, mu, f0, device, re=10.0):
        self.e, self.w = _velocities(q)
        self.rev = [self.e.index([-s for s in v]) for v in self.e]
        self.letters, self.tau, self.shape = letters, float(np.float32(3 * mu + 0.5)), shape
        self.re_mu = re * mu
        self.f = f0
        self.F = [torch.zeros(shape, dtype=torch.float64, device=device) for _ in range(3)]
        self.profile = None
        if letters[0] == "N":
            self.profile = torch.tensor(_duct_profile(*shape[1:]), device=device)
        self.moments()
        self.collide()

    def dot(self, v, t):
        return sum(float(s) * t[k] for k, s in enumerate(v) if s) if any(v) else 0.0

    def plane(self, face, at=None):
        idx = [slice(None)] * 3
        idx[face // 2] = (0 if face % 2 == 0 else -1) if at is None else at
        return tuple(idx)

    def moments(self):
        rho = sum(self.f)
        u = []
        for k in range(3):
            j = 0.5 * self.F[k]
            for v, f in zip(self.e, self.f):
                if v[k]:
                    j = j + v[k] * f
            u.append(j / rho)
        for face in range(6):
            for k in range(3):
                u[k][self.plane(face)] = 0
        if self.letters[0] == "N":
            speed = self.re_mu / float(rho.max()) / min(self.shape[1:])
            u[0][0] = speed * self.profile
            rho[0] = rho[1]
        if self.letters[1] == "N":
            rho[-1] = rho[-2]
            for k in range(3):
                u[k][-1] = u[k][-2]
        self.rho, self.u = rho, u

    def equilibrium(self, i):
        t = 3.0 * self.dot(self.e[i], self.u)
        usq = 1.5 * (self.u[0] ** 2 + self.u[1] ** 2 + self.u[2] ** 2)
        return self.w[i] * self.rho * (1 + t + t * t / 2 - usq)

    def collide(self):
        keep = "N" in self.letters
        self.feq = {}
        for i in range(len(self.f)):
            feq = self.equilibrium(i)
            self.f[i] = self.f[i] - (self.f[i] - feq) / self.tau
            if keep:
                self.feq[i] = feq

    def stream(self):
        old = self.f
        new = [torch.roll(f, v, (0, 1, 2)) for f, v in zip(old, self.e)]
        for face, letter in enumerate(self.letters):
            axis, sign = face // 2, 1 if face % 2 == 0 else -1
            at = self.plane(face)
            for i, v in enumerate(self.e):
                if letter == "N":
                    near = self.plane(face, 1 if sign > 0 else -2)
                    new[i][at] = self.feq[i][at] + new[i][near] - self.feq[i][near]
                elif v[axis] != sign:
                    continue
                elif letter == "P":
                    new[i][at] = old[i][self.plane(face ^ 1)]
                else:
                    new[i][at] = old[self.rev[i]][at]
                    if letter == "S":
                        new[i][at] = new[i][at] - 6.0 * self.rho[at] * self.w[i] * (0.03 * v[1])
        self.f = new

    def add_force(self):
        c = 1 - 1 / (2 * self.tau)
        uF = sum(self.u[k] * self.F[k] for k in range(3))
        for i, v in enumerate(self.e):
            t = 3.0 * (self.dot(v, self.F) - uF)
            for k, s in enumerate(v):
                if s:
                    t = t + 9.0 * self.u[k] * self.F[k]
            self.f[i] = self.f[i] + c * self.w[i] * t


def _surface(a, b, c):
    """Markers on an ellipsoid: for every unit cube that the surface cuts at
    three or more corner pairs, the mean of the crossings on its corner
    pairs."""
    ax = [np.arange(-r - 2, r + 2, 1.0) for r in (a, b, c)]
    inside = ((ax[0] ** 2 / a ** 2)[:, None, None] + (ax[1] ** 2 / b ** 2)[None, :, None]
              + (ax[2] ** 2 / c ** 2)[None, None, :] - 1) < 0
    corners = [(i, j, k) for i in (0, 1) for j in (0, 1) for k in (0, 1)]
    pts = []
    for i in range(len(ax[0]) - 1):
        for j in range(len(ax[1]) - 1):
            for k in range(len(ax[2]) - 1):
                cut = inside[i:i + 2, j:j + 2, k:k + 2]
                if cut.all() or not cut.any():
                    continue
                cross = []
                for m, p in enumerate(corners):
                    for r in corners[m + 1:]:
                        if cut[p] == cut[r]:
                            continue
                        p1 = np.array([ax[0][i + p[0]], ax[1][j + p[1]], ax[2][k + p[2]]])
                        d = np.subtract(r, p).astype(float)
                        s = np.array([a, b, c], float) ** -2
                        A, B, C = (d * d * s).sum(), 2 * (p1 * d * s).sum(), (p1 * p1 * s).sum() - 1
                        sq = math.sqrt(max(B * B - 4 * A * C, 0.0))
                        t = min(((-B - sq) / (2 * A), (-B + sq) / (2 * A)), key=lambda v: abs(v - 0.5))
                        cross.append(p1 + t * d)
                if len(cross) >= 3:
                    pts.append(np.mean(cross, axis=0))
    return np.array(pts)


class _Bodies64:
    """Rigid bodies with surface markers."""

    def __init__(self, configs, gl, device):
        t = lambda v: torch.tensor(np.array(v, np.float64), device=device)  # noqa: E731
        X, who, lm, self.mass, inertia, known = [], [], [], [], [], {}
        for j, p in enumerate(configs):
            axes = (p["r"],) * 3 if p["type"] == "sphere" else (p["a"], p["b"], p["c"])
            if axes not in known:
                known[axes] = _surface(*axes)
            pts, (a, b, c) = known[axes], axes
            area = (4 * math.pi * a * a if p["type"] == "sphere"
                    else 4 / 3 * math.pi * (a * b * c) ** (2 / 3))
            X.append(pts)
            who.append(np.full(len(pts), j))
            lm.append(np.full(len(pts), area / len(pts)))
            self.mass.append(4 / 3 * math.pi * a * b * c)
            inertia.append(np.array([b * c, a * c, a * b]) * self.mass[-1] / 5)
        self.X, self.lm, self.I, self.mass = t(np.concatenate(X)), t(np.concatenate(lm)), t(inertia), t(self.mass)
        self.who = torch.tensor(np.concatenate(who), device=device)
        self.rou, self.gl = t([p["rou"] for p in configs]), float(np.float32(gl))
        self.cx = t([p["coord"]["center"] for p in configs])
        self.angle = t([[p["coord"][k] for k in ("alpha", "beta", "gamma")] for p in configs])
        self.cu, self.cw = torch.zeros_like(self.cx), torch.zeros_like(self.cx)
        self.lx = torch.zeros_like(self.X)

    def stencil(self, shape):
        size = torch.tensor([s - 1 for s in shape], device=self.X.device, dtype=torch.float64)
        lo = torch.minimum((self.lx.floor() - 1).clamp(min=0), size)
        hi = torch.minimum(lo + 4, size)
        off = torch.cartesian_prod(*[torch.arange(4, device=self.X.device)] * 3).double()
        at = lo[:, None] + off[None]
        ok = (at < hi[:, None]).all(-1)
        r = (at - self.lx[:, None]).abs()
        wt = ((1 + torch.cos(r * math.pi / 2)) / 4 * (r <= 2)).prod(-1) * ok
        total = wt.sum(1, keepdim=True)
        wt = torch.where(total > 0, wt / total, wt)
        at = at.long().clamp(min=0)
        return ok, wt, (at[..., 0] * shape[1] + at[..., 1]) * shape[2] + at[..., 2]

    def couple(self, flow):
        """Marker forces from the flow, the wall spring, the forces on the
        nodes and the bodies' new state."""
        shape = flow.shape
        ok, wt, at = self.stencil(shape)
        flat = at.clamp(max=shape[0] * shape[1] * shape[2] - 1)
        s = (flow.u[0] + flow.u[1] + flow.u[2]).reshape(-1)[flat]
        lus, lrho = (wt * s).sum(1), (wt * flow.rho.reshape(-1)[flat]).sum(1)
        arm = self.lx - self.cx[self.who]
        v = self.cu[self.who] + torch.linalg.cross(self.cw[self.who], arm)
        self.lF = 2 * lrho[:, None] * (v - lus[:, None])
        for j in range(len(self.mass)):
            mine = (self.who == j).nonzero()[:, 0]
            pos = self.lx[mine].cpu().numpy()
            ext = list(pos.argmin(0)) + list(pos.argmax(0))
            wall = [0.0] * 3 + [n - 1.0 for n in shape]
            d = [max(300 * (1 - abs(pos[m, k % 3] - wall[k]) / 2), 0.0) for k, m in enumerate(ext)]
            if max(d) > 0:
                new = [self.lF[mine[m]].clone() for m in ext]
                for k in range(6):
                    new[k][k % 3] += d[k] if k < 3 else -d[k]
                for k in range(6):
                    self.lF[mine[ext[k]]] = new[k]
        pull = wt[..., None] * self.lF[:, None] * self.lm[:, None, None]
        n = shape[0] * shape[1] * shape[2]
        field = torch.zeros((n, 3), dtype=torch.float64, device=self.X.device)
        # of the markers that reach a node the last one writes it
        m = torch.arange(len(self.lx), device=self.X.device)[:, None].expand_as(flat)
        last = torch.full((n,), -1, device=self.X.device)
        last.scatter_reduce_(0, flat[ok], m[ok], "amax")
        win = ok & (last[flat] == m)
        field[flat[win]] = pull[win]
        flow.F = [field[:, k].reshape(shape) for k in range(3)]
        sums = lambda t: torch.zeros_like(self.cx).index_add_(0, self.who, t)  # noqa: E731
        load = self.lF * self.lm[:, None]
        cF = -sums(load)
        cF[:, 0] += (1 - self.rou) * self.mass * self.gl
        self.cu = self.cu + cF / self.mass[:, None]
        self.cx = self.cx + self.cu
        cT = -sums(torch.linalg.cross(self.lx - self.cx[self.who], load))
        self.cw = self.cw + 0.1 * cT / self.I

    def move(self):
        self.angle = self.angle + self.cw
        th = self.angle.norm(dim=1, keepdim=True)
        k = (self.angle / th.clamp(min=1e-300))[self.who]
        c, s = torch.cos(th)[self.who], torch.sin(th)[self.who]
        turned = self.X * c + torch.linalg.cross(k, self.X) * s + k * (k * self.X).sum(1, keepdim=True) * (1 - c)
        self.lx = turned + self.cx[self.who]


def _solve64(flow, bodies, steps, force=0.0):
    for _ in range(steps):
        flow.collide()
        flow.stream()
        flow.moments()
        if bodies is not None:
            bodies.couple(flow)
        else:
            flow.F = [torch.zeros_like(flow.rho) for _ in range(3)]
        if force:
            flow.F[2] = flow.F[2] + float(np.float32(force))
        if bodies is not None or force:
            flow.add_force()
            flow.moments()
        if bodies is not None:
            bodies.move()
    out = {"u": torch.stack(flow.u, -1), "rho": flow.rho[..., None]}
    if bodies is not None:
        out.update(cx=bodies.cx, cu=bodies.cu, cw=bodies.cw, lx=bodies.lx, lF=bodies.lF)
    return out


def _served64(cfg, steps, device):
    f = cfg["flow"]
    shape = tuple(d + 1 for d in f["size"])
    x, y, z = (2 * math.pi / s * torch.arange(s, device=device, dtype=torch.float64) for s in shape)
    x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]
    u0 = f["init_field"]["u0"]
    u = [u0 * torch.sin(x) * torch.cos(y) * torch.cos(z), -u0 * torch.cos(x) * torch.sin(y) * torch.cos(z)]
    q = int(f["param_type"][3:])
    f0 = []
    for v, w in zip(*_velocities(q)):
        t = 3.0 * (v[0] * u[0] + v[1] * u[1])
        f0.append(w * (1 + t + t * t / 2 - 1.5 * (u[0] ** 2 + u[1] ** 2)))
    letters = "".join(f["boundary"][k]["code"][0] for k in FACES)
    flow = _Flow64(q, shape, letters, f["param"]["mu"], f0, device)
    bodies = _Bodies64(cfg["particles"], f["param"]["gl"], device) if cfg["particles"] else None
    out = _solve64(flow, bodies, steps)
    return {k: out[k] for k in ("rho", "u", "cx", "cu", "cw") if k in out}


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "serve":
        return [_served64(cfg, steps, device) for cfg, steps in _requests(case, seed)]
    n = case["x"] * case["y"] * case["z"]
    if n * case["q"] > 1 << 30:      # (512^3: too long in float64)
        return None
    e, w = _velocities(case["q"])
    f0 = [None] * case["q"]
    for i, plane in _initial(case, seed, e, w, device):
        f0[i] = plane.to(torch.float64)
    cfg = _config(case, seed)
    flow = _Flow64(case["q"], _shape(case), LAYOUTS[case["layout"]], case["mu"], f0, device)
    bodies = _Bodies64(cfg["particles"], case["gl"], device) if cfg["particles"] else None
    out = _solve64(flow, bodies, 1 + case["steps"], case["force"])
    if case["how"] == "logged":
        e3 = [torch.stack(flow.f), out["u"], out["rho"]]
        out["stats"] = torch.stack([v for t in e3 for v in (t.min(), t.mean(), t.max())])
    return out
