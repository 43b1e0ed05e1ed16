"""The work that users of this package have it do, as cases that can be timed and checked.

A case is one call sequence of the public entry points on one wall ensemble:

``advance``   ``GPUSolidSolver.Advance``: the time loop between two saves of a run
``solve``     ``RefreshContext`` + ``Solve`` + ``Norms`` per step, as a host code that
              drives the wall solver step by step (and watches it) calls it
``geo``       ``Advance`` with the stiffness and follower pressure rebuilt on x + u every
              ``interval`` steps (``stiffness_update_interval``)
``batch``     ``BatchedSolidSolver.Advance``: many uneven tubes together
``gradient``  ``wall_mismatch`` and its backward pass: one objective and gradient of the
              inverse wall-stiffness problem
``stress``    ``GPUSolidSolver.Stress``: the element stresses that every save writes

Every wall is the structured tube of :mod:`cvfes_b200.mesh` (straight or stenosed); its
material is a smooth log-normal field per sample (sigma 0.2 for E, 0.1 for h, the law of
:mod:`cvfes_b200.cases`, from a few Fourier modes in place of the host-side GMRF draw), its
time step the CFL rule's.  Runs start from a smooth displacement and velocity, as a restart
does.  ``exact`` restates the same computations in FP64 with plain torch.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

NU, RHO, DAMP = 0.49, 1.0, 100.0
P_REF = 1.33e5


def listed():
    return [
        # the smallest calls: one step at a time with its norms on the default wall and
        # sample count (64 x 128 nodes, 8 samples), host and launch latency
        dict(name="solve_small_f32", path="solve", nc=64, na=128, stenosed=False, S=8,
             precision=32, steps=1, lumping="reference"),
        # the default configuration: FP64, 8 samples, 400 steps with 4 saves
        dict(name="advance_default_f64", path="advance", nc=64, na=128, stenosed=False, S=8,
             precision=64, steps=100, lumping="reference"),
        # large FP32 ensemble, many steps between saves (CUDA graph replays)
        dict(name="advance_large_f32", path="advance", nc=256, na=512, stenosed=False, S=256,
             precision=32, steps=50, lumping="rowsum"),
        # large FP64 ensemble, short runs (plain launches)
        dict(name="advance_large_f64", path="advance", nc=256, na=512, stenosed=False, S=64,
             precision=64, steps=20, lumping="rowsum"),
        # a sample count and a mesh that are multiples of nothing convenient
        dict(name="advance_ragged_f32", path="advance", nc=90, na=301, stenosed=True, S=100,
             precision=32, steps=24, lumping="reference"),
        # step-by-step driving of a large ensemble, norms and watchdog every step
        dict(name="solve_large_f32", path="solve", nc=256, na=400, stenosed=True, S=128,
             precision=32, steps=4, lumping="rowsum"),
        # stiffness on the deformed wall every step (the reference cfgs' setting)
        dict(name="geo_f32", path="geo", nc=128, na=400, stenosed=True, S=128, precision=32,
             steps=10, interval=1, lumping="reference"),
        dict(name="geo_f64", path="geo", nc=96, na=200, stenosed=False, S=50, precision=64,
             steps=10, interval=1, lumping="reference"),
        # an uneven batch of tubes
        dict(name="batch_f32", path="batch", tubes=10, na_max=400, precision=32, steps=60),
        # inverse estimation: the small wall with its usual intervals, and a larger
        # stenosed one with the thickness gradient, FP32 and FP64
        dict(name="gradient_small_f32", path="gradient", nc=64, na=128, stenosed=False, S=64,
             precision=32, steps=100, n_obs=512, obs_every=10, ckpt_every=50, logh=False),
        dict(name="gradient_large_f64", path="gradient", nc=128, na=320, stenosed=True, S=64,
             precision=64, steps=60, n_obs=1024, obs_every=10, ckpt_every=30, logh=True),
        # stress recovery at a save
        dict(name="stress_f32", path="stress", nc=256, na=400, stenosed=True, S=128,
             precision=32, lumping="rowsum"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["advance", "advance", "solve", "geo", "batch", "gradient", "stress"])
    precision = rng.choice([32, 32, 64])
    if path == "batch":
        return dict(path=path, tubes=rng.randint(3, 9), na_max=rng.randint(80, 380),
                    precision=precision, steps=rng.randint(12, 58 * 32 // precision))
    nc = _log_int(rng, 24, 256)
    na = _log_int(rng, 40, 512)
    S = rng.choice([_log_int(rng, 3, 256), rng.choice([8, 16, 32, 50, 64, 100, 128, 256])])
    limit = {"advance": 12e6, "solve": 12e6, "geo": 6e6, "gradient": 2.5e6, "stress": 12e6}[path]
    while nc * na * S * (precision // 32) > limit:
        if na > 40:
            na = max(40, int(na * 0.7))
        else:
            nc = max(24, int(nc * 0.7))
    case = dict(path=path, nc=nc, na=na, stenosed=rng.random() < 0.5, S=S, precision=precision)
    if path == "gradient":
        case.update(steps=rng.randint(20, 55), n_obs=_log_int(rng, 20, 800),
                    obs_every=rng.choice([3, 5, 10]), ckpt_every=rng.choice([10, 17, 25]),
                    logh=rng.random() < 0.5)
        return case
    case["lumping"] = rng.choice(["reference", "rowsum"])
    if path == "advance":
        case["steps"] = rng.choice([rng.randint(1, 40), rng.randint(48, 50)])
    elif path == "solve":
        case["steps"] = rng.randint(1, 4)
    elif path == "geo":
        case["steps"] = rng.randint(2, 10)
        case["interval"] = rng.choice([1, 1, 1, 3])
    return case


# ------------------------------------------------------------------ inputs
def _batch_cases(case, seed):
    """The tubes of a batch: the ranges of :func:`cvfes_b200.cases.batched_cases`, shorter.
    The mix of shapes is the case's, only the material is the seed's."""
    r = np.random.default_rng(1000 + 7 * case["tubes"] + case["na_max"])
    out = []
    for i in range(case["tubes"]):
        out.append(dict(nc=int(r.choice([32, 64, 128, 256])),
                        na=int(r.integers(64, case["na_max"] + 1)), stenosed=False,
                        S=int(r.choice([16, 32, 64, 128, 256])), lumping="reference",
                        radius=float(r.uniform(0.15, 0.6)), length=float(r.uniform(1.0, 6.0)),
                        precision=case["precision"], steps=case["steps"], constant=True,
                        seed=100 * seed + i))
    return out


def _geometry(case):
    """Ring-major tube (nodes, triangles, boundary ids) and its radius and length."""
    nc, na = case["nc"], case["na"]
    radius = case.get("radius", 0.3)
    length = case.get("length", 5.0 if case["stenosed"] else 3.0 * na / (2.0 * nc))
    x = np.linspace(0.0, length, na)
    r = np.full(na, radius)
    if case["stenosed"]:
        r = r * (1.0 - 0.5 * np.exp(-((x - 2.5) / 0.3) ** 2))
    th = 2.0 * np.pi * np.arange(nc) / nc
    nodes = np.stack([r[:, None] * np.cos(th), r[:, None] * np.sin(th),
                      np.broadcast_to(x[:, None], (na, nc))], axis=-1).reshape(-1, 3)
    j, i = np.arange(na - 1)[:, None], np.arange(nc)[None, :]
    n00, n01 = j * nc + i, j * nc + (i + 1) % nc
    n10, n11 = n00 + nc, n01 + nc
    elems = np.stack([np.stack([n00, n01, n11], -1), np.stack([n00, n11, n10], -1)],
                     axis=2).reshape(-1, 3).astype(np.int64)
    boundary = np.concatenate([np.arange(nc), (na - 1) * nc + np.arange(nc)])
    return nodes, elems, boundary, radius, length


def _fields(case, seed):
    """Everything random of one wall, from the seed, on the GPU in FP64: E and h per element
    and sample, the start displacement and velocity per node, and the pressures."""
    dev = "cuda"
    nodes, elems, boundary, radius, length = _geometry(case)
    g = torch.Generator(device=dev)
    g.manual_seed(int(case.get("seed", seed)) * 2654435761 % (1 << 31))
    rnd = lambda *shape: torch.randn(*shape, generator=g, device=dev, dtype=torch.float64)
    p = torch.from_numpy(nodes).to(dev)
    el = torch.from_numpy(elems).to(dev)
    theta = torch.atan2(p[:, 1], p[:, 0])
    z = p[:, 2] / length
    modes = [(m, k) for m in range(4) for k in range(1, 5)]
    tn = torch.stack([torch.cos(m * theta) * torch.sin(math.pi * k * z) for m, k in modes] +
                     [torch.sin(m * theta) * torch.sin(math.pi * k * z) for m, k in modes
                      if m > 0], dim=1)
    te = tn[el].mean(dim=1)
    scale = 1.0 / te.square().sum(1).mean().sqrt()
    S = case["S"]
    E = 7.0e6 * torch.exp(0.2 * scale * (te @ rnd(te.shape[1], S)).clamp(-8, 8))
    h = 0.04 * torch.exp(0.1 * scale * (te @ rnd(te.shape[1], S)).clamp(-8, 8))
    radial = torch.stack([torch.cos(theta), torch.sin(theta), torch.zeros_like(theta)], 1)
    amp = 2.0e-3 * scale * (tn @ rnd(tn.shape[1], 3))  # vanishes on the end rings
    u0 = amp + 2.0e-3 * torch.sin(math.pi * z)[:, None] * radial
    du0 = 1.0 * scale * (tn @ rnd(tn.shape[1], 3))
    u0[torch.from_numpy(boundary).to(dev)] = 0.0
    du0[torch.from_numpy(boundary).to(dev)] = 0.0
    steps = case.get("steps", 1)
    phase = float(rnd(1).cpu())
    pres = P_REF * (0.8 + 0.2 * np.sin(0.05 * np.arange(steps) + phase))
    if case.get("constant"):
        pres = P_REF * np.ones(steps)
    if case.get("path") == "geo":
        pres = 0.1 * pres  # the follower load on a wall that stays near its shape
    return SimpleNamespace(nodes=nodes, elems=elems, boundary=boundary, E=E, h=h, u0=u0, du0=du0,
                           pres=pres, radial=radial, S=S)


def _dt(f):
    from cvfes_b200.mesh import cfl_dt
    return cfl_dt(f.nodes, f.elems, 7.0e6 * math.exp(0.2 * 4.0), RHO)


def _mesh(case, f):
    from cvfes_b200.mesh import SolidMesh
    c, h = (f.E * f.h).cpu().numpy(), f.h.cpu().numpy()
    return SolidMesh(nodes=f.nodes, elementNodeIds=f.elems, boundary=f.boundary, nSmp=f.S,
                     density=RHO, v=NU, damp=DAMP, bdyU=0.0, coefK=c, gthick=h,
                     iniU=f.u0.reshape(-1).cpu().numpy(), iniDu=f.du0.reshape(-1).cpu().numpy(),
                     mass_lumping=case.get("lumping", "reference"))


def _config(case, dt):
    # the ramp of a run: full pressure after 100 steps
    return SimpleNamespace(dt=dt, nSmp=case["S"], constant_pressure=P_REF, constant_T=100 * dt,
                           pressure_ramp="linear", update_interval=case.get("interval", 0),
                           gpu=SimpleNamespace(precision=case["precision"], use_graph=True,
                                               graph_chunk=48, watchdog=True, device=-1,
                                               norms_every=1 if case["path"] == "solve" else 0))


def _observations(case, f, dt):
    """Measured displacements (K, n_obs, 3, S): a radial motion with noise, and the nodes."""
    n = len(f.nodes)
    free = np.setdiff1d(np.arange(n), f.boundary)
    nodes = np.sort(np.random.default_rng(99).choice(free, min(case["n_obs"], len(free)),
                                                     replace=False))
    K = case["steps"] // case["obs_every"]
    t = dt * case["obs_every"] * torch.arange(1, K + 1, device="cuda", dtype=torch.float64)
    rise = P_REF / (RHO * 0.04) * t.square() * 0.3
    rad = f.radial[torch.from_numpy(nodes).cuda()]
    g = torch.Generator(device="cuda")
    g.manual_seed(4 + len(nodes))
    noise = torch.randn(K, len(nodes), 1, f.S, generator=g, device="cuda", dtype=torch.float64)
    return nodes, rise[:, None, None, None] * rad[None, :, :, None] * (1.0 + 0.1 * noise)


def _gradient_pressures(case):
    return P_REF * np.minimum(np.arange(case["steps"]) / 20.0, 1.0)


def prepare(case, seed):
    from cvfes_b200.solver import FluidSolver, GPUSolidSolver, LocalComm
    path = case["path"]
    if path == "batch":
        from cvfes_b200.batched import BatchedSolidSolver
        meshes, dts = [], []
        for c in _batch_cases(case, seed):
            f = _fields(c, seed)
            meshes.append(_mesh(c, f))
            dts.append(_dt(f))
        b = BatchedSolidSolver(meshes, dts, precision=case["precision"],
                               device="cuda:%d" % torch.cuda.current_device())
        return dict(path=path, batch=b, pres=P_REF * np.ones(case["steps"]))
    f = _fields(case, seed)
    dt = _dt(f)
    if path == "gradient":
        from cvfes_b200.adjoint import MismatchProblem
        nodes, obs = _observations(case, f, dt)
        problem = MismatchProblem(_mesh(case, f), dt, _gradient_pressures(case), nodes,
                                  obs_every=case["obs_every"], ckpt_every=case["ckpt_every"],
                                  precision=case["precision"], grad_logh=case["logh"])
        problem.set_observations(obs)
        logE = torch.log(f.E).requires_grad_(True)
        logh = torch.log(f.h).requires_grad_(bool(case["logh"]))
        return dict(path=path, problem=problem, logE=logE, logh=logh)
    solver = GPUSolidSolver(LocalComm(), _mesh(case, f), _config(case, dt))
    state = dict(path=path, solver=solver, pres=f.pres, dt=dt)
    if path == "solve":
        state.update(fluid=FluidSolver(LocalComm(), None, SimpleNamespace(dt=dt)), t=0.0,
                     steps=case["steps"],
                     norms=torch.empty((case["S"], 4), dtype=torch.float64, pin_memory=True))
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    path = state["path"]
    if path == "batch":
        b = state["batch"]
        b.Advance(state["pres"])
        return [(s.bufs[s.cur], s.bufs[s.prev]) for s in b.solvers]
    if path == "gradient":
        from cvfes_b200.adjoint import wall_mismatch
        logE, logh = state["logE"], state["logh"]
        logE.grad = logh.grad = None
        J = wall_mismatch(logE, logh, state["problem"])
        J.sum().backward()
        return {"J": J.detach(), "logE": logE.grad, "logh": logh.grad}
    solver = state["solver"]
    if path == "stress":
        return solver.Stress()
    if path == "solve":
        fluid, dt = state["fluid"], state["dt"]
        for _ in range(state["steps"]):
            fluid.Solve(state["t"], dt)
            solver.RefreshContext(fluid)
            solver.Solve(state["t"], dt)
            solver.Norms(out=state["norms"])
            state["t"] += dt
        return {"u": solver.local_displacement(), "du": solver.bufs[solver.prev],
                "norms": state["norms"]}
    solver.Advance(state["pres"], dt=state["dt"])
    return {"u": solver.local_displacement(), "prev": solver.bufs[solver.prev]}


# ------------------------------------------------------------------ work of one pass
def _counts(case):
    N, E = case["nc"] * case["na"], 2 * case["nc"] * (case["na"] - 1)
    return N, E, case["S"], case["precision"] // 8


def _step_bytes(case):
    """One step streams the wall's state: u and the second state row read, both new rows
    written where the state form has two (FP32), the inverse mass and the coefficient of
    every element read, and the mesh shared by all samples."""
    N, E, S, b = _counts(case)
    rows = 13 if case["precision"] == 32 and case["path"] != "geo" else 10
    return S * b * (rows * N + E) + E * (12 + 45 * b) + 3 * N * b


def work(case):
    path = case["path"]
    if path == "batch":
        parts = [work(dict(c, path="advance")) for c in _batch_cases(case, 0)]
        return {k: sum(w[k] for w in parts) for k in ("bytes", "flops")}
    N, E, S, b = _counts(case)
    if path == "stress":
        return {"bytes": E * S * (8 + 5 * b) + 3 * N * S * b, "flops": 150.0 * E * S}
    n = case["steps"]
    if path == "gradient":
        fwd = S * b * (10 * N + E)
        rev = S * b * (19 * N + 3 * E + (2 * N if case["logh"] else 0))
        return {"bytes": n * (fwd + rev) + E * S * 8 * (4 if case["logh"] else 3),
                "flops": n * S * (E * (3 * 126.0 + 100.0) + 90.0 * N)}
    # each element: three 3 x 6 row blocks and their coefficient; the geometric form also
    # builds the blocks (about 130 operations a row)
    per_elem = 3 * (42.0 if path != "geo" else 130.0)
    return {"bytes": n * _step_bytes(case) + (32 * S if path == "solve" else 0),
            "flops": n * S * (per_elem * E + 24.0 * N)}


# ------------------------------------------------------------------ the same in FP64
class _Wall:
    """The wall in FP64 with plain torch, boundary nodes first (the solver's local order)."""

    def __init__(self, case, f):
        n = len(f.nodes)
        bdy = torch.from_numpy(f.boundary).cuda()
        mask = torch.ones(n, dtype=torch.bool, device="cuda")
        mask[bdy] = False
        self.l2g = torch.cat([bdy, torch.nonzero(mask).ravel()])
        self.g2l = torch.empty_like(self.l2g)
        self.g2l[self.l2g] = torch.arange(n, device="cuda")
        self.el = self.g2l[torch.from_numpy(f.elems).cuda()]
        self.x = torch.from_numpy(f.nodes).cuda()[self.l2g]
        self.n, self.nb = n, len(f.boundary)
        self.c, self.h = f.E * f.h, f.h
        self.u0, self.du0 = f.u0[self.l2g], f.du0[self.l2g]
        B, area, nrm = self._strain(self.x[self.el].unsqueeze(-1))
        self.area, D = area[:, 0], self._D()
        self.K = torch.einsum("epi,pq,eqj->eij", B[..., 0], D, B[..., 0]) * area[:, :, None]
        fe = (area / 3.0) * nrm[..., 0]
        self.f = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        for a in range(3):
            self.f.index_add_(0, self.el[:, a], fe)
        w = RHO / 9.0 if case.get("lumping", "reference") == "reference" else RHO / 3.0
        self.alpha = w * self.area  # mass of a node per unit thickness of the element
        self.m = torch.zeros(n, f.S, dtype=torch.float64, device="cuda")
        for a in range(3):
            self.m.index_add_(0, self.el[:, a], self.alpha[:, None] * self.h)

    @staticmethod
    def _D():
        q = 1.0 - NU * NU
        D = torch.zeros(5, 5, dtype=torch.float64, device="cuda")
        D[0, 0] = D[1, 1] = 1.0 / q
        D[0, 1] = D[1, 0] = NU / q
        D[2, 2] = 0.5 * (1 - NU) / q
        D[3, 3] = D[4, 4] = 0.5 * (5.0 / 6.0) * (1 - NU) / q
        return D

    @staticmethod
    def _frame(P):
        """Local axes (E,3,s each) and area of triangles P (E, 3 nodes, 3, s)."""
        ex = P[:, 2] - P[:, 1]
        ex = ex / ex.norm(dim=1, keepdim=True)
        ey = P[:, 0] - P[:, 2]
        ey = ey - (ex * ey).sum(1, keepdim=True) * ex
        ey = ey / ey.norm(dim=1, keepdim=True)
        ez = torch.linalg.cross(ex, ey, dim=1)
        cr = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0], dim=1)
        return ex, ey, ez, 0.5 * cr.norm(dim=1)

    @classmethod
    def _strain(cls, P):
        """B (E,5,9,s): local strains from global displacements; area (E,s); normal (E,3,s)."""
        ex, ey, ez, area = cls._frame(P)
        lx = (P * ex.unsqueeze(1)).sum(2)
        ly = (P * ey.unsqueeze(1)).sum(2)
        B = torch.zeros(P.shape[0], 5, 9, P.shape[3], dtype=P.dtype, device=P.device)
        for a in range(3):
            i, j = (a + 1) % 3, (a + 2) % 3
            by = ((ly[:, i] - ly[:, j]) / (2 * area)).unsqueeze(1)
            bx = ((lx[:, j] - lx[:, i]) / (2 * area)).unsqueeze(1)
            s = slice(3 * a, 3 * a + 3)
            B[:, 0, s], B[:, 1, s] = by * ex, bx * ey
            B[:, 2, s] = bx * ex + by * ey
            B[:, 3, s], B[:, 4, s] = by * ez, bx * ez
        return B, area, ez

    def chunks(self, width):
        S = self.c.shape[1]
        return [slice(s, min(S, s + width)) for s in range(0, S, width)]

    def ku(self, u, cols):
        """K u for u (n, 3, s) of these samples."""
        d = torch.bmm(self.K, u[self.el].reshape(len(self.el), 9, -1)) * self.c[:, None, cols]
        return self._scatter(d, u.shape)

    def _scatter(self, d, shape):
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
        d = d.reshape(len(self.el), 3, 3, -1)
        for a in range(3):
            out.index_add_(0, self.el[:, a], d[:, a])
        return out

    def geo(self, u, ug, cols):
        """K(x + ug) u and the follower load of a unit pressure on x + ug."""
        out = torch.zeros_like(u)
        load = torch.zeros_like(u)
        D = self._D()
        for lo in range(0, len(self.el), 40000):
            el = self.el[lo:lo + 40000]
            B, area, nrm = self._strain(self.x[el].unsqueeze(-1) + ug[el])
            ue = u[el].reshape(len(el), 9, -1)
            sig = torch.einsum("pq,eqis,eis->eps", D, B, ue)
            d = torch.einsum("epis,eps->eis", B, sig) * (area * self.c[lo:lo + 40000, cols])[:, None]
            fe = (area / 3.0).unsqueeze(1) * nrm
            for a in range(3):
                out.index_add_(0, el[:, a], d[:, 3 * a:3 * a + 3])
                load.index_add_(0, el[:, a], fe)
        return out, load

    def start(self, dt, cols):
        """u_0 and u_{-1} of these samples (no load at the start)."""
        s = len(range(*cols.indices(self.c.shape[1])))
        u = self.u0.unsqueeze(-1).expand(-1, -1, s).contiguous()
        du = self.du0.unsqueeze(-1).expand(-1, -1, s)
        m = self.m[:, None, cols]
        acc = (-DAMP * m * du - self.ku(u, cols)) / m
        return u, u - dt * du + 0.5 * dt * dt * acc

    def step(self, u, up, r, dt, cols):
        """u_{n+1} from the force r = p f - K u."""
        g = 0.5 * dt * DAMP
        eta, w = dt * DAMP / (1 + g), dt * dt / (1 + g) / self.m[:, None, cols]
        v = (u - up) * (1 - eta) + w * r
        un = u + v
        un[: self.nb] = 0.0
        return un


def _rows(parts):
    """Samples side by side, (3n, S)."""
    u = torch.cat(parts, dim=-1)
    return u.reshape(3 * u.shape[0], -1)


def _exact_advance(case, seed):
    f = _fields(case, seed)
    wall, dt = _Wall(case, f), _dt(f)
    us, second = [], []
    interval = case.get("interval", 0) if case.get("path") == "geo" else 0
    for cols in wall.chunks(16 if interval else 32):
        u, up = wall.start(dt, cols)
        ug, count = torch.zeros_like(u), 0
        for p in f.pres:
            if interval:
                if count >= interval:
                    ug, count = u, 1
                else:
                    count += 1
                ku, load = wall.geo(u, ug, cols)
                r = p * load - ku
            else:
                r = p * wall.f.unsqueeze(-1) - wall.ku(u, cols)
            u, up = wall.step(u, up, r, dt, cols), u
        us.append(u)
        second.append(u - up if case["precision"] == 32 and not interval else up)
    return _rows(us), _rows(second)


def _exact_solve(case, seed):
    f = _fields(case, seed)
    wall, dt = _Wall(case, f), _dt(f)
    us, vs, norms = [], [], []
    for cols in wall.chunks(32):
        u, up = wall.start(dt, cols)
        for k in range(case["steps"]):
            p = P_REF * min(k / 100.0, 1.0)
            u, up = wall.step(u, up, p * wall.f.unsqueeze(-1) - wall.ku(u, cols), dt, cols), u
        v = u - up
        us.append(u)
        vs.append(v if case["precision"] == 32 else up)
        m = wall.m[:, cols]
        norms.append(torch.stack([u.square().sum((0, 1)), v.square().sum((0, 1)),
                                  (m * v.square().sum(1)).sum(0),
                                  torch.zeros(u.shape[-1], dtype=u.dtype, device=u.device)], 1))
    return {"u": _rows(us), "du": _rows(vs), "norms": torch.cat(norms).cpu()}


def _exact_gradient(case, seed):
    f = _fields(case, seed)
    wall, dt = _Wall(case, f), _dt(f)
    nodes, obs = _observations(case, f, dt)
    ids = wall.g2l[torch.from_numpy(nodes).cuda()]
    pres, every, T = _gradient_pressures(case), case["obs_every"], case["steps"]
    g = 0.5 * dt * DAMP
    eta = dt * DAMP / (1 + g)
    J, gE, gh = [], [], []
    for cols in wall.chunks(16):
        W = dt * dt / (1 + g) / wall.m[:, None, cols]
        u = torch.zeros(wall.n, 3, len(range(*cols.indices(case["S"]))), dtype=torch.float64,
                        device="cuda")
        hist, up, j = [u], u, 0.0
        for n in range(T):
            r = pres[n] * wall.f.unsqueeze(-1) - wall.ku(u, cols)
            u, up = wall.step(u, up, r, dt, cols), u
            hist.append(u)
            if (n + 1) % every == 0:
                j = j + (u[ids] - obs[(n + 1) // every - 1, :, :, cols]).square().sum((0, 1))
        zero = torch.zeros_like(u)

        def force(n, chi):
            if n % every == 0 and n > 0:
                chi = chi.clone()
                d = 2.0 * (hist[n][ids] - obs[n // every - 1, :, :, cols])
                chi.index_add_(0, ids, W[ids] * d)
            return chi

        gamma = torch.zeros(len(wall.el), u.shape[-1], dtype=torch.float64, device="cuda")
        G = torch.zeros(wall.n, u.shape[-1], dtype=torch.float64, device="cuda")
        x1, x2 = force(T, zero), zero
        for n in range(T - 1, -1, -1):
            un = hist[n]
            kun = torch.bmm(wall.K, un[wall.el].reshape(len(wall.el), 9, -1))
            gamma += (x1[wall.el].reshape(len(wall.el), 9, -1) * kun).sum(1)
            r = pres[n] * wall.f.unsqueeze(-1) - wall._scatter(kun * wall.c[:, None, cols], un.shape)
            G += (x1 * r).sum(1)
            chi = x1 + (1 - eta) * (x1 - x2) - W * wall.ku(x1, cols)
            chi[: wall.nb] = 0.0
            x1, x2 = force(n, chi), x1
        J.append(j)
        c, h = wall.c[:, cols], wall.h[:, cols]
        gE.append(-c * gamma)
        s = (G / wall.m[:, cols])[wall.el].sum(1)
        gh.append(-c * gamma - h * wall.alpha[:, None] * s)
    return {"J": torch.cat(J), "logE": torch.cat(gE, 1),
            "logh": torch.cat(gh, 1) if case["logh"] else None}


def _exact_stress(case, seed):
    f = _fields(case, seed)
    wall = _Wall(case, f)
    q = 1.0 - NU * NU
    ex, ey, ez, _ = wall._frame(wall.x[wall.el].unsqueeze(-1))
    B, _, _ = wall._strain(wall.x[wall.el].unsqueeze(-1))
    e = torch.einsum("epis,ei->ep", B, wall.u0[wall.el].reshape(-1, 9))
    s = e @ wall._D().T
    R = torch.stack([ex[..., 0], ey[..., 0], ez[..., 0]], 1)  # rows: local axes
    L = torch.zeros(len(e), 3, 3, dtype=torch.float64, device="cuda")
    L[:, 0, 0], L[:, 1, 1] = s[:, 0], s[:, 1]
    L[:, 0, 1] = L[:, 1, 0] = s[:, 2]
    L[:, 0, 2] = L[:, 2, 0] = s[:, 3]
    L[:, 1, 2] = L[:, 2, 1] = s[:, 4]
    G = torch.einsum("epi,epq,eqj->eij", R, L, R)
    unit = torch.stack([G[:, 0, 0], G[:, 1, 1], G[:, 0, 1], G[:, 0, 2], G[:, 1, 2]], 1)
    return f.E[:, :, None] * unit[:, None, :]


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        return [_exact_advance(dict(c, path="advance"), seed) for c in _batch_cases(case, seed)]
    if path == "gradient":
        return _exact_gradient(case, seed)
    if path == "stress":
        return _exact_stress(case, seed)
    if path == "solve":
        return _exact_solve(case, seed)
    u, prev = _exact_advance(case, seed)
    return {"u": u, "prev": prev}

