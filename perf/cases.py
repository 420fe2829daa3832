"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the Python binding of the C ABI (spoc_b200.api):

  rhs       one right-hand side on the caller's host arrays (Solver.cal_var),
            the call a Fortran driver makes four times per RK4 step;
  run       RK4 steps between two outputs on the caller's pinned host arrays
            (Solver.rk4_steps_host): the time loop of every simulation;
  ensemble  RK4 steps of several basins together (Ensemble.steps), states set
            before and read after;
  gradient  cost and gradient of an assimilation window (Solver.bwd_window).

Meshes are jittered square basins with the cell size, physics and rules of the
benchmark configurations (spoc_b200/workloads.py); the state is eight seeded
geostrophic eddies.  Regridding is left out: the adaptive driver calls it once
in tens of steps, where the steps take nearly all of the time.
"""
import numpy as np
import torch

from spoc_b200 import api, workloads

# degree -> triangle and edge rule, as the configurations pair them
RULES = {3: (12, 4), 4: (25, 5), 5: (27, 6), 6: (33, 7), 7: (42, 9)}
# fraction of the checkcfl step a run takes: that step is at the edge of
# stability from degree 5 on for some jittered meshes
DT_SCALE = {3: 1.0, 4: 1.0, 5: 0.5, 6: 0.5, 7: 0.25}
FIELDS = ("u", "v", "h")
# operations of the contractions (3 nm^2 ne per right-hand side, a quarter for
# the mixed form) that no drawn case exceeds: just under the largest listed one
MOST = 8.0e9


def listed():
    return [
        # the drop-in call on a small basin, 45-strided arrays as the Fortran
        # driver holds them: launch and copy latency
        dict(name="rhs_fs4_small", kind="rhs", variant="fs", nc=4, n=6, ld=45, precision="fp64", wind=False),
        # a short run of a small basin (a test set-up, a laptop-sized problem)
        dict(name="run_ns3_small", kind="run", variant="ns", nc=3, n=13, steps=10, precision="fp64", wind=False),
        # the linear benchmark configuration (2048 triangles, degree 3)
        dict(name="run_lin3", kind="run", variant="lin", nc=3, n=32, steps=100, precision="fp64", wind=False),
        # a linear run too large for one pass of the GPU, an odd size
        dict(name="run_lin5_mid", kind="run", variant="lin", nc=5, n=73, steps=30, precision="fp64", wind=False),
        # a mid-sized wind-driven basin of odd size
        dict(name="run_fs5_wind", kind="run", variant="fs", nc=5, n=45, steps=30, precision="fp64", wind=True),
        # the free-slip headline configuration (32768 triangles, degree 6)
        dict(name="run_fs6", kind="run", variant="fs", nc=6, n=128, steps=20, precision="fp64", wind=False),
        # the inviscid configuration (131072 triangles, degree 7)
        dict(name="run_inv7", kind="run", variant="inv", nc=7, n=256, steps=4, precision="fp64", wind=False),
        # the no-slip configuration's forward model (32768 triangles, degree 4)
        dict(name="run_ns4", kind="run", variant="ns", nc=4, n=128, steps=20, precision="fp64", wind=False),
        # the two large configurations in the mixed-precision form
        dict(name="run_fs6_mixed", kind="run", variant="fs", nc=6, n=128, steps=40, precision="mixed", wind=False),
        dict(name="run_inv7_mixed", kind="run", variant="inv", nc=7, n=256, steps=10, precision="mixed", wind=False),
        # an ensemble of basins of degrees 3 to 6
        dict(name="ensemble_fs", kind="ensemble", members=12, nc=3, n=72, steps=40),
        # the assimilation window of the no-slip configuration, shortened
        dict(name="gradient_ns4", kind="gradient", variant="ns", nc=4, n=128, steps=20, snaps=5, nobs=500),
    ]


def draw(rng):
    kind = rng.choice(["rhs", "run", "run", "run", "run", "ensemble", "gradient"])
    nc = rng.randint(3, 7)
    n = int(round(4 * 64 ** rng.random()))  # 4 .. 256 cells a side, by logarithm
    if kind == "ensemble":
        c = dict(kind=kind, members=rng.randint(2, 12), nc=rng.randint(3, 6), n=min(n, 72),
                 steps=rng.randint(5, 40))
    elif kind == "gradient":
        c = dict(kind=kind, variant=rng.choice(["lin", "fs", "ns", "inv"]), nc=nc, n=min(n, 128),
                 steps=rng.randint(4, 20), snaps=rng.randint(2, 6), nobs=rng.randint(20, 500))
    else:
        variant = rng.choice(["lin", "fs", "fs", "ns", "inv"])
        precision = rng.choice(["fp64", "fp64", "fp64", "mixed"])
        c = dict(kind=kind, variant=variant, nc=nc, n=n, precision=precision, wind=rng.random() < 0.3)
        if kind == "rhs":
            c["ld"] = rng.choice([_nm(nc), 45])
        else:
            c["steps"] = int(round(100 ** rng.random()))
    while _cost(c) > MOST and c["n"] > 4:
        if c.get("steps", 1) > 4:
            c["steps"] = max(4, c["steps"] // 2)
        else:
            c["n"] = c["n"] * 9 // 10
    return c


# ---------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------

def _nm(nc):
    return (nc + 1) * (nc + 2) // 2


def _parts(case):
    """(variant, degree, cells a side) of each basin of a case."""
    if case["kind"] != "ensemble":
        return [(case["variant"], case["nc"], case["n"])]
    # degrees 3 to 6 from nc on; sizes from n down to about two thirds of it
    return [("fs", 3 + (case["nc"] - 3 + i) % 4, max(4, case["n"] - (i * 5 % 26) * case["n"] // 72))
            for i in range(case["members"])]


def _rhs_count(case):
    k = 4 * case.get("steps", 1) if case["kind"] != "rhs" else 1
    return k * (4 if case["kind"] == "gradient" else 1)  # reverse sweep: about three forward ones


def _cost(case):
    per = sum(3 * _nm(nc) * 2 * n * n * _nm(nc) for _, nc, n in _parts(case))
    return per * _rhs_count(case) * (0.25 if case.get("precision") == "mixed" or case["kind"] == "ensemble" else 1)


def work(case):
    flops = bytes_ = 0.0
    for variant, nc, n in _parts(case):
        nm, ne = _nm(nc), 2 * n * n
        q, g = RULES[nc]
        nf = 3 * ne / 2
        if variant == "lin":
            macs = ne * (9 * nm * nm + 12 * nm * g) + nf * 3 * 2 * nm * g
            static = 0
        else:  # q-phase, quadrature points, tendencies; traces once per face
            macs = ne * (25 * nm * nm + 30 * nm * g + 17 * nm * q) + nf * 8 * 2 * nm * g
            static = 4  # hb, fc, w0, z0
        flops += 2.0 * macs * _rhs_count(case)
        # state in, state (or tendency, gradient) out, fixed fields, mesh
        bytes_ += ne * (nm * 8 * (3 + 3 + static) + 130)
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _problem(case, part, seed, member=0):
    variant, nc, n = part
    ng, ngf = RULES[nc]
    base = workloads.Config("case", variant, nc, ng, ngf, 128, jitter=0.2, beta=2.0e-11, ic="gauss8",
                            mu0=0.0 if variant in ("lin", "inv") else 100.0,
                            mb0=0.0 if variant in ("lin", "inv") else 1.0e-3,
                            seed=int(seed) * 64 + member, dt_scale=DT_SCALE[nc])
    p = workloads.build_problem(workloads.small(base, n))
    if case.get("wind"):  # a double-gyre wind stress on the element means
        y = p.mesh.ygr[p.mesh.inn - 1].mean(axis=1) / p.cfg.length
        rng = np.random.default_rng(seed)
        p.w0[:, 0] = -1.0e-4 * rng.uniform(0.5, 1.5) * np.cos(2.0 * np.pi * y)
        p.z0[:, 0] = 1.0e-5 * rng.uniform(0.5, 1.5) * np.sin(2.0 * np.pi * y)
    return p


def _observations(case, p, seed):
    """Eta observed at points of random elements, at half and at the end of
    the window: (element, basis values, steps, values)."""
    rng = np.random.default_rng(seed + 77)
    nobs = case["nobs"]
    elem = rng.integers(1, p.mesh.ne + 1, nobs).astype(np.int32)
    a, b = rng.random(nobs), rng.random(nobs)
    a, b = np.where(a + b > 1, 1 - a, a), np.where(a + b > 1, 1 - b, b)
    basis = workloads.basis_at(p.cfg.nc, 2 * a - 1, 2 * b - 1)
    steps = np.array(sorted({max(1, case["steps"] // 2), case["steps"]}), dtype=np.int32)
    now = np.sum(p.h[elem - 1] * basis, axis=1)
    return elem, basis, steps, now + 0.05 * rng.normal(size=(steps.size, nobs))


def prepare(case, seed):
    parts = _parts(case)
    problems = [_problem(case, part, seed, i) for i, part in enumerate(parts)]
    precision = "mixed" if case["kind"] == "ensemble" else case.get("precision", "fp64")
    solvers = [workloads.make_solver(p, precision) for p in problems]
    state = {"case": case, "p": problems, "s": solvers}
    p, s = problems[0], solvers[0]
    if case["kind"] == "rhs":
        state["x"] = [np.zeros((p.mesh.ne, case["ld"])) for _ in FIELDS]
        for a, f in zip(state["x"], FIELDS):
            a[:, :p.T.nm] = getattr(p, f)
    elif case["kind"] == "run":
        state["x"] = [torch.from_numpy(getattr(p, f)).pin_memory() for f in FIELDS]
        state["y"] = [torch.empty_like(t).pin_memory() for t in state["x"]]
        state["host"] = [t.numpy() for t in state["y"]]
    elif case["kind"] == "ensemble":
        state["ens"] = api.Ensemble(solvers)
        state["ens"].configure(4, 2)
        state["dt"] = [q.dt for q in problems]
    else:
        s.set_observations(*_observations(case, p, seed))
        state["x"] = [p.u, p.v, p.h]
    return state


def run(state):
    case, p, s = state["case"], state["p"][0], state["s"][0]
    if case["kind"] == "rhs":
        return s.cal_var(*state["x"])
    if case["kind"] == "run":
        for y, x in zip(state["y"], state["x"]):
            y.copy_(x)
        s.rk4_steps_host(*state["host"], p.dt, case["steps"])
        return state["y"]
    if case["kind"] == "ensemble":
        for q, m in zip(state["p"], state["s"]):
            m.set_state(q.u, q.v, q.h)
        state["ens"].steps(state["dt"], case["steps"])
        return [m.get_state() for m in state["s"]]
    cost, grad = s.bwd_window(state["x"], p.dt, case["steps"], case["snaps"])
    return {"cost": cost, "gradient": grad}


# ---------------------------------------------------------------------------
# the same outputs in plain torch, 64 bits
# ---------------------------------------------------------------------------

def _legendre(nc, x):
    """P_0 .. P_nc and their derivatives at x, by numpy's Legendre series."""
    from numpy.polynomial import legendre as L
    eye = np.eye(nc + 1)
    val = np.stack([L.legval(x, c) for c in eye])
    der = np.stack([L.legval(x, L.legder(c)) for c in eye])
    return val, der


class _Exact:
    """The discontinuous-Galerkin right-hand side of one basin, every field
    (ne, nm): basis P_k1(x) P_k2(y), k1 + k2 <= nc, k2 fastest."""

    def __init__(self, p):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.variant = p, p.cfg.variant
        nc, m = p.cfg.nc, p.mesh
        wi, xi, yi, wif, tif = api.quadrature(p.cfg.ng, p.cfg.ngf)
        modes = [(a, b) for a in range(nc + 1) for b in range(nc + 1 - a)]
        k1, k2 = np.array(modes).T

        def phi(x, y):
            (px, dx), (py, dy) = _legendre(nc, x), _legendre(nc, y)
            return px[k1] * py[k2], dx[k1] * py[k2], px[k1] * dy[k2]
        f, fx, fy = phi(xi, yi)
        t = self._t
        self.P, self.W = t(f), t(wi)
        self.M = t((f * wi) @ f.T)
        self.AX, self.AY = t((f * wi) @ fx.T), t((f * wi) @ fy.T)  # [j, i] = int phi_j d phi_i
        sides = [(tif, -np.ones_like(tif)), (-tif, tif), (-np.ones_like(tif), -tif)]
        self.TR = t(np.concatenate([phi(x, y)[0] for x, y in sides], axis=1))  # nm x 3G
        self.G, self.wif = tif.size, t(wif)
        # sub-basis that vanishes on y = -1: P_k1 (P_k2 - (-1)^k2 P_0)
        R = np.zeros((len(modes), len(modes) - nc - 1))
        for c, j in enumerate(np.nonzero(k2 > 0)[0]):
            R[j, c] = 1.0
            R[modes.index((k1[j], 0)), c] = -((-1.0) ** k2[j])
        self.R = t(R)
        self.U, self.UR = torch.linalg.cholesky(self.M), torch.linalg.cholesky(self.R.T @ self.M @ self.R)
        i = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev).long()  # noqa: E731
        self.t1, self.t2 = i(m.tseg[:, 0] - 1), i(m.tseg[:, 1] - 1)
        self.s1, self.s2 = i(m.ssit[:, 0] - 1), i(np.maximum(m.ssit[:, 1], 1) - 1)
        self.inner = (self.t2 >= 0)[:, None]
        self.itm, self.sgn = i(m.itm - 1), t(m.its)
        self.nx, self.ny = t(m.norm[:, :1]), t(m.norm[:, 1:])
        ax, bx, ay, by, self.di = (t(m.vect[:, k:k + 1]) for k in range(5))
        self.ax, self.bx, self.ay, self.by = (c * self.di for c in (ax, bx, ay, by))
        self.wall = torch.from_numpy(m.bdl != 0).to(self.dev)[:, None]
        self.cx, self.cy = t(m.normt[:, :1]), t(m.normt[:, 1:])
        self.fc, self.hb, self.w0, self.z0 = (t(a) for a in (p.fc, p.hb, p.w0, p.z0))

    def _t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(self.dev)

    def flux(self, a):
        """Central face values, (nf, G)."""
        tr = (a @ self.TR).view(-1, 3, self.G)
        one, two = tr[self.t1, self.s1], tr[self.t2.clamp(min=0), self.s2].flip(-1)
        return torch.where(self.inner, 0.5 * (one + two), one)

    def weak(self, fx, fy, bx, by):
        """- int F . grad phi + boundary, over det: volume fields fx, fy and
        their face values bx, by (either pair may be None)."""
        out = 0.0
        for f, cx, cy in ((fx, -self.by, self.ay), (fy, self.bx, -self.ax)):
            if f is not None:
                out = out + cx * (f @ self.AX) + cy * (f @ self.AY)
        b = (bx * self.nx if bx is not None else 0.0) + (by * self.ny if by is not None else 0.0)
        e = (0.5 * self.wif * b)[self.itm]
        e = torch.where(self.sgn[..., None] > 0, e, e.flip(-1)) * self.sgn[..., None]
        return out + self.di * (e.reshape(e.shape[0], -1) @ self.TR.T)

    def solve(self, b):
        return torch.cholesky_solve(b.T, self.U).T

    def solve0(self, b):
        return torch.cholesky_solve((b @ self.R).T, self.UR).T @ self.R.T

    def rot(self, a, b):
        return a * self.cx + b * self.cy, a * self.cy - b * self.cx

    def solve_uv(self, a, b):
        """Mass solve of a vector, strongly constrained on wall elements."""
        fa, fb = self.solve(a), self.solve(b)
        if self.variant == "ns":
            wa, wb = self.solve0(a), self.solve0(b)
        else:
            n, t = self.rot(a, b)
            wa, wb = self.rot(self.solve0(n), self.solve(t))
        return torch.where(self.wall, wa, fa), torch.where(self.wall, wb, fb)

    def rhs(self, u, v, h):
        c = self.p.cfg
        if self.variant == "lin":
            hh0, f = float(self.p.hb[0, 0]), -c.g0 * h
            bf, bu, bv = self.flux(f), self.flux(u) * hh0, self.flux(v) * hh0
            du, dv = self.solve_uv(self.weak(f, None, bf, None), self.weak(None, f, None, bf))
            return du, dv, self.solve(-self.weak(u * hh0, v * hh0, bu, bv))
        bu, bv = self.flux(u), self.flux(v)
        q = [self.weak(u, None, bu, None), self.weak(None, u, None, bu),
             self.weak(v, None, bv, None), self.weak(None, v, None, bv)]
        s = [self.solve(a) for a in q]
        if self.variant == "fs":  # the normal derivative of the tangential velocity vanishes
            gnx, gtx = self.rot(q[0], q[2])
            gny, gty = self.rot(q[1], q[3])
            gnn, gnt = self.rot(gnx, gny)
            gtn, gtt = self.rot(gtx, gty)
            gnn, gnt, gtt, gtn = self.solve(gnn), self.solve(gnt), self.solve(gtt), self.solve0(gtn)
            gnx, gny = self.rot(gnn, gnt)
            gtx, gty = self.rot(gtn, gtt)
            w = [*self.rot(gnx, gtx), *self.rot(gny, gty)]
            s = [torch.where(self.wall, a, b) for a, b in zip((w[0], w[2], w[1], w[3]), s)]
        qxx, qxy, qyx, qyy = s
        pt = [a @ self.P for a in (u, v, qxx, qxy - self.fc, qyx + self.fc, qyy, h + self.hb,
                                   self.w0 - c.mb0 * u, self.z0 - c.mb0 * v)]
        load = lambda a: (a * self.W) @ self.P.T  # noqa: E731
        gx = load(pt[7] / pt[6] - pt[0] * pt[2] - pt[1] * pt[3])
        gy = load(pt[8] / pt[6] - pt[0] * pt[4] - pt[1] * pt[5])
        uh, vh = self.solve_uv(load(pt[0] * pt[6]), load(pt[1] * pt[6]))
        f = [c.mu0 * qxx - c.g0 * h, c.mu0 * qxy, c.mu0 * qyx, c.mu0 * qyy - c.g0 * h]
        b = [self.flux(a) for a in f]
        du, dv = self.solve_uv(gx + self.weak(f[0], f[1], b[0], b[1]), gy + self.weak(f[2], f[3], b[2], b[3]))
        return du, dv, self.solve(-self.weak(uh, vh, self.flux(uh), self.flux(vh)))

    def step(self, u, v, h):
        dt, x = self.p.dt, (u, v, h)
        k = [self.rhs(*x)]
        for w in (0.5, 0.5, 1.0):
            k.append(self.rhs(*[a + w * dt * d for a, d in zip(x, k[-1])]))
        return tuple(a + dt / 6.0 * (p + 2 * q + 2 * r + s) for a, p, q, r, s in zip(x, *k))

    def state(self):
        return tuple(self._t(getattr(self.p, f)) for f in FIELDS)


def _gradient(case, e, seed):
    from torch.utils.checkpoint import checkpoint
    elem, basis, steps, values = _observations(case, e.p, seed)
    at, phi = torch.from_numpy(elem - 1).long().to(e.dev), e._t(basis)
    x0 = [a.requires_grad_() for a in e.state()]
    x, cost = tuple(x0), 0.0
    for k in range(1, case["steps"] + 1):
        x = checkpoint(e.step, *x, use_reentrant=False)
        for i in np.nonzero(steps == k)[0]:
            cost = cost + 0.5 * ((x[2][at] * phi).sum(1) - e._t(values[i])).square().sum()
    cost.backward()
    return {"cost": float(cost.detach()), "gradient": tuple(a.grad.cpu().numpy() for a in x0)}


def exact(case, seed):
    if case["kind"] == "gradient":
        return _gradient(case, _Exact(_problem(case, _parts(case)[0], seed)), seed)
    out = []
    with torch.no_grad():
        for i, part in enumerate(_parts(case)):
            e = _Exact(_problem(case, part, seed, i))
            x = e.state()
            if case["kind"] == "rhs":
                x = tuple(torch.nn.functional.pad(a, (0, case["ld"] - a.shape[1])) for a in e.rhs(*x))
            else:
                for _ in range(case["steps"]):
                    x = e.step(*x)
            out.append(tuple(a.cpu().numpy() for a in x))
    return out if case["kind"] == "ensemble" else out[0] if case["kind"] == "rhs" else list(out[0])
