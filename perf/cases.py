"""Performance cases of the Richards Newton-Krylov path: what a user's program
has the library do through its public entry points, over the sizes it is used
at.  Kinds of case:

``step``      one implicit timestep of a device-resident problem: set the old
              pressure, ``RichardsGPU.advance``, read the new pressure into a
              device buffer (the step body of a simulation loop).
``solve``     one timestep through the drop-in boundary, as ParFlow's nonlinear
              solver module calls it: ``pfgpu_newton_solve_sat`` with p, p_old
              and s_old in pinned host memory, p and s back in host memory.
``residual``  F(p) through ``pfgpu_nl_function_eval`` on device buffers.
``matvec``    J(p) x through ``pfgpu_jacobian_matvec`` on device buffers
              (assembles J at p, then multiplies: what KINSOL's first product
              of an iteration costs).
``ensemble``  one timestep of several problems of uneven size at once
              (``ensemble_advance``).
``adjoint``   a recorded trajectory of a few steps and the gradient of an
              observation misfit with respect to ln K, alpha and n.

Every problem is made from the seed: correlated lognormal permeability,
van Genuchten parameters, a smoothly varying water table and rain.  Sizes and
physics are those of ``parflow_b200.configs`` (the 64x64x32 box, the 512x512x50
heterogeneous box, the 256x256x20 hillslope, the uneven ensemble, the adjoint
box) and of the repository's tests (small and odd grids).
"""

import ctypes as C
import math

import numpy as np
import torch

from parflow_b200.problem import (BC, BC_DIRICHLET, BC_FLUX, BC_OVERLAND_KIN, RichardsProblem,
                                  SolverSettings)
from parflow_b200.solver import RichardsGPU, ensemble_advance

DEV = "cuda"
MEMBERS = ((64, 16), (96, 24), (128, 32), (64, 40), (192, 16), (96, 32), (128, 24), (192, 40))


def listed():
    return [
        # a unit-test or teaching column of a few hundred cells: nothing but latency
        dict(name="step tiny fp64", kind="step", physics="box", nx=12, ny=10, nz=8,
             precision="fp64"),
        # the plain box of the configurations, the library's default precision
        dict(name="step box fp64", kind="step", physics="box", nx=64, ny=64, nz=32,
             precision="fp64"),
        # a catchment cut to its bounding box: no size is a multiple of anything
        dict(name="step ragged mixed16", kind="step", physics="hetero", nx=197, ny=123, nz=37,
             precision="mixed16"),
        # hillslope with overland flow on a terrain-following grid
        dict(name="step hillslope mixed16", kind="step", physics="overland", nx=256, ny=256,
             nz=20, precision="mixed16"),
        # a regional model with the FP32 multigrid
        dict(name="step regional mixed", kind="step", physics="hetero", nx=256, ny=256, nz=50,
             precision="mixed"),
        # the benchmark's heterogeneous box in the fast form and in the default precision
        dict(name="step large mixed16", kind="step", physics="hetero", nx=512, ny=512, nz=50,
             precision="mixed16"),
        dict(name="step large fp64", kind="step", physics="hetero", nx=512, ny=512, nz=50,
             precision="fp64"),
        # the same solver behind ParFlow's module: host vectors in and out
        dict(name="solve host mixed16", kind="solve", physics="hetero", nx=192, ny=160, nz=40,
             precision="mixed16"),
        # parameter uncertainty: members of uneven size, a step of all at once
        dict(name="ensemble 8 mixed16", kind="ensemble", members=8, scale=1.0,
             precision="mixed16"),
        # calibration: forward trajectory and gradient
        dict(name="adjoint fp64", kind="adjoint", physics="box", nx=96, ny=96, nz=32, steps=3,
             precision="fp64"),
        # operators, for a caller with its own nonlinear or Krylov solver
        dict(name="residual fp64", kind="residual", physics="hetero", nx=512, ny=512, nz=50,
             precision="fp64"),
        dict(name="matvec mixed", kind="matvec", physics="hetero", nx=250, ny=310, nz=45,
             precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "solve", "residual", "matvec", "ensemble",
                       "adjoint"])
    precision = rng.choice(["fp64", "mixed", "mixed16", "mixed16"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 8), scale=round(rng.uniform(0.4, 1.0), 3),
                    precision=precision)
    if kind == "adjoint":
        return dict(kind=kind, physics="box", nx=_log_int(rng, 16, 96), ny=_log_int(rng, 16, 96),
                    nz=rng.randint(8, 32), steps=rng.randint(1, 3), precision="fp64")
    hi = {"step": 512, "solve": 192, "residual": 512, "matvec": 400}[kind]
    physics = rng.choice(["box", "hetero", "overland"])
    nz = rng.randint(8, 20) if physics == "overland" else rng.randint(8, 50)
    return dict(kind=kind, physics=physics, nx=_log_int(rng, 10, hi), ny=_log_int(rng, 10, hi),
                nz=nz, precision=precision)


# ---- inputs ------------------------------------------------------------------
def _field(shape, corr, gen):
    """Correlated Gaussian field (mean 0, std 1), correlation lengths in cells."""
    k2 = 0.0
    for a, (n, c) in enumerate(zip(shape, corr)):
        f = torch.fft.rfftfreq(n) if a == len(shape) - 1 else torch.fft.fftfreq(n)
        f = f.to(DEV, torch.float64) * (2.0 * math.pi * c)
        k2 = k2 + (f * f).reshape([-1 if b == a else 1 for b in range(len(shape))])
    w = torch.randn(shape, generator=gen, device=DEV, dtype=torch.float64)
    g = torch.fft.irfftn(torch.fft.rfftn(w) / (1.0 + k2), s=shape)
    g = g - g.mean()
    return g / g.std().clamp_min(1e-30)


def _problem(physics, nx, ny, nz, seed, steps=1):
    """(problem, its fields as device tensors)."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1000003 * (seed % 1000003) + 17)
    u = torch.rand(8, generator=gen, device=DEV, dtype=torch.float64).tolist()
    shape = (nz, ny, nx)
    solver = SolverSettings(max_iter=40, residual_tol=1e-12 if steps > 1 else 1e-9)
    p = RichardsProblem(nx=nx, ny=ny, nz=nz, dx=1.0, dy=1.0, dz=0.5, nsteps=steps, solver=solver,
                        dt=0.1, name=physics)
    flat = {f: BC(BC_FLUX, (0.0,)) for f in ("x_lower", "x_upper", "y_lower", "y_upper")}
    if physics == "overland":
        p.dx = p.dy = 10.0
        p.dz, p.dt = 0.2, 0.25
        top = (torch.arange(nz, device=DEV) >= nz // 2).reshape(nz, 1, 1)
        layer = lambda a, b: torch.where(top, a, b).expand(shape).to(torch.float64)
        k = layer(0.1, 0.005) * torch.exp(0.2 * _field(shape, (2.0, 8.0, 8.0), gen))
        alpha, n = layer(3.5, 1.0), layer(2.0, 1.8)
        p.terrain_following = True
        slopes = []
        for _ in range(2):
            g = _field((ny, nx), (8.0, 8.0), gen)
            mag = 1e-4 + (5e-2 - 1e-4) * (g.abs() / 3.0).clamp(0.0, 1.0)
            slopes.append(torch.where(g >= 0, mag, -mag).cpu().numpy())
        p.slope_x, p.slope_y = slopes
        p.bc = dict(flat, z_lower=BC(BC_FLUX, (0.0,)),
                    z_upper=BC(BC_OVERLAND_KIN, (-0.01 - 0.005 * u[0], 0.0), lengths=(8, 8)))
        table = nz * p.dz - (0.6 + 0.4 * u[1])
        swing = 0.1
    else:
        if physics == "hetero":  # per-cell alpha, anisotropic correlation
            p.dt = 0.05
            k = 0.01 * torch.exp(1.5 * _field(shape, (4.0, 32.0, 32.0), gen))
            alpha = 2.0 * (1.0 + 0.4 * (torch.rand(shape, generator=gen, device=DEV,
                                                   dtype=torch.float64) - 0.5))
            n = torch.full(shape, 3.0, device=DEV, dtype=torch.float64)
            flux = -0.05
        elif physics == "member":  # a realisation with its own soil
            k = 0.01 * torch.exp((0.5 + 1.0 * u[2]) * _field(shape, (8.0, 8.0, 8.0), gen))
            alpha, n = 0.5 + 2.5 * u[3], 1.8 + 1.2 * u[4]
            flux = -0.1 + 0.08 * u[5]
        else:
            k = 0.01 * torch.exp(_field(shape, (8.0, 8.0, 8.0), gen))
            alpha, n = 2.0, 3.0
            flux = -0.05 - 0.02 * u[0]
        p.bc = dict(flat, z_lower=BC(BC_DIRICHLET, (2.0,), ref_patch="z_lower"),
                    z_upper=BC(BC_FLUX, (flux,)))
        table, swing = 2.0, 0.1
    host = lambda a: a.cpu().numpy() if torch.is_tensor(a) else a
    p.perm, p.vg_alpha, p.vg_n = host(k), host(alpha), host(n)
    z = (torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5) * p.dz
    level = table + swing * _field((ny, nx), (8.0, 8.0), gen).clamp(-2.0, 2.0)
    p0 = level.reshape(1, ny, nx) - z.reshape(nz, 1, 1)
    return p, dict(k=k, alpha=alpha, n=n, p0=p0), gen


def _pad(a):
    """Interior cells in ParFlow's ghost-framed layout."""
    return torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1)).contiguous()


def _member_problems(case, seed):
    out = []
    for m, (nxy, nz) in enumerate(MEMBERS[: case["members"]]):
        s = case["scale"]
        nx, ny, nz = (max(8, int(round(v * s))) for v in (nxy, nxy, nz))
        out.append(_problem("member", nx, ny, nz, seed * 31 + m))
    return out


def _observations(case, seed):
    rng = np.random.default_rng(seed)
    ncell = case["nx"] * case["ny"] * case["nz"]
    cells = np.sort(rng.choice(ncell, size=min(256, ncell // 4), replace=False)).astype(np.int64)
    steps = np.arange(1, case["steps"] + 1, dtype=np.int32)
    return steps, cells, 0.5 * rng.standard_normal((len(steps), len(cells)))


def _operands(case, seed):
    """Problem, fields, and an iterate p near p_old and a direction x."""
    prob, f, gen = _problem(case["physics"], case["nx"], case["ny"], case["nz"], seed)
    f["p"] = f["p0"] + 0.05 * _field(prob.shape, (2.0, 4.0, 4.0), gen)
    f["x"] = torch.randn(prob.shape, generator=gen, device=DEV, dtype=torch.float64)
    f["s_old"] = _vg(f["p0"], f["alpha"], f["n"])[1]
    return prob, f


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        st = []
        for prob, f, _ in _member_problems(case, seed):
            st.append((RichardsGPU(prob, precision=case["precision"]), _pad(f["p0"]),
                       torch.zeros_like(_pad(f["p0"]))))
        return dict(kind=kind, members=st)
    if kind in ("step", "adjoint"):
        prob, f, _ = _problem(case["physics"], case["nx"], case["ny"], case["nz"], seed,
                              case.get("steps", 1))
        p0 = _pad(f["p0"])
        s = dict(kind=kind, g=RichardsGPU(prob, precision=case["precision"]), p0=p0, dt=prob.dt,
                 out=torch.zeros_like(p0))
        if kind == "adjoint":
            s["obs"] = _observations(case, seed)
        return s
    prob, f = _operands(case, seed)
    g = RichardsGPU(prob, precision=case["precision"])
    s = dict(kind=kind, g=g, dt=prob.dt)
    if kind == "solve":
        pin = lambda a: _pad(a).cpu().pin_memory()
        s.update(p0=pin(f["p0"]), s_old=pin(f["s_old"]))
        s.update(p=s["p0"].clone().pin_memory(), s=torch.zeros_like(s["p0"]).pin_memory())
        return s
    for q in ("p", "p0", "s_old", "x"):
        s[q] = _pad(f[q])
    s["out"] = torch.zeros_like(s["p"])
    return s


def _at(t):
    return C.c_void_p(t.data_ptr())


def _ok(rc):
    if rc != 0:
        raise RuntimeError("the library returned %d" % rc)


def run(s):
    kind = s["kind"]
    if kind == "ensemble":
        for g, p0, _ in s["members"]:
            g.set_pressure(p0)
        ensemble_advance([m[0] for m in s["members"]], 1)
        return [g.get_pressure(out) for g, _, out in s["members"]]
    g, dt = s["g"], s["dt"]
    if kind == "step":
        g.set_pressure(s["p0"])
        g.advance(1, dt)
        return g.get_pressure(s["out"])
    if kind == "adjoint":
        steps, cells, obs = s["obs"]
        g.set_pressure(s["p0"])
        g.adjoint_record(len(steps))
        g.advance(len(steps), dt)
        misfit, g_lnk, g_alpha, g_n = g.adjoint_gradient(steps, cells, obs)
        return dict(p=g.get_pressure(s["out"]), misfit=misfit, lnk=g_lnk, alpha=g_alpha, n=g_n)
    if kind == "solve":
        s["p"].copy_(s["p0"])  # the initial guess is the old pressure, in its own vector
        _ok(g.lib.pfgpu_newton_solve_sat(g.h, _at(s["p0"]), _at(s["s_old"]), dt, _at(s["p"]),
                                         _at(s["s"]), None))
        return s["p"], s["s"]
    if kind == "residual":
        _ok(g.lib.pfgpu_nl_function_eval(g.h, _at(s["p"]), _at(s["p0"]), _at(s["s_old"]), dt,
                                         _at(s["out"])))
    else:
        _ok(g.lib.pfgpu_jacobian_matvec(g.h, _at(s["p"]), dt, _at(s["x"]), _at(s["out"])))
    return s["out"]


# ---- what a pass cannot do without ---------------------------------------------
def _cells(case):
    if case["kind"] == "ensemble":
        n = 0
        for nxy, nz in MEMBERS[: case["members"]]:
            nx, nz = (max(8, int(round(v * case["scale"]))) for v in (nxy, nz))
            n += nx * nx * nz
        return n
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Inputs read once, outputs written once; for the solves the arithmetic
    of four Newton iterations (residual, Jacobian row, two V-cycles of 13
    smoothing-like passes over twice the cells) at the flops of a plain
    evaluation."""
    n = _cells(case)
    soil = 8 * (2 if case.get("physics") in ("hetero", "overland") else 1)
    if case.get("physics") == "overland":
        soil += 8
    residual, jacobian, vcycle = 250, 300, 2 * 13 * 13
    newton = 4 * (residual + jacobian + 2 * vcycle)
    kind = case["kind"]
    if kind == "residual":  # p, p_old, s_old, soil -> F
        return dict(bytes=n * (32 + soil), flops=n * residual)
    if kind == "matvec":    # p, x, soil -> y
        return dict(bytes=n * (24 + soil), flops=n * (jacobian + 13))
    if kind == "solve":     # p, p_old, s_old, soil -> p, s
        return dict(bytes=n * (40 + soil), flops=n * newton)
    if kind == "adjoint":   # p0, soil -> p, three gradients
        return dict(bytes=n * (40 + soil), flops=n * case["steps"] * 2 * newton)
    return dict(bytes=n * (16 + soil), flops=n * newton)


def tolerance(case):
    """The operators are FP64 sums (FP32 face terms in the mixed Jacobian).
    A solve ends at max |F| <= 1e-9, so two correct ones differ by what that
    leaves in p; the reduced-precision preconditioners move the last iterate
    within it."""
    kind, fp64 = case["kind"], case["precision"] == "fp64"
    if kind == "residual" or (kind == "matvec" and fp64):
        # measured against the plain form below: up to 2e-15
        return {"rel": 1e-13, "max": 1e-11}
    if kind == "matvec":  # measured: 2.6e-8
        return {"rel": 1e-7, "max": 1e-5}
    # measured: up to 6e-11 (fp64), the limits of the repository's parity tests
    return {"rel": 1e-9, "max": 1e-7} if fp64 else {"rel": 1e-8, "max": 1e-6}


# ---- the same in plain torch, 64 bits ------------------------------------------
def _vg(p, alpha, n, s_res=0.1, s_sat=1.0):
    """van Genuchten (kr, S) at pressure p."""
    wet = p >= 0
    ah = torch.where(wet, torch.ones_like(p), -alpha * p)
    m = 1.0 - 1.0 / n
    d = 1.0 + ah ** n
    kr = (1.0 - ah ** (n - 1.0) / d ** m) ** 2 / d ** (0.5 * m)
    s = (s_sat - s_res) / d ** m + s_res
    return torch.where(wet, torch.ones_like(p), kr), torch.where(wet, s_sat * torch.ones_like(p), s)


class _Exact:
    """F(p), its Jacobian and one implicit step of a problem of this file."""

    def __init__(self, prob, f):
        self.prob, self.k, self.alpha, self.n = prob, f["k"], f["alpha"], f["n"]
        t = lambda a: torch.as_tensor(np.asarray(a), device=DEV, dtype=torch.float64)
        if prob.terrain_following:
            self.sx, self.sy = t(prob.slope_x), t(prob.slope_y)
            mean = lambda a, ax: 0.5 * (a.narrow(ax, 0, a.shape[ax] - 1)
                                        + a.narrow(ax, 1, a.shape[ax] - 1))
            self.grav = [(mean(torch.sin(torch.atan(s)), ax), mean(torch.cos(torch.atan(s)), ax))
                         for s, ax in ((self.sx, 1), (self.sy, 0))]
        else:
            self.grav = [(0.0, 1.0), (0.0, 1.0)]
        nz, ny, nx = prob.shape
        a = [torch.arange(v, device=DEV) for v in (nz, ny, nx)]
        self.colour = (a[2].reshape(1, 1, -1) + 2 * a[1].reshape(1, -1, 1)
                       + 3 * a[0].reshape(-1, 1, 1)) % 7

    def residual(self, p, p_old, s_old, dt):
        q = self.prob
        area = (q.dy * q.dz, q.dx * q.dz, q.dx * q.dy)
        vol = q.dx * q.dy * q.dz
        kr, s = _vg(p, self.alpha, self.n)
        f = (s - s_old) * q.porosity * vol + q.specific_storage * vol * (p * s - p_old * s_old)
        for ax, d, (gs, gc), ar in ((2, q.dx, self.grav[0], area[0]),
                                    (1, q.dy, self.grav[1], area[1]), (0, q.dz, (1.0, 1.0), area[2])):
            m = p.shape[ax] - 1
            if m < 1:
                continue
            lo, hi = (lambda a: a.narrow(ax, 0, m)), (lambda a: a.narrow(ax, 1, m))
            drop = (lo(p) - hi(p)) / d * gc - gs
            ka, kb = lo(self.k), hi(self.k)
            u = dt * ar * (2.0 * ka * kb / (ka + kb)) * drop * torch.where(drop >= 0, lo(kr), hi(kr))
            pad = [0, 0, 0, 0, 0, 0]
            pad[2 * (2 - ax) + 1] = 1
            out = torch.nn.functional.pad(u, pad)
            f = f + out - torch.roll(out, 1, ax)  # the padded last face is zero
        top = q.bc["z_upper"]
        rain = dt * area[2] * float(top.values[0])
        extra = torch.full_like(p[-1], rain)
        if top.kind == BC_OVERLAND_KIN:
            extra = extra + self._overland(p[-1], p_old[-1], dt, vol)
        f = torch.cat([f[:-1], (f[-1] + extra)[None]])
        low = q.bc["z_lower"]
        if low.kind == BC_DIRICHLET:
            v = float(low.values[0])
            drop = (v - p[0]) / q.dz - 0.5
            u = dt * area[2] * 2.0 * self.k[0] * drop * torch.where(drop >= 0, torch.ones_like(kr[0]),
                                                                    kr[0])
            f = torch.cat([(f[0] - u)[None], f[1:]])
        return f

    def _overland(self, pt, pt_old, dt, vol):
        q = self.prob
        h = pt.clamp(min=0.0)
        sq = (self.sx ** 2 + self.sy ** 2).sqrt().clamp(min=1e-5).sqrt() * q.mannings
        div = 0.0
        for s, ax, d in ((self.sx, 1, q.dx), (self.sy, 0, q.dy)):
            up = torch.cat([h.narrow(ax, 1, h.shape[ax] - 1),
                            torch.zeros_like(h.narrow(ax, 0, 1))], ax)
            ke = -(s / sq) * torch.where(-s >= 0, h, up) ** (5.0 / 3.0)
            s0, q0, h0 = (a.narrow(ax, 0, 1) for a in (s, sq, h))
            edge = torch.where(s0 > 0, -(s0 / q0) * h0 ** (5.0 / 3.0), torch.zeros_like(h0))
            kw = torch.cat([edge, ke.narrow(ax, 0, ke.shape[ax] - 1)], ax)
            div = div + (ke - kw) / d
        return vol / q.dz * ((h - pt_old.clamp(min=0.0)) + dt * div)

    OFFSETS = ((0, 0, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0))

    def jacobian(self, p, p_old, s_old, dt):
        """Columns of J by neighbour: entry d of cell c is dF(c + d) / dp(c).
        Cells of one colour share no neighbour, so seven products with the
        transpose give them all."""
        with torch.enable_grad():
            p = p.detach().requires_grad_(True)
            f = self.residual(p, p_old, s_old, dt)
        by = torch.stack([torch.autograd.grad(f, p, (self.colour == c).double(),
                                              retain_graph=c < 6)[0] for c in range(7)])
        out = []
        for dz, dy, dx in self.OFFSETS:
            out.append(by.gather(0, ((self.colour + dx + 2 * dy + 3 * dz) % 7)[None])[0])
        return out

    @classmethod
    def _shift(cls, a, d):
        """b(c) = a(c - d), zero where c - d is outside."""
        for ax, s in enumerate(d):
            if s:
                z = torch.zeros_like(a.narrow(ax, 0, 1))
                m = a.shape[ax] - 1
                a = torch.cat([z, a.narrow(ax, 0, m)] if s > 0 else [a.narrow(ax, 1, m), z], ax)
        return a

    def times(self, j, x, transpose=False):
        y = j[0] * x
        for e, d in zip(j[1:], self.OFFSETS[1:]):
            if transpose:
                y = y + e * self._shift(x, tuple(-v for v in d))
            else:
                y = y + self._shift(e * x, d)
        return y

    def solve(self, j, b, tol, transpose=False):
        """BiCGSTAB with the diagonal as preconditioner."""
        x = torch.zeros_like(b)
        r, rh = b.clone(), b.clone()
        rho = al = om = 1.0
        v = w = torch.zeros_like(b)
        stop = tol * float(b.norm())
        if stop == 0.0:
            return x
        for _ in range(4000):
            rho1 = float((rh * r).sum())
            w = r + (rho1 / rho) * (al / om) * (w - om * v)
            rho = rho1
            y = w / j[0]
            v = self.times(j, y, transpose)
            al = rho / float((rh * v).sum())
            r = r - al * v
            z = r / j[0]
            t = self.times(j, z, transpose)
            om = float((t * r).sum() / (t * t).sum().clamp_min(1e-300))
            x = x + al * y + om * z
            r = r - om * t
            if not float(r.norm()) > stop or om == 0.0 or rho == 0.0:
                break
        return x

    def step(self, p_old, dt):
        """p with F(p) = 0 to rounding."""
        s_old = _vg(p_old, self.alpha, self.n)[1]
        p, last = p_old.clone(), math.inf
        norm = lambda v: float(v.norm())
        f = self.residual(p, p_old, s_old, dt)
        for _ in range(40):
            now = norm(f)
            if float(f.abs().max()) <= 1e-14 or (now < 1e-10 and now > 0.3 * last):
                break
            last = now
            d = self.solve(self.jacobian(p, p_old, s_old, dt), -f, 1e-6)
            lam = 1.0
            for _ in range(20):
                f1 = self.residual(p + lam * d, p_old, s_old, dt)
                if norm(f1) < now or now < 1e-10:
                    break
                lam *= 0.5
            p, f = p + lam * d, f1
        return p


#: cells above which the plain solve takes longer than is useful
SOLVE_CELLS = 1_500_000


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("residual", "matvec") and _cells(case) > SOLVE_CELLS:
        return None
    if kind == "ensemble":
        return [_pad(_Exact(p, f).step(f["p0"], p.dt)) for p, f, _ in _member_problems(case, seed)]
    if kind == "step":
        prob, f, _ = _problem(case["physics"], case["nx"], case["ny"], case["nz"], seed)
        return _pad(_Exact(prob, f).step(f["p0"], prob.dt))
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    prob, f = _operands(case, seed)
    e = _Exact(prob, f)
    if kind == "residual":
        return _pad(e.residual(f["p"], f["p0"], f["s_old"], prob.dt))
    if kind == "matvec":
        return _pad(e.times(e.jacobian(f["p"], f["p0"], f["s_old"], prob.dt), f["x"]))
    p = e.step(f["p0"], prob.dt)
    return _pad(p).cpu(), _pad(_vg(p, f["alpha"], f["n"])[1]).cpu()


def _exact_adjoint(case, seed):
    """Trajectory, misfit and its gradient: the transposed solves backwards
    over the steps, the parameter derivatives by autograd of F."""
    prob, f, _ = _problem(case["physics"], case["nx"], case["ny"], case["nz"], seed, case["steps"])
    steps, cells, obs = _observations(case, seed)
    obs = torch.as_tensor(obs, device=DEV)
    cells = torch.as_tensor(cells, device=DEV)
    e = _Exact(prob, f)
    p = [f["p0"]]
    for _ in steps:
        p.append(e.step(p[-1], prob.dt).detach())
    lnk = f["k"].log()
    like = lambda v: torch.as_tensor(v, device=DEV, dtype=torch.float64).expand(prob.shape).clone()
    theta = [lnk, like(f["alpha"]), like(f["n"])]
    grads = [torch.zeros_like(lnk) for _ in range(3)]
    carry = torch.zeros_like(lnk)
    misfit = 0.0
    for i in range(len(steps), 0, -1):
        err = p[i].reshape(-1)[cells] - obs[i - 1]
        misfit += float((err * err).sum())
        rhs = carry.reshape(-1).index_add(0, cells, -2.0 * err).reshape(prob.shape)
        s_old = _vg(p[i - 1], e.alpha, e.n)[1]
        lam = e.solve(e.jacobian(p[i], p[i - 1], s_old, prob.dt), rhs, 1e-13, transpose=True)
        th = [t.detach().requires_grad_(True) for t in theta]
        po = p[i - 1].detach().requires_grad_(True)
        v = _Exact(prob, dict(k=th[0].exp(), alpha=th[1], n=th[2]))
        r = v.residual(p[i], po, _vg(po, th[1], th[2])[1], prob.dt)
        g = torch.autograd.grad((lam * r).sum(), th + [po])
        for a, b in zip(grads, g):
            a += b
        carry = -g[3]
    host = lambda a: a.cpu().numpy()
    return dict(p=_pad(p[-1]), misfit=misfit, lnk=host(grads[0]), alpha=host(grads[1]),
                n=host(grads[2]))
