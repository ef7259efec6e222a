"""What is timed: the calls a user of this framework makes, over the sizes and
options they are made at.

Kinds of case
  calls      the reference's host loop over the drop-in boundary: one
             calculateStep at a time, u, v and p read back after each (its
             SIMPLE::runIterations samples the host fields every iteration)
  dispatch   the three solver calls alone (solveUMomentumImplicit,
             solveVMomentumImplicit, solvePressureSystem) on a host's fields
  flow       a forward solve on a kept solver object: reset, new density up,
             a number of outer iterations, u, v and p back
  objective  the optimiser's flow objective (PressureDrop), forward only, as
             a line search evaluates it
  gradient   PressureDrop forward and backward: one flow sensitivity
  batch      many fields of uneven sizes advanced together (Batch)
  thermal    a kept thermal solver: new inputs, solve, temperatures and the
             p-norm gradient back
  thermal_objective  the optimiser's thermal objective (ThermalPNorm),
             forward and backward

The forward solves run a set number of outer iterations, because at most
sizes the reference's iteration needs hundreds to thousands of them and each
costs the same.  Geometries, inlet velocities and heat fluxes are those of
coldplate_b200.cases (straight channel, channel network, projected Gaussian
random density), drawn from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "coldplate-solver_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from coldplate_b200 import cases as geometries  # noqa: E402
from coldplate_b200.autograd import PressureDrop, ThermalPNorm  # noqa: E402
from coldplate_b200.solver import Batch, Simple  # noqa: E402
from coldplate_b200.thermal import Thermal  # noqa: E402

H = geometries.H


def listed():
    return [
        # the smallest calls: the reference's own 256 x 64 channel, one outer
        # iteration at a time; launches and latencies count
        dict(name="calls_channel_64x256", kind="calls", geometry="channel", Ny=64, Nx=256, solver=1,
             precision="fp64", outer=4),
        # a host code that replaces only its three linear solvers, on a ragged
        # medium grid with the default pressure solver
        dict(name="dispatch_density_241x517", kind="dispatch", geometry="density", Ny=241, Nx=517, solver=4,
             precision="fp64", outer=1),
        # the channel network, plain FP64 with the reference's Jacobi-PCG
        dict(name="flow_network_fp64_512x1024", kind="flow", geometry="network", Ny=512, Nx=1024, solver=1,
             precision="fp64", outer=12),
        # a medium design in mixed precision on an odd grid, as an objective
        # evaluation on a float32 design
        dict(name="objective_density_389x811", kind="objective", geometry="density", Ny=389, Nx=811, solver=4,
             precision="mixed", outer=100),
        # the largest density field in FP64 with the default pressure solver
        dict(name="flow_density_fp64_1024x2048", kind="flow", geometry="density", Ny=1024, Nx=2048, solver=4,
             precision="fp64", outer=16),
        # the headline workload: the largest density field in mixed precision
        # up to where its pressure drop has settled to 1e-5
        dict(name="objective_density_1024x2048", kind="objective", geometry="density", Ny=1024, Nx=2048, solver=4,
             precision="mixed", outer=154),
        # one flow sensitivity of a medium design in mixed precision
        dict(name="gradient_density_384x768", kind="gradient", geometry="density", Ny=384, Nx=768, solver=4,
             precision="mixed", outer=300),
        # one flow sensitivity of a small ragged design in FP64
        dict(name="gradient_density_fp64_127x253", kind="gradient", geometry="density", Ny=127, Nx=253, solver=4,
             precision="fp64", outer=200),
        # a set of designs of uneven sizes solved together
        dict(name="batch_density_24", kind="batch", geometry="density", fields=24, Ny=512, Nx=1024, solver=4,
             precision="mixed", outer=20),
        # the thermal objective of the 3-D workload (8 plate + 4 channel
        # layers) and its sensitivity, FP64
        dict(name="thermal_objective_512x1024x12", kind="thermal_objective", Ny=512, Nx=1024, nz_solid=8, nz_fluid=4,
             precision="fp64", rtol=1e-6),
        # the same in mixed precision on a ragged grid with the default layers
        dict(name="thermal_objective_mixed_259x501x9", kind="thermal_objective", Ny=259, Nx=501, nz_solid=2,
             nz_fluid=7, precision="mixed", rtol=1e-6),
        # a small ragged plate solved to a tight tolerance, temperatures and
        # gradient in double
        dict(name="thermal_tight_97x151x9", kind="thermal", Ny=97, Nx=151, nz_solid=2, nz_fluid=7, precision="fp64",
             rtol=1e-12),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calls", "dispatch", "flow", "flow", "objective", "gradient", "batch", "thermal",
                       "thermal_objective"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "calls":
        Ny = _size(rng, 40, 160)
        return dict(kind=kind, geometry="channel", Ny=Ny, Nx=Ny * 2 + rng.randrange(2 * Ny), solver=1,
                    precision="fp64", outer=rng.randrange(2, 5))
    if kind == "dispatch":
        Ny = _size(rng, 96, 420)
        return dict(kind=kind, geometry="density", Ny=Ny, Nx=Ny + rng.randrange(2 * Ny), solver=rng.choice([1, 4]),
                    precision="fp64", outer=1)
    if kind in ("flow", "objective"):
        Ny = _size(rng, 96, 900)
        geometry = rng.choice(["network", "density"]) if kind == "flow" else "density"
        return dict(kind=kind, geometry=geometry, Ny=Ny, Nx=Ny + rng.randrange(Ny),
                    solver=1 if geometry == "network" else 4,
                    precision="fp64" if kind == "flow" else precision,
                    outer=rng.randrange(8, 17) if kind == "flow" else rng.randrange(100, 155))
    if kind == "gradient":
        Ny = _size(rng, 96, 360)
        return dict(kind=kind, geometry="density", Ny=Ny, Nx=2 * Ny + rng.randrange(Ny // 8), solver=4,
                    precision=precision, outer=rng.randrange(200, 301) if precision == "fp64" else 300)
    if kind == "batch":
        return dict(kind=kind, geometry="density", fields=rng.randrange(6, 24), Ny=_size(rng, 200, 512),
                    Nx=_size(rng, 400, 1024), solver=4, precision="mixed", outer=rng.randrange(8, 21))
    Ny = _size(rng, 48, 180) if kind == "thermal" else _size(rng, 80, 420)
    layers = rng.choice([(2, 7), (8, 4), (3, 4)])
    return dict(kind=kind, Ny=Ny, Nx=Ny + rng.randrange(Ny), nz_solid=layers[0], nz_fluid=layers[1],
                precision="fp64" if kind == "thermal" else precision, rtol=1e-12 if kind == "thermal" else 1e-6)


# ------------------------------------------------------------------ inputs
def _flow_case(case, seed):
    """Geometry (cell types), inlet velocity and the knobs of a flow case."""
    rng = np.random.default_rng([seed, 1])
    Ny, Nx, g = case["Ny"], case["Nx"], case["geometry"]
    over = dict(maxIterations=100000, pressureSolverType=case["solver"], precision=case["precision"])
    if case["solver"] == 4:
        over["pTol"] = 1e-6          # relative for type 4: the default
    if g == "channel":
        c = geometries.straight_channel(Ny, Nx, U=float(rng.uniform(0.3, 0.7)), **over)
    elif g == "network":
        c = geometries.random_network(Ny, Nx, seed=seed, **over)
    else:
        c = geometries.density_field(Ny, Nx, seed=seed, U=float(rng.uniform(0.3, 0.7)), **over)
        if case["kind"] == "gradient":
            # openings that leave the design permeable at every size, as a
            # design being optimised is
            c.cellType = (1.0 - geometries.density_gamma(Ny, Nx, seed, corr=16.0, mean=0.9)) \
                .astype(np.float32).astype(np.float64)
    return c, c.params(historyCapacity=max(case["outer"], 64))


def _smooth(Ny, Nx, corr, rng):
    """A smooth random field, zero mean and unit variance."""
    g = geometries.gaussian_random_field(Ny, Nx, corr, rng)
    return (g - g.mean()) / max(g.std(), 1e-300)


def _host_fields(case, c, seed):
    """u, v, p of a host code in the middle of its iteration: a through-flow
    in the open cells with eddies on it and a falling pressure."""
    rng = np.random.default_rng([seed, 2])
    M, N = case["Ny"] + 1, case["Nx"] + 1
    open_ = 1.0 - np.pad(c.cellType, ((0, 1), (0, 1)), mode="edge")          # M x N
    u, v, p = np.zeros((M + 1, N)), np.zeros((M, N + 1)), np.zeros((M + 1, N + 1))
    u[1:M] = c.U * open_[:-1] * (1.0 + 0.2 * _smooth(M - 1, N, 24, rng))
    v[1:M - 1, 1:N] = 0.1 * c.U * open_[:-2, :-1] * _smooth(M - 2, N - 1, 24, rng)
    p[:, :] = 4000.0 * (1.0 - np.arange(N + 1) / N)[None, :] + 20.0 * _smooth(M + 1, N + 1, 32, rng)
    p[:, N] = 0.0
    return u, v, p


def _batch_sizes(case, seed):
    """Sizes of the batch's fields: between a quarter and all of Ny x Nx per
    side, the same for every seed; geometry and velocity follow the seed."""
    rng = np.random.default_rng([case["fields"], case["Ny"], case["Nx"]])
    return [(int(rng.integers(case["Ny"] // 4, case["Ny"] + 1)), int(rng.integers(case["Nx"] // 4, case["Nx"] + 1)))
            for _ in range(case["fields"])]


def _thermal_inputs(case, seed):
    """Density, a divergence-free flow through its open cells, heat flux."""
    rng = np.random.default_rng([seed, 3])
    Ny, Nx = case["Ny"], case["Nx"]
    gamma = geometries.density_gamma(Ny, Nx, seed)
    psi = 12.0 * _smooth(Ny + 1, Nx + 1, 32, rng)
    u = 0.5 + (psi[1:, :-1] - psi[:-1, :-1]) * 0.5
    v = -(psi[:-1, 1:] - psi[:-1, :-1]) * 0.5
    q0 = geometries.power_map(Ny, Nx, seed) * 1e4
    return gamma, u * gamma, v * gamma, q0


def _thermal_params(case):
    p = dict(geometries.THERMAL_3D) if case["nz_solid"] == 8 else dict(H_t=2e-4)
    p.update(Nx=case["Nx"], Ny=case["Ny"], dx=H, dy=H, nz_solid=case["nz_solid"], nz_fluid=case["nz_fluid"],
             rtol=case["rtol"], precision=1 if case["precision"] == "mixed" else 0)
    return p


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("thermal", "thermal_objective"):
        gamma, u, v, q0 = _thermal_inputs(case, seed)
        s = dict(kind=kind, u=u, v=v, q0=q0, params=_thermal_params(case))
        if kind == "thermal":
            s.update(gamma=gamma, solver=Thermal(**s["params"]))
        else:
            s["gamma"] = torch.tensor(gamma, dtype=torch.float32, device="cuda", requires_grad=True)
        return s
    if kind == "batch":
        fields, densities = [], []
        for k, (Ny, Nx) in enumerate(_batch_sizes(case, seed)):
            c, knobs = _flow_case(dict(case, Ny=Ny, Nx=Nx), 1000 * (seed % 1000003) + k)
            densities.append(1.0 - c.cellType)
            fields.append(Simple(gamma=densities[-1], **knobs))
        # a team size such as the autotuner picks for a set like this one (it
        # chooses by timing, so its choice may differ from run to run)
        batch = Batch(fields)
        batch.set_team(6)
        return dict(kind=kind, fields=fields, densities=densities, batch=batch, outer=case["outer"])
    c, knobs = _flow_case(case, seed)
    s = dict(kind=kind, outer=case["outer"])
    if kind in ("objective", "gradient"):
        knobs["maxIterations"] = case["outer"]
        s["knobs"] = knobs
        s["gamma"] = torch.tensor(1.0 - c.cellType, dtype=torch.float32, device="cuda",
                                  requires_grad=kind == "gradient")
        return s
    s["gamma"] = 1.0 - c.cellType
    s["solver"] = Simple(cellType=c.cellType, **knobs)
    if kind == "dispatch":
        s["u"], s["v"], s["p"] = _host_fields(case, c, seed)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "calls":
        solver, errors = s["solver"], []
        solver.reset()
        for _ in range(s["outer"]):
            errors.append(solver.calculateStep())
            u, v, p = solver.get("u"), solver.get("v"), solver.get("p")
        return dict(u=u, v=v, p=p, error=errors[-1])
    if kind == "dispatch":
        solver = s["solver"]
        for f in ("u", "v", "p"):
            solver.set(f, s[f])
        residU = solver.solveUMomentumImplicit()[1]
        residV = solver.solveVMomentumImplicit()[1]
        residMass = solver.solvePressureSystem()[1]
        return dict(uStar=solver.get("uStar"), vStar=solver.get("vStar"), pStar=solver.get("pStar"),
                    dE=solver.get("dE"), dN=solver.get("dN"), residU=residU, residV=residV, residMass=residMass)
    if kind == "flow":
        solver = s["solver"]
        solver.reset()
        solver.set_gamma(s["gamma"])
        report = solver.step(s["outer"])
        return dict(u=solver.get("u"), v=solver.get("v"), p=solver.get("p"), dp=report["fullTotalDrop"])
    if kind == "objective":
        flow = {}
        dp = PressureDrop.apply(s["gamma"], s["knobs"], s["outer"], 1e-8, flow)
        # the flow in the design's type, as it goes into the rest of a float32 program
        return dict(dp=dp, **{f: torch.from_numpy(flow[f]).to(s["gamma"].dtype) for f in ("u", "v", "p")})
    if kind == "gradient":
        s["gamma"].grad = None
        dp = PressureDrop.apply(s["gamma"], s["knobs"], s["outer"], 1e-8)
        dp.backward()
        return dict(dp=dp.detach(), gradient=s["gamma"].grad)
    if kind == "batch":
        for f, g in zip(s["fields"], s["densities"]):
            f.reset()
            f.set_gamma(g)
        s["batch"].run(s["outer"])
        out = [torch.from_numpy(np.concatenate([f.get(name).ravel() for name in ("u", "v", "p")])).float()
               for f in s["fields"]]
        return dict(fields=out)
    if kind == "thermal":
        th = s["solver"]
        th.set_inputs(s["gamma"], s["u"], s["v"], s["q0"])
        th.solve()
        J, gradient, _ = th.pnorm_gradient(8.0)
        return dict(T=th.T, J=J, gradient=gradient)
    s["gamma"].grad = None
    J = ThermalPNorm.apply(s["gamma"], s["u"], s["v"], s["q0"], s["params"], 8.0)
    J.backward()
    return dict(J=J.detach(), gradient=s["gamma"].grad)


def work(case):
    """Bytes: every outer iteration (flow) or every solve (thermal) reads its
    inputs once and writes its results once; flops: one assembly, two Jacobi
    sweeps of each component and ten CG iterations an outer iteration, and
    forty matvecs of the 7-point system a thermal solve."""
    kind = case["kind"]
    if kind in ("thermal", "thermal_objective"):
        plane, n = case["Ny"] * case["Nx"], case["Ny"] * case["Nx"] * (case["nz_solid"] + case["nz_fluid"])
        return dict(bytes=8.0 * (5 * plane + 4 * n), flops=2.0 * 40 * 14 * n)
    if kind == "batch":
        cells, outer = sum(a * b for a, b in _batch_sizes(case, 0)), case["outer"]
    else:
        cells, outer = case["Ny"] * case["Nx"], case["outer"]
    backward = 2.0 if kind == "gradient" else 1.0
    return dict(bytes=backward * outer * cells * 8.0 * 8, flops=backward * outer * cells * (150.0 + 4 * 12 + 10 * 20))


# ------------------------------------------------------------------ 64-bit results
def _t(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


class _Flow:
    """The SIMPLE outer iteration in plain torch, 64 bits: staggered u
    (M+1) x N, v M x (N+1), p (M+1) x (N+1); upwind or second-order-upwind
    convection, Brinkman and 2.5-D sinks, Jacobi momentum sweeps, conjugate
    gradients on the pressure correction."""

    def __init__(self, case, seed):
        c, k = _flow_case(case, seed)
        self.k, self.U = k, c.U
        self.M, self.N = case["Ny"] + 1, case["Nx"] + 1
        self.rho, self.hx, self.hy, self.eta = k["rho"], k["hx"], k["hy"], k["eta"]
        if case["kind"] == "objective":    # the density as the float32 tensor holds it
            cell = 1.0 - (1.0 - c.cellType).astype(np.float32).astype(np.float64)
        else:
            cell = c.cellType
        self.gamma = 1.0 - _t(np.pad(cell, ((0, 1), (0, 1)), mode="edge")).clamp(0.0, 1.0)
        amax = self.eta / max(k["brinkmanKMin"] if "brinkmanKMin" in k else 1e-14, 1e-20)
        q = k.get("brinkmanQ", 1.0)
        self.alpha = amax * (1.0 - self.gamma) / (1.0 + q * self.gamma + 1e-10)
        flat = k.get("enableTwoPointFiveD", 0) and c.Ht > 0
        self.conv = k.get("twoPointFiveDConvectionFactor", 1.2) if flat else 1.0
        self.sink = 12.0 * self.eta / c.Ht ** 2 * self.hx * self.hy if flat else 0.0
        self.sou = k.get("convectionScheme", 0) == 1
        self.ua, self.pa = k.get("uvAlpha", 0.7), k.get("pAlpha", 0.3)
        self.maxv = 3.0 * max(abs(self.U), 0.1)
        self.maxP, self.pTol = k.get("maxPressureIter", 30), k["pTol"]
        M, N = self.M, self.N
        self.u, self.v, self.p = _t(np.zeros((M + 1, N))), _t(np.zeros((M, N + 1))), _t(np.zeros((M + 1, N + 1)))
        rows = [0 if i <= 0 else max(M - 2, 0) if i >= M else i - 1 for i in range(M + 1)]
        self.inlet = torch.where(self.gamma[rows, 0] > 0.5, self.U, 0.0).to(torch.float64)

    def boundaries(self, u, v, p=None):
        M, N = self.M, self.N
        u[:, 0] = self.inlet
        u[0, 1:] = 0.0
        u[M, 1:] = 0.0
        u[1:M, N - 1] = u[1:M, N - 2]
        v[0] = 0.0
        v[M - 1] = 0.0
        v[1:M - 1, 0] = 0.0
        v[1:M - 1, N] = v[1:M - 1, N - 1]
        if p is not None:
            p[0, 1:N], p[M, 1:N] = p[1, 1:N].clone(), p[M - 1, 1:N].clone()
            p[1:M, 0] = p[1:M, 1]
            p[1:M, N] = 0.0

    def momentum(self, is_u):
        """(u* or v*, d, max change) of one momentum system."""
        M, N, u, v, p, hx, hy = self.M, self.N, self.u, self.v, self.p, self.hx, self.hy
        w = u if is_u else v
        I, J = (M - 1, N - 2) if is_u else (M - 2, N - 1)
        W = torch.nn.functional.pad(w, (2, 2, 2, 2))

        def at(a, b):
            return W[3 + a:3 + a + I, 3 + b:3 + b + J]

        def face(x):
            return x.clamp(-self.maxv, self.maxv)

        al, ga = self.alpha, self.gamma
        if is_u:
            al, ga = 0.5 * (al[:I, :J] + al[:I, 1:J + 1]), 0.5 * (ga[:I, :J] + ga[:I, 1:J + 1])
            ue, uw = face(0.5 * (at(0, 0) + at(0, 1))), face(0.5 * (at(0, -1) + at(0, 0)))
            vn = face(0.5 * (v[1:M, 1:N - 1] + v[1:M, 2:N]))
            vs = face(0.5 * (v[0:M - 1, 1:N - 1] + v[0:M - 1, 2:N]))
            S = (p[1:M, 1:N - 1] - p[1:M, 2:N]) * hy
        else:
            al, ga = 0.5 * (al[:I, :J] + al[1:I + 1, :J]), 0.5 * (ga[:I, :J] + ga[1:I + 1, :J])
            ue, uw = face(0.5 * (u[1:M - 1, 1:N] + u[2:M, 1:N])), face(0.5 * (u[1:M - 1, 0:N - 1] + u[2:M, 0:N - 1]))
            vn, vs = face(0.5 * (at(0, 0) + at(1, 0))), face(0.5 * (at(-1, 0) + at(0, 0)))
            S = (p[1:M - 1, 1:N] - p[2:M, 1:N]) * hx
        Fe, Fw = self.conv * self.rho * hy * ue, self.conv * self.rho * hy * uw
        Fn, Fs = self.conv * self.rho * hx * vn, self.conv * self.rho * hx * vs
        De, Dn = self.eta * hy / hx, self.eta * hx / hy
        aE, aW = De + (-Fe).clamp(min=0), De + Fw.clamp(min=0)
        aN, aS = Dn + (-Fn).clamp(min=0), Dn + Fs.clamp(min=0)
        if is_u:    # half cells at the walls (v's side walls: the inlet moves and the outlet is open)
            aS[0] += torch.where(ga[0] >= 0.999, Dn, 0.0)
            aN[-1] += torch.where(ga[-1] >= 0.999, Dn, 0.0)
        aP0 = (aE + aW + aN + aS + (Fe - Fw + Fn - Fs) + self.sink + al * hx * hy).clamp(min=1e-10)
        S = S + (1.0 - self.ua) / self.ua * aP0 * at(0, 0)
        if self.sou:
            i = torch.arange(1, I + 1, device=w.device)[:, None]
            j = torch.arange(1, J + 1, device=w.device)[None, :]
            R, C = w.shape
            for F, sign, a, b, lo, hi, near in ((Fe, -1, 0, 1, j >= 2, j + 2 < C, 0), (Fw, 1, 0, 1, j >= 2, j + 1 < C, -1),
                                                (Fn, -1, 1, 0, i >= 1, i + 2 < R, 0), (Fs, 1, 1, 0, i >= 2, i + 1 < R, -1)):
                x = [at(a * (near + n), b * (near + n)) for n in (-1, 0, 1, 2)]
                up = torch.where(lo, 0.5 * (x[1] - x[0]), 0.0)
                down = torch.where(hi, 0.5 * (x[2] - x[3]), 0.0)
                S = S + sign * F * torch.where(F >= 0, up, down)
        aP, x0 = aP0 / self.ua, at(0, 0)
        # neighbours on the boundary go to the right-hand side
        for edge, a, nb in (((slice(None), -1), aE, at(0, 1)), ((slice(None), 0), aW, at(0, -1)),
                            ((-1, slice(None)), aN, at(1, 0)), ((0, slice(None)), aS, at(-1, 0))):
            S[edge] += (a * nb)[edge]
            a[edge] = 0.0
        x, limit = torch.nn.functional.pad(x0, (1, 1, 1, 1)), self.k.get("momentumTol", 1e-6) ** 2 * I * J
        for _ in range(400):
            r = S - (aP * x[1:-1, 1:-1] - aS * x[:-2, 1:-1] - aW * x[1:-1, :-2] - aE * x[1:-1, 2:] - aN * x[2:, 1:-1])
            x[1:-1, 1:-1] += r / aP
            if float((r * r).sum()) < limit:
                break
        star, d = torch.zeros_like(w), torch.zeros_like(w)
        star[1:1 + I, 1:1 + J] = x[1:-1, 1:-1].clamp(-self.maxv, self.maxv)
        d[1:1 + I, 1:1 + J] = (hy if is_u else hx) / aP0
        return star, d, (star - w)[1:1 + I, 1:1 + J].abs().max()

    def pressure(self, us, vs, dE, dN, converge=False):
        """(p', max imbalance): Jacobi-preconditioned conjugate gradients, to
        the iteration limit or (converge) as far as 64 bits go."""
        M, N, hx, hy = self.M, self.N, self.hx, self.hy
        b = self.rho * hy * (us[1:M, 0:N - 1] - us[1:M, 1:N]) + self.rho * hx * (vs[0:M - 1, 1:N] - vs[1:M, 1:N])
        worst, r = b.abs().max(), b[:, :-1].clone()
        E, Nn = self.rho * hy * dE[1:M, 1:N - 1], self.rho * hx * dN[1:M, 1:N - 1].clone()
        Nn[-1] = 0.0
        d = E.clone()
        d[:, 1:] += E[:, :-1]
        d += Nn
        d[1:] += Nn[:-1]
        d = torch.where(d < 1e-20, 1.0, d)

        def apply(x):
            y = d * x
            y[:, :-1] -= E[:, :-1] * x[:, 1:]
            y[:, 1:] -= E[:, :-1] * x[:, :-1]
            y[:-1] -= Nn[:-1] * x[1:]
            y[1:] -= Nn[:-1] * x[:-1]
            return y

        x, z = torch.zeros_like(r), r / d
        q, rz, stop = z.clone(), float((r * z).sum()), 1e-13 * float(r.norm()) if converge else self.pTol
        for _ in range(20000 if converge else self.maxP):
            Aq = apply(q)
            qq = float((q * Aq).sum())
            if abs(qq) < (0.0 if converge else 1e-20) or qq == 0.0:
                break
            a = rz / qq
            x += a * q
            r -= a * Aq
            if float(r.norm()) < stop:
                break
            z = r / d
            new = float((r * z).sum())
            q = z + (new / rz) * q
            rz = new
        ps = torch.zeros_like(self.p)
        ps[1:M, 1:N - 1] = x
        return ps, worst

    def step(self):
        M, N, mv = self.M, self.N, self.maxv
        self.boundaries(self.u, self.v, self.p)
        us, dE, _ = self.momentum(True)
        vs, dN, _ = self.momentum(False)
        self.boundaries(us, vs)
        nU, nV, nM = (M - 1) * (N - 2), (M - 2) * (N - 1), (M - 1) * (N - 1)
        du, dv = (us - self.u)[1:M, 1:N - 1], (vs - self.v)[1:M - 1, 1:N]
        b = self.rho * self.hy * (us[1:M, 0:N - 1] - us[1:M, 1:N]) + self.rho * self.hx * (vs[0:M - 1, 1:N] - vs[1:M, 1:N])
        self.error = max(float(x.square().sum() / n) ** 0.5 for x, n in ((du, nU), (dv, nV), (b, nM)))
        ps, _ = self.pressure(us, vs, dE, dN)
        self.p[1:M, 1:N] += self.pa * ps[1:M, 1:N]
        cu = (dE[1:M, 1:N - 1] * (ps[1:M, 1:N - 1] - ps[1:M, 2:N])).clamp(-mv, mv)
        self.u[1:M, 1:N - 1] = (us[1:M, 1:N - 1] + cu).clamp(-mv, mv)
        cv = (dN[1:M - 1, 1:N] * (ps[1:M - 1, 1:N] - ps[2:M, 1:N])).clamp(-mv, mv)
        self.v[1:M - 1, 1:N] = (vs[1:M - 1, 1:N] + cv).clamp(-mv, mv)
        self.boundaries(self.u, self.v, self.p)

    def drop(self):
        """Mass-flux-weighted total pressure, inlet patch minus outlet patch."""
        M, N, out = self.M, self.N, []
        for cell, uc, pc in ((0, 0, 0), (N - 2, N - 1, N)):
            rows = self.gamma[:M - 1, cell] >= 1.0 - 1e-6
            un, v = self.u[1:M, uc], self.v[:, pc]
            below = torch.cat([v[1:M - 1], v[M - 1:M]])
            vt = 0.5 * (v[0:M - 1] + below)
            total = self.p[1:M, pc] + 0.5 * self.rho * (un * un + vt * vt)
            f = torch.where(rows, (self.rho * un * self.hy).abs(), 0.0)
            # weighted by area where nothing flows yet
            f = f if float(f.sum()) > 0 else rows.to(f.dtype)
            out.append(float((total * f).sum() / f.sum()) if float(f.sum()) > 0 else 0.0)
        return out[0] - out[1]


def _thermal_system(case, gamma, u, v, q0):
    """Coefficients of the 7-point conduction / upwind-advection system
    (entries towards W, E, S, N, below, above, the diagonal) and b as tensors
    Nz x Ny x Nx, differentiable in gamma; the fluid mask held fixed."""
    prm = _thermal_params(case)
    nzS, nzF = case["nz_solid"], case["nz_fluid"]
    kS, kF = prm.get("k_s", 400.0), prm.get("k_f", 0.6)
    rhoCp, Tin = prm.get("rho", 998.0) * prm.get("Cp", 4180.0), prm.get("T_inlet", 30.0)
    Hb, Ht = prm.get("H_b", 5e-4), prm["H_t"]
    nz, (Ny, Nx) = nzS + nzF, gamma.shape
    g = gamma.clamp(0.0, 1.0)
    kc = kF + (kS - kF) * (1.0 - g) / (1.0 + g)
    k = torch.cat([torch.full((nzS, Ny, Nx), kS, dtype=g.dtype, device=g.device), kc.expand(nzF, Ny, Nx)])
    dz = _t([Hb / nzS] * nzS + [Ht / nzF] * nzF)[:, None, None]
    fluid = (gamma.detach() > 0.01).expand(nz, Ny, Nx).clone()
    fluid[:nzS] = False
    zc = (torch.arange(nzF, dtype=g.dtype, device=g.device) + 0.5) / nzF
    po = torch.cat([torch.zeros(nzS, dtype=g.dtype, device=g.device), 4.0 * zc * (1.0 - zc)])[:, None, None]
    U, V = u * po * fluid, v * po * fluid
    Ax, Ay, Az = H * dz, H * dz, H * H
    zero = torch.zeros((nz, Ny, Nx), dtype=g.dtype, device=g.device)

    def harm(a, b):
        return 2.0 * a * b / (a + b + 1e-30)

    def pad(x, dim, before):
        shape = list(x.shape)
        shape[dim] = 1
        z = torch.zeros(shape, dtype=x.dtype, device=x.device)
        return torch.cat([z, x] if before else [x, z], dim)

    both_x, both_y = fluid[:, :, 1:] & fluid[:, :, :-1], fluid[:, 1:] & fluid[:, :-1]
    Dx, Dy = harm(k[:, :, 1:], k[:, :, :-1]) * Ax / H, harm(k[:, 1:], k[:, :-1]) * Ay / H
    Fx = rhoCp * 0.5 * (U[:, :, 1:] + U[:, :, :-1]) * Ax * both_x
    Fy = rhoCp * 0.5 * (V[:, 1:] + V[:, :-1]) * Ay * both_y
    kz = (dz[1:] + dz[:-1]) / (dz[1:] / k[1:] + dz[:-1] / k[:-1])
    Dz = kz * Az / (0.5 * (dz[1:] + dz[:-1]))
    aW, aE = -pad(Dx + Fx.clamp(min=0), 2, True), -pad(Dx + (-Fx).clamp(min=0), 2, False)
    aS, aN = -pad(Dy + Fy.clamp(min=0), 1, True), -pad(Dy + (-Fy).clamp(min=0), 1, False)
    aB, aT = -pad(Dz, 0, True), -pad(Dz, 0, False)
    # the outflow of each cell: its conductances, and the upwind flux that leaves it
    diag = pad(Dx + (-Fx).clamp(min=0), 2, True) + pad(Dx + Fx.clamp(min=0), 2, False)
    diag = diag + pad(Dy + (-Fy).clamp(min=0), 1, True) + pad(Dy + Fy.clamp(min=0), 1, False)
    diag = diag + pad(Dz, 0, True) + pad(Dz, 0, False) + 1e-12
    inlet, b = zero.clone(), zero.clone()
    west = fluid[:, :, 0]
    Dbc, Fbc = 2.0 * k[:, :, 0] * Ax[:, :, 0] / H * west, rhoCp * U[:, :, 0] * Ax[:, :, 0] * west
    out_x = rhoCp * U[:, :, -1].clamp(min=0) * Ax[:, :, 0] * fluid[:, :, -1]
    out_y = rhoCp * V[:, -1].clamp(min=0) * Ay[:, 0] * fluid[:, -1]
    first, last = [torch.zeros(Nx, dtype=g.dtype, device=g.device) for _ in range(2)]
    first[0], last[-1] = 1.0, 1.0
    top = torch.zeros(Ny, dtype=g.dtype, device=g.device)
    top[-1] = 1.0
    bottom = torch.zeros(nz, dtype=g.dtype, device=g.device)
    bottom[0] = 1.0
    diag = diag + (Dbc + (-Fbc).clamp(min=0))[:, :, None] * first + out_x[:, :, None] * last
    diag = diag + out_y[:, None, :] * top[:, None]
    b = (Dbc + Fbc.clamp(min=0))[:, :, None] * first * Tin + (q0 * Az)[None] * bottom[:, None, None]
    return [aW, aE, aS, aN, aB, aT, diag, b]


def _thermal_solve(coef, rhs, transpose):
    """A x = rhs (or A^T x = rhs) by block elimination along x: dense blocks
    over one y-z plane."""
    aW, aE, aS, aN, aB, aT, diag = [c.detach().permute(2, 0, 1) for c in coef[:7]]      # Nx x Nz x Ny
    nx, nz, ny = diag.shape
    n = nz * ny
    if transpose:    # the block towards the west holds the east entries of the west plane
        west = torch.cat([torch.zeros_like(aE[:1]), aE[:-1]])
        east = torch.cat([aW[1:], torch.zeros_like(aW[:1])])
        aW, aE = west, east
    r = rhs.permute(2, 0, 1).reshape(nx, n)
    at = torch.arange(n, device=diag.device)
    G, h, prev = [], [], None
    for i in range(nx):
        D = torch.diag(diag[i].reshape(n))
        for c, off in ((aS, -1), (aN, 1), (aB, -ny), (aT, ny)):
            v = c[i].reshape(n)
            on = (at + off >= 0) & (at + off < n) & (v != 0)
            rows, cols = at[on], at[on] + off
            if transpose:
                rows, cols = cols, rows
            D[rows, cols] += v[on]
        b = r[i].clone()
        if prev is not None:
            w = aW[i].reshape(n)
            D -= w[:, None] * prev[0]
            b -= w * prev[1]
        sol = torch.linalg.solve(D, torch.cat([torch.diag(aE[i].reshape(n)), b[:, None]], 1))
        prev = (sol[:, :n].contiguous(), sol[:, n].contiguous())
        G.append(prev[0])
        h.append(prev[1])
    x = [h[-1]]
    for i in range(nx - 2, -1, -1):
        x.append(h[i] - G[i] @ x[-1])
    return torch.stack(x[::-1]).reshape(nx, nz, ny).permute(1, 2, 0)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("thermal", "thermal_objective"):
        block = case["Ny"] * (case["nz_solid"] + case["nz_fluid"])
        if block * block * case["Nx"] * 8.0 > 12e9 or block ** 3 * case["Nx"] > 3e12:
            return None
        g, u, v, q0 = _thermal_inputs(case, seed)
        gamma = _t(g if kind == "thermal" else g.astype(np.float32).astype(np.float64)).requires_grad_(True)
        coef = _thermal_system(case, gamma, _t(u), _t(v), _t(q0))
        T = _thermal_solve(coef, coef[7].detach(), False)
        J = float((T[0] ** 8.0).mean() ** (1.0 / 8.0))
        rhs = torch.zeros_like(T)
        rhs[0] = (T[0] / J) ** 7.0 / T[0].numel()
        lam = _thermal_solve(coef, rhs, True)
        aW, aE, aS, aN, aB, aT, diag, b = coef
        x = torch.nn.functional.pad(T, (1, 1, 1, 1, 1, 1))
        res = diag * T + aW * x[1:-1, 1:-1, :-2] + aE * x[1:-1, 1:-1, 2:] + aS * x[1:-1, :-2, 1:-1]
        res = res + aN * x[1:-1, 2:, 1:-1] + aB * x[:-2, 1:-1, 1:-1] + aT * x[2:, 1:-1, 1:-1] - b
        grad, = torch.autograd.grad(-(lam * res).sum(), gamma)
        if kind == "thermal":
            return dict(T=T.cpu(), J=J, gradient=grad.cpu())
        return dict(J=J, gradient=grad.cpu())
    if kind in ("gradient", "batch"):
        return None       # no closed form short of the solver under test
    if kind == "dispatch":
        if case["Ny"] * case["Nx"] > 400000:
            return None
        f = _Flow(case, seed)
        c, _ = _flow_case(case, seed)
        f.u, f.v, f.p = (_t(a) for a in _host_fields(case, c, seed))
        us, dE, ru = f.momentum(True)
        vs, dN, rv = f.momentum(False)
        ps, rm = f.pressure(us, vs, dE, dN, converge=case["solver"] == 4)
        return dict(uStar=us.cpu(), vStar=vs.cpu(), pStar=ps.cpu(), dE=dE.cpu(), dN=dN.cpu(), residU=float(ru),
                    residV=float(rv), residMass=float(rm))
    if case["solver"] != 1 or case["Ny"] * case["Nx"] * case["outer"] > 14e6:
        return None       # multigrid CG stops short of the solution by a rule of its own
    f = _Flow(case, seed)
    for _ in range(case["outer"]):
        f.step()
    if kind == "calls":
        return dict(u=f.u.cpu(), v=f.v.cpu(), p=f.p.cpu(), error=f.error)
    return dict(u=f.u.cpu(), v=f.v.cpu(), p=f.p.cpu(), dp=f.drop())
