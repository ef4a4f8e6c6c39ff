"""The workloads by which this framework's speed is followed.

listed() holds the work that users of the Euler solvers have them do, each through the
package's public entry points (Solver, Batch, Checkpoints): whole short runs of small
problems, where latency and launches count; time steps of ordinary and large grids in
1-3 dimensions, both precisions and all three solvers; a self-gravitating step; a sweep of
many problems; a trajectory with its gradient; a step of a program that keeps its state on
the host.  draw() gives more cases of the same ranges.  Sizes count the two ghost layers
on each side of an axis, as the solvers' own `size` does.

exact() restates the schemes with torch in 64 bits: ghost fill, Roe eigenbasis or
HLLC/HLL wave speeds of u^n frozen for the step, CFL timestep, limited flux, Shu-Osher
Runge-Kutta stages, self-gravity relaxation; the gradient is autograd's.
"""
import math

import numpy as np
import torch

import hydrodynamicsgpu_gb300 as hg
from hydrodynamicsgpu_gb300 import _abi

# ---------------------------------------------------------------- the cases

INTEGRATORS = ("ForwardEuler", "RungeKutta2", "RungeKutta2Heun", "RungeKutta4", "RungeKutta2TVD", "RungeKutta3TVD")
LIMITERS = ("MinMod", "Superbee", "MonotizedCentral", "Koren", "DonorCell")


def _case(kind, ic, sx, sy=1, sz=1, solver="EulerRoe", integrator="RungeKutta4", limiter="MinMod",
          boundary="PERIODIC", fp32=False, steps=1, **more):
    return dict({"kind": kind, "ic": ic, "sx": sx, "sy": sy, "sz": sz, "solver": solver, "integrator": integrator,
                 "limiter": limiter, "boundary": boundary, "fp32": fp32, "steps": steps}, **more)


def listed():
    return [
        # a shock tube from initial state to result: the smallest call, all latency
        dict(_case("run", "sod", 1028, integrator="RungeKutta2", limiter="Superbee", boundary="FREEFLOW", steps=200),
             name="sod_1d_run"),
        # the reference's default scheme on one small four-quadrant problem, run to a result
        dict(_case("run", "quadrants", 133, 97, integrator="ForwardEuler", limiter="Superbee", boundary="FREEFLOW",
                   steps=50), name="quadrants_2d_run"),
        # the headline workload: one step of the 2048^2 shear layer
        dict(_case("step", "shear", 2048, 2048), name="shear_2d_fp64"),
        # the same in single precision
        dict(_case("step", "shear", 2048, 2048, fp32=True, steps=2), name="shear_2d_fp32"),
        # the other solver families on ordinary and ragged grids, walls and periodic sides
        dict(_case("step", "shear", 1021, 1030, solver="EulerHLLC", steps=2), name="shear_2d_hllc"),
        dict(_case("step", "shear", 517, 509, solver="EulerHLL", integrator="RungeKutta2Heun", boundary="MIRROR",
                   steps=5), name="shear_2d_hll"),
        # turbulence-like density field in a closed box, 3D
        dict(_case("step", "lognormal", 160, 144, 136, solver="EulerHLLC", integrator="RungeKutta2TVD",
                   limiter="VanLeer", boundary="MIRROR"), name="lognormal_3d_hllc"),
        # the Roe solver in 3D on a ragged grid
        dict(_case("step", "shear", 99, 90, 86, integrator="RungeKutta3TVD", limiter="Superbee"), name="shear_3d_roe"),
        # self-gravity: the relaxation sweeps of every stage beside the Euler step
        dict(_case("step", "blobs", 1024, 1024, boundary="FREEFLOW", sweeps=20), name="gravity_2d"),
        # a parameter sweep: many uneven problems uploaded, advanced together, read back
        dict(_case("sweep", "quadrants", 256, 32, integrator="RungeKutta2", limiter="Superbee", steps=10, problems=48),
             name="sweep_2d"),
        # a differentiated trajectory: checkpointed forward and its backward
        dict(_case("gradient", "shear", 512, 512, integrator="RungeKutta2", steps=20, every=10), name="gradient_2d"),
        # a host program that hands its state over and takes it back every step
        dict(_case("host", "shear", 2048, 1024), name="host_step_2d"),
    ]


def _span(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run1", "run2", "step2", "step2", "step3", "gravity", "sweep", "gradient", "host"))
    integrator, limiter = rng.choice(INTEGRATORS), rng.choice(LIMITERS)
    solver = rng.choice(("EulerRoe", "EulerRoe", "EulerHLLC", "EulerHLL"))
    boundary = rng.choice(("PERIODIC", "MIRROR", "FREEFLOW"))
    fp32 = rng.random() < .3
    if kind == "run1":
        return _case("run", "sod", _span(rng, 24, 60000), solver=solver, integrator=integrator, limiter=limiter,
                     boundary=rng.choice(("FREEFLOW", "MIRROR")), fp32=fp32, steps=rng.randint(20, 200))
    if kind == "run2":
        return _case("run", "quadrants", _span(rng, 20, 400), _span(rng, 20, 400), solver=solver,
                     integrator=integrator, limiter=limiter, boundary="FREEFLOW", steps=rng.randint(5, 50))
    if kind == "step2":
        return _case("step", "shear", _span(rng, 48, 1800), _span(rng, 48, 1800), solver=solver, integrator=integrator,
                     limiter=limiter, boundary=boundary, fp32=fp32, steps=rng.randint(1, 2))
    if kind == "step3":
        return _case("step", rng.choice(("shear", "lognormal")), _span(rng, 24, 150), _span(rng, 24, 150),
                     _span(rng, 24, 150), solver=rng.choice(("EulerHLLC", "EulerHLL")) if rng.random() < .5 else "EulerRoe",
                     integrator=rng.choice(INTEGRATORS[:3]), limiter=limiter, boundary=boundary, fp32=fp32)
    if kind == "gravity":
        return _case("step", "blobs", _span(rng, 64, 1000), _span(rng, 64, 1000), integrator=rng.choice(INTEGRATORS[1:4]),
                     limiter=limiter, boundary=rng.choice(("PERIODIC", "FREEFLOW")), sweeps=rng.randint(5, 20))
    if kind == "sweep":
        return _case("sweep", "quadrants", rng.randint(96, 256), rng.randint(20, 64), integrator=rng.choice(INTEGRATORS[:4]),
                     limiter=limiter, steps=rng.randint(3, 10), problems=rng.randint(8, 48))
    if kind == "gradient":
        steps = rng.randint(4, 20)
        return _case("gradient", "shear", _span(rng, 64, 512), _span(rng, 64, 512),
                     integrator=rng.choice(INTEGRATORS[1:4]), limiter="MinMod", steps=steps, every=rng.randint(2, steps))
    return _case("host", "shear", _span(rng, 256, 1500), _span(rng, 256, 1500), solver=solver, integrator=integrator,
                 limiter=limiter, fp32=fp32)


# ---------------------------------------------------------------- inputs

def _sizes(case):
    return [s for s in (case["sx"], case["sy"], case["sz"]) if s > 1]


def _gamma(case):
    return 5. / 3. if case["ic"] == "lognormal" else 1.4


def _conserved(gamma, rho, vel, p, fp32=False):
    kinetic = .5 * sum(v * v for v in vel)
    u = np.stack([rho] + [rho * v for v in vel] + [rho * kinetic + p / (gamma - 1)], axis=-1)
    return np.ascontiguousarray(u.astype(np.float32 if fp32 else np.float64))


def _quadrants(rng, sx, sy, gamma, fp32=False):
    q = np.stack([rng.uniform(lo, hi, 4) for lo, hi in ((.5, 2.), (-.6, .6), (-.6, .6), (.5, 2.))])
    at = 2 * (np.arange(sy)[:, None] * 2 > sy) + (np.arange(sx)[None, :] * 2 > sx)
    rho, u, v, p = (q[k][at] for k in range(4))
    return _conserved(gamma, rho, (u, v), p, fp32)


def _initial(case, seed):
    """The initial state, shaped (z, y, x, N) over the active axes."""
    rng = np.random.default_rng(seed)
    sizes, gamma, fp32 = _sizes(case), _gamma(case), case["fp32"]
    shape = tuple(reversed(sizes))
    if case["ic"] == "sod":                       # shock tube, its diaphragm and strength from the seed
        left = np.arange(sizes[0]) < rng.uniform(.4, .6) * sizes[0]
        return _conserved(gamma, np.where(left, rng.uniform(.9, 1.1), .125), (np.zeros(shape),),
                          np.where(left, 1., .1), fp32)
    if case["ic"] == "quadrants":
        return _quadrants(rng, sizes[0], sizes[1], gamma, fp32)
    if case["ic"] == "shear":                     # shear layer with noise
        y = ((np.arange(sizes[1]) + .5) / sizes[1] - .5).reshape((-1, 1))
        x = (np.arange(sizes[0]) + .5) / sizes[0] - .5
        inside = np.broadcast_to(np.abs(y) < .25, shape)
        vel = [np.where(inside, .5, -.5) + rng.uniform(-1e-3, 1e-3, shape),
               .01 * np.sin(4 * math.pi * x) + rng.uniform(-1e-3, 1e-3, shape)]
        vel += [rng.uniform(-1e-3, 1e-3, shape)] * (len(sizes) - 2)
        return _conserved(gamma, np.where(inside, 2., 1.), vel, np.full(shape, 2.5), fp32)
    if case["ic"] == "lognormal":                 # log-normal density, correlated over some cells, at rest
        k2 = sum(np.square(np.fft.fftfreq(n)).reshape([-1 if a == b else 1 for b in range(3)])
                 for a, n in enumerate(shape))
        f = np.fft.ifftn(np.fft.fftn(rng.standard_normal(shape)) * np.exp(-k2 * (2 * math.pi * 4) ** 2 / 2)).real
        rho = np.exp(.5 * (f - f.mean()) / f.std())
        return _conserved(gamma, rho / rho.mean(), [np.zeros(shape)] * 3, np.ones(shape), fp32)
    grid = np.meshgrid(*[(np.arange(n) + .5) / n - .5 for n in shape], indexing="ij")   # blobs: over-densities at rest
    rho = np.ones(shape)
    for _ in range(3):
        centre, height, width = rng.uniform(-.25, .25, len(sizes)), rng.uniform(1., 3.), rng.uniform(.05, .12)
        rho += height * np.exp(-sum((g - c) ** 2 for g, c in zip(grid, centre)) / (2 * width * width))
    return _conserved(gamma, rho, [np.zeros(shape)] * len(sizes), np.full(shape, 10.), fp32)


def _sweep_problems(case, seed):
    """(size x, size y, boundary, state) of every problem: sides from `sy` to `sx` cells."""
    rng = np.random.default_rng(seed)
    shapes = np.random.default_rng(case["problems"])        # the sizes are the case's, the states the seed's
    out = []
    for i in range(case["problems"]):
        sx, sy = (int(round(math.exp(shapes.uniform(math.log(case["sy"]), math.log(case["sx"]))))) for _ in range(2))
        out.append((sx, sy, ("PERIODIC", "FREEFLOW")[i % 2], _quadrants(rng, sx, sy, _gamma(case))))
    return out


def _config(case, sizes, boundary):
    more = {"use_gravity": True, "gauss_seidel_max_iter": case["sweeps"]} if "sweeps" in case else {}
    return _abi.make_config(solver=case["solver"], size=sizes, gamma=_gamma(case), cfl=.4, boundary=boundary,
                            limiter=case["limiter"], integrator=case["integrator"],
                            precision=_abi.FP32 if case["fp32"] else _abi.FP64, **more)


class _OnDevice:
    """The solver's own state buffer, for torch.as_tensor."""

    def __init__(self, solver):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (solver.count,), "typestr": np.dtype(solver.dtype).str,
                                         "data": (solver.state_device_ptr(), False), "version": 3}


def prepare(case, seed):
    if case["kind"] == "sweep":
        problems = _sweep_problems(case, seed)
        batch = hg.Batch([_config(case, p[:2], p[2]) for p in problems])
        batch.set_tuning(tile=(16, 16, 1), staged=1, blocks_per_sm=-1)     # what the autotuner picks for such a sweep
        return {"case": case, "batch": batch, "states": [p[3] for p in problems]}
    u = _initial(case, seed)
    solver = hg.Solver(_config(case, _sizes(case), case["boundary"]))
    st = {"case": case, "solver": solver, "initial": u.reshape(-1)}
    if case["kind"] == "host":
        st["in"] = torch.from_numpy(st["initial"]).pin_memory()
        st["out"] = torch.empty_like(st["in"], pin_memory=True)
        return st
    if case["kind"] in ("step", "gradient"):
        st["state"] = torch.as_tensor(_OnDevice(solver), device="cuda")
    if case["kind"] == "step":
        solver.resetState(st["initial"])
    if case["kind"] == "gradient":
        solver.resetState(st["initial"])
        st["trajectory"] = hg.Checkpoints(solver, case["steps"], case["every"])
        st["cotangent"] = torch.from_numpy(_cotangent(u, seed).reshape(-1)).cuda()
        st["gradient"] = torch.zeros_like(st["cotangent"])
    return st


def _cotangent(u, seed):
    return np.random.default_rng(seed + 1).standard_normal(u.shape)


def run(st):
    case = st["case"]
    if case["kind"] == "sweep":
        batch = st["batch"]
        for i, s in enumerate(st["states"]):
            batch.set_state(i, s)
        batch.update(case["steps"])
        return {"states": np.concatenate([batch.get_state(i) for i in range(batch.n)]), "dts": batch.dts()}
    solver = st["solver"]
    if case["kind"] == "run":
        solver.resetState(st["initial"])
        dt = solver.update(case["steps"])
        return {"state": solver.getState(), "dt": dt}
    if case["kind"] == "step":
        dt = solver.update(case["steps"])
        return {"state": st["state"], "dt": dt}
    if case["kind"] == "host":
        _, dt = solver.update_host(st["in"].numpy(), case["steps"], st["out"].numpy())
        return {"state": st["out"], "dt": dt}
    solver.resetState(st["initial"])
    st["trajectory"].forward()
    st["trajectory"].backward(st["cotangent"].data_ptr(), st["gradient"].data_ptr())
    solver.synchronize()
    return {"state": st["state"], "gradient": st["gradient"]}


def work(case):
    """The state read and written once a step (and the host copies); the scheme's operations, zeros and ones skipped."""
    if case["kind"] == "sweep":
        sizes = [p[:2] for p in _sweep_problems(dict(case, ic="quadrants"), 0)]
        cells, dim = sum(a * b for a, b in sizes), 2
    else:
        dim, cells = len(_sizes(case)), case["sx"] * case["sy"] * case["sz"]
    n, stages, item = dim + 2, len(_TABLES[case["integrator"]][0]), 4 if case["fp32"] else 8
    face_stage = 3 * (2 * n * n - n) + 9 * n if case["solver"] == "EulerRoe" else 12 * n + 40
    flops = cells * (dim * (60 + 10 * n) + stages * (dim * face_stage + n * (2 * dim + 4)))
    state = cells * n * item
    moved = 2 * state
    if "sweeps" in case:
        flops += cells * stages * case["sweeps"] * (3 * dim + 2)
        moved += 2 * cells * item
    total = {"bytes": moved * case["steps"], "flops": flops * case["steps"]}
    if case["kind"] == "gradient":
        return {"bytes": 3 * total["bytes"], "flops": 4 * total["flops"]}
    return total


# ---------------------------------------------------------------- the schemes in 64 bits

_TABLES = {   # Shu-Osher rows: the input of stage m + 1 is sum_k alpha[m][k] u_k + beta[m][k] dt L(u_k)
    "ForwardEuler": ([[1]], [[1]]),
    "RungeKutta2": ([[1], [1, 0]], [[.5], [0, 1]]),
    "RungeKutta2Heun": ([[1], [1, 0]], [[1], [.5, .5]]),
    "RungeKutta4": ([[1], [1, 0], [1, 0, 0], [1, 0, 0, 0]],
                    [[.5], [0, .5], [0, 0, 1], [1 / 6, 2 / 6, 2 / 6, 1 / 6]]),
    "RungeKutta2TVD": ([[1], [.5, .5]], [[1], [0, .5]]),
    "RungeKutta3TVD": ([[1], [3 / 4, 1 / 4], [1 / 3, 2 / 3, 0]], [[1], [0, 1 / 4], [0, 0, 2 / 3]]),
}


def _limited(name, r):
    zero, lo, hi = torch.zeros_like(r), torch.fmin, torch.fmax      # a NaN ratio yields the other operand
    c = lambda v: torch.full_like(r, v)                             # noqa: E731
    if name == "MinMod":
        return hi(zero, lo(r, c(1.)))
    if name == "Superbee":
        return hi(zero, hi(lo(c(1.), 2 * r), lo(c(2.), r)))
    if name == "MonotizedCentral":
        return hi(zero, lo(c(2.), lo(.5 * (1 + r), 2 * r)))
    if name == "Koren":
        return hi(zero, lo(2 * r, lo((1 + 2 * r) / 3, c(2.))))
    return zero                                                     # DonorCell


class _Scheme:
    """One problem in 64 bits; fields have the grid's axes first, components last."""

    def __init__(self, case, sizes, boundary, device):
        self.case, self.sizes, self.dim, self.device = case, sizes, len(sizes), device
        self.boundary = boundary
        f = np.float32 if case["fp32"] else np.float64
        self.dx = [float("%g" % float((f(.5) - f(-.5)) / f(n))) for n in sizes]
        self.gamma, self.cfl = float(f(_gamma(case))), float(np.float32(.4))
        self.shape = tuple(reversed(sizes))
        self.interior = self._cells(lambda side, a: (2, 2))
        self.phi = None

    def _axis(self, side):
        return self.dim - 1 - side

    def _cells(self, bounds, side=None):
        m = torch.ones(self.shape, dtype=torch.bool, device=self.device)
        for a in range(self.dim):
            lo, hi = bounds(side, a)
            i = torch.arange(self.sizes[a], device=self.device)
            m = m & ((i >= lo) & (i < self.sizes[a] - hi)).reshape([-1 if self._axis(a) == d else 1 for d in range(self.dim)])
        return m

    def _faces(self, side):          # the faces the divergence of the interior reads
        return self._cells(lambda s, a: (2, 1 if a == s else 2), side)

    def _below(self, x, side):
        return torch.roll(x, 1, self._axis(side))

    def _above(self, x, side):
        return torch.roll(x, -1, self._axis(side))

    def ghosts(self, u, scalar=False):
        for side in range(self.dim):
            n, axis = self.sizes[side], self._axis(side)
            src = torch.arange(n)
            sign = torch.ones(n, 1 if scalar else self.dim + 2, dtype=torch.float64)
            ends = {"PERIODIC": (n - 4, n - 3, 2, 3), "FREEFLOW": (2, 2, n - 3, n - 3), "MIRROR": (3, 2, n - 3, n - 4)}
            edge = [0, 1, n - 2, n - 1]
            src[edge] = torch.tensor(ends[self.boundary])
            if self.boundary == "MIRROR" and not scalar:
                sign[edge, 1 + side] = -1.
            u = torch.index_select(u, axis, src.to(self.device))
            u = u * sign.to(self.device).reshape([n if d == axis else 1 for d in range(self.dim)] + [-1])
        return u

    def _primitives(self, u):
        rho = u[..., 0]
        v = u[..., 1:1 + self.dim] / rho[..., None]
        e = u[..., -1] / rho
        inner = e - .5 * (v * v).sum(-1)
        if self.phi is not None:
            inner = inner - self.phi[..., 0]
        p = (self.gamma - 1) * rho * inner
        return rho, v, p, e + p / rho

    def _roe_average(self, side, prim):
        rho, v, _, h = prim
        w = torch.sqrt(rho)
        wl = self._below(w, side)
        mean = lambda x: (wl * self._below(x, side) + w * x) / (wl + w)         # noqa: E731
        v = torch.stack([mean(v[..., k]) for k in range(self.dim)], -1)
        h = mean(h)
        c2 = h - .5 * (v * v).sum(-1)
        if self.phi is not None:
            c2 = c2 - mean(self.phi[..., 0])
        return v, h, torch.sqrt(c2 * (self.gamma - 1))

    def _basis(self, side, prim):
        """Eigenvalues and both eigenvector matrices of the faces along `side`."""
        v, h, c = self._roe_average(side, prim)
        g1, n = self.gamma - 1, self.dim + 2
        order = [side] + [k for k in range(self.dim) if k != side]              # the normal velocity first
        vx, vt = v[..., order[0]], [v[..., k] for k in order[1:]]
        vv, one, zero = (v * v).sum(-1), torch.ones_like(vx), torch.zeros_like(vx)
        at = [0] + [1 + k for k in order] + [n - 1]                             # where a row's entries belong
        def put(rows):
            m = [[zero] * n for _ in range(n)]
            for i, row in enumerate(rows):
                for j, x in enumerate(row):
                    m[i][at[j]] = x
            return torch.stack([torch.stack(r, -1) for r in m], -2)
        unit = lambda j: [one if j == k else zero for k in range(self.dim - 1)]  # noqa: E731
        s = .5 / (c * c)
        left = [[(.5 * g1 * vv + c * vx) * s, -(c + g1 * vx) * s] + [-g1 * t * s for t in vt] + [g1 * s],
                [1 - g1 * vv * s, 2 * g1 * vx * s] + [2 * g1 * t * s for t in vt] + [-2 * g1 * s]]
        left += [[-vt[j], zero] + unit(j) + [zero] for j in range(self.dim - 1)]
        left += [[(.5 * g1 * vv - c * vx) * s, (c - g1 * vx) * s] + [-g1 * t * s for t in vt] + [g1 * s]]
        right = [[one, vx - c] + vt + [h - c * vx], [one, vx] + vt + [.5 * vv]]  # its columns
        right += [[zero, zero] + unit(j) + [vt[j]] for j in range(self.dim - 1)]
        right += [[one, vx + c] + vt + [h + c * vx]]
        lam = torch.stack([vx - c] + [vx] * self.dim + [vx + c], -1)
        return lam, put(left), put(right).transpose(-1, -2)

    def _flux_roe(self, side, u, dt):
        lam, left, right = self.frozen[side]
        mask = self._faces(side)[..., None]
        ul = self._below(u, side)
        apply = lambda m, x: torch.einsum("...ij,...j->...i", m, x)              # noqa: E731
        dq = torch.where(mask, apply(left, u - ul), 0.)
        up = lam >= 0
        theta = torch.where(up, 1., -1.).to(u.dtype)
        upwind = torch.where(up, self._below(dq, side), self._above(dq, side))
        flat = dq == 0                       # an infinite or NaN ratio picks a branch and carries no derivative
        r = torch.where(flat, (upwind / dq).detach(), upwind / torch.where(flat, 1., dq))
        fine = torch.isfinite(r)
        phi = torch.where(fine, _limited(self.case["limiter"], torch.where(fine, r, 0.)),
                          _limited(self.case["limiter"], r).detach())
        f = lam * apply(left, .5 * (u + ul)) - .5 * lam * dq * (theta + phi * (lam * dt / self.dx[side] - theta))
        return torch.where(mask, apply(right, f), 0.)

    def _waves(self, side, prim):
        rho, v, p, h = prim
        g1, vx, bel = self.gamma - 1, v[..., side], lambda x: self._below(x, side)
        c = torch.sqrt(g1 * (h - .5 * (v * v).sum(-1)))
        if self.case["solver"] == "EulerHLL":
            va, _, ca = self._roe_average(side, prim)
            sl, sr = torch.fmin(bel(vx - c), va[..., side] - ca), torch.fmax(vx + c, va[..., side] + ca)
        else:
            star = torch.clamp(.5 * (bel(p) + p) - (vx - bel(vx)) * (bel(rho) + rho) * (bel(c) + c) / 8, min=0.)
            q = lambda p: torch.where(star <= p, 1., torch.sqrt(1 + (self.gamma + 1) / (2 * self.gamma) * (star / p - 1)))  # noqa: E731
            sl, sr = bel(vx) - bel(c) * q(bel(p)), vx + c * q(p)
        known = self._cells(lambda s, a: (2, 1))
        return torch.where(known, sl, 0.), torch.where(known, sr, 0.)

    def _flux_hll(self, side, u, dt):
        sl, sr = (x[..., None] for x in self.frozen[side])
        rho, v, p, h = self._primitives(u)
        vx = v[..., side]
        f = u * vx[..., None]
        f[..., 1 + side] += p
        f[..., -1] = rho * h * vx
        bel = lambda x: self._below(x, side)                                     # noqa: E731
        fl, ul = bel(f), bel(u)
        if self.case["solver"] == "EulerHLL":
            mid = (sr * fl - sl * f + sl * sr * (u - ul)) / (sr - sl)
            out = torch.where(sl >= 0, fl, torch.where(sr >= 0, mid, f))
        else:
            rl, vl, pl = bel(rho)[..., None], bel(vx)[..., None], bel(p)[..., None]
            rr, vr, pr = rho[..., None], vx[..., None], p[..., None]
            s = (rr * vr * (sr - vr) - rl * vl * (sl - vl) + pl - pr) / (rr * (sr - vr) - rl * (sl - vl))
            plr = .5 * (pl + pr + rl * (sl - vl) * (s - vl) + rr * (sr - vr) * (s - vr))
            e = torch.zeros_like(u)
            e[..., 1 + side], e[..., -1:] = 1., s
            inner = lambda w, us, fs: (s * (w * us - fs) + w * plr * e) / (w - s)   # noqa: E731
            out = torch.where(sl >= 0, fl, torch.where(s >= 0, inner(sl, ul, fl), torch.where(sr >= 0, inner(sr, u, f), f)))
        return torch.where(self._faces(side)[..., None], out, 0.)

    def _rows(self, u, dt, derivative):
        us, ds = [u], []
        for alpha, beta in zip(*_TABLES[self.case["integrator"]]):
            ds.append(derivative(us[-1]) if any(row[len(ds)] for row in _TABLES[self.case["integrator"]][1]
                                                if len(row) > len(ds)) else torch.zeros_like(u))
            us.append(sum(a * x for a, x in zip(alpha, us) if a) + sum(b * dt * x for b, x in zip(beta, ds) if b))
        return us[-1]

    def step(self, u, dt=None):
        """(the next state, dt); the timestep is the CFL condition's unless given."""
        u = self.ghosts(u)
        prim = self._primitives(u)
        roe = self.case["solver"] == "EulerRoe"
        self.frozen = [self._basis(s, prim) if roe else self._waves(s, prim) for s in range(self.dim)]
        if dt is None:
            dt = math.inf
            for s in range(self.dim):
                lo, hi = (self.frozen[s][0][..., 0], self.frozen[s][0][..., -1]) if roe else self.frozen[s]
                speed = torch.clamp(hi, min=0.) - torch.clamp(self._above(lo, s), max=0.) + (1e-9 if roe else 0.)
                cells = self.interior if roe else self._cells(lambda _, a: (2, 1))
                dt = min(dt, self.dx[s] / float(speed[cells].max()))
            dt = dt * self.cfl
        flux = self._flux_roe if roe else self._flux_hll

        def divergence(x):
            d = torch.zeros_like(x)
            for s in range(self.dim):
                f = flux(s, x, dt)
                d = d - (self._above(f, s) - f) / self.dx[s]
            return torch.where(self.interior[..., None], d, 0.)

        out = self._rows(u, dt, divergence)
        if self.phi is not None:
            if self.case["integrator"] == "ForwardEuler":
                out = self.ghosts(out)
            return self._rows(out, dt, self._gravity), dt
        return (self.ghosts(out) if self.case["integrator"] == "ForwardEuler" else out), dt

    def attract(self, u):
        """Self-gravity from now on: the potential starts as -density and is relaxed."""
        self.phi = -u[..., :1]
        u = torch.cat([u[..., :-1], u[..., -1:] + self.phi], -1)
        self._relax(u, 100 * self.case["sweeps"])
        return u

    def _relax(self, u, sweeps):
        inside = tuple(slice(2, n - 2) for n in self.shape)
        rhs = 4 * math.pi * u[inside][..., 0]
        diag = -2. * sum(1 / (d * d) for d in self.dx)
        parity = sum(torch.arange(n - 4, device=self.device).reshape([-1 if a == d else 1 for d in range(self.dim)])
                     for a, n in enumerate(self.shape)) % 2 == 0
        for i in range(sweeps):
            if i == sweeps - 1:
                self.phi = self.ghosts(self.phi, scalar=True)
            p = self.phi[inside][..., 0]
            for colour in (parity, ~parity):
                skew = torch.zeros_like(p)
                for s in range(self.dim):
                    a, n, d2 = self._axis(s), self.sizes[s] - 4, self.dx[s] ** 2
                    skew.narrow(a, 0, n - 1).add_(p.narrow(a, 1, n - 1) / d2)
                    skew.narrow(a, 1, n - 1).add_(p.narrow(a, 0, n - 1) / d2)
                p = torch.where(colour, (rhs - skew) / diag, p)
            self.phi[inside] = p[..., None]

    def _gravity(self, u):
        self._relax(u, self.case["sweeps"])
        d = torch.zeros_like(u)
        for s in range(self.dim):
            pull = -(self._above(self.phi, s) - self._below(self.phi, s))[..., 0] / (2 * self.dx[s]) * u[..., 0]
            d[..., 1 + s] -= pull
            d[..., -1] -= pull * u[..., 1 + s]
        return torch.where(self.interior[..., None], d, 0.)


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "sweep":
        states, dts = [], []
        for sx, sy, boundary, u in _sweep_problems(case, seed):
            scheme, u = _Scheme(case, [sx, sy], boundary, device), torch.from_numpy(u).to(device)
            for _ in range(case["steps"]):
                u, dt = scheme.step(u)
            states.append(u.reshape(-1))
            dts.append(dt)
        return {"states": torch.cat(states), "dts": np.array(dts)}
    scheme = _Scheme(case, _sizes(case), case["boundary"], device)
    first = torch.from_numpy(_initial(case, seed)).to(device).double()
    u, dts = first, []
    if "sweeps" in case:
        u = scheme.attract(u)
    for _ in range(case["steps"]):
        u, dt = scheme.step(u)
        dts.append(dt)
    if case["kind"] != "gradient":
        return {"state": u.reshape(-1), "dt": dts[-1]}
    back = torch.from_numpy(_cotangent(first, seed)).to(device)
    at = [first]
    for dt in dts:                          # the states before each step, then one step's gradient at a time
        at.append(scheme.step(at[-1], dt)[0])
    for x, dt in zip(reversed(at[:-1]), reversed(dts)):
        x = x.detach().requires_grad_(True)
        back, = torch.autograd.grad(scheme.step(x, dt)[0], x, back)
    return {"state": u.reshape(-1), "gradient": back.reshape(-1)}
