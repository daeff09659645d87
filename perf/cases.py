"""Measured workloads of the ensemble engine.

Each case is one call a program makes through the package's public entry points:

  simulate   ``Context.simulate``: host arrays in, ensemble mean out (the drop-in for the
             reference's per-particle simulation loop)
  resident   ``Context.ensemble``: an ensemble kept on the device, advanced in pieces, read once
  serve      ``Context.server``: parameter sets submitted together, results awaited

The particles and fields are those of ``stochasticphysics_b200.provider``; the runs are cut to
a few windows so that a pass stays short.  The Brown+Neel, analytic-midpoint and batched runs
take a smaller time step than the workloads', as a convergence study does: there the paths of
two programs agree over thousands of steps, where at the workloads' steps a last-bit
difference grows by many orders of magnitude.  ``exact`` integrates the same ensembles in 64
bits with plain torch operations: the Philox4x32-10 stream of every particle and step, the
reference's step formulas and the moment-weighted mean.
"""
import dataclasses
import math

import numpy as np
import torch

import stochasticphysics_b200 as sp
from stochasticphysics_b200 import provider
from stochasticphysics_b200._abi import Anisotropy, Jacobian, Noise, Precision, Problem, Solver

SOLVERS = {"em": Solver.EulerMaruyama, "heun": Solver.Heun_Strong, "milstein": Solver.Millstein,
           "midpoint": Solver.Implicit_Midpoint, "midpoint_exact": Solver.Implicit_Midpoint}
PROBLEMS = {"neel": Problem.Neel, "neel_spherical": Problem.NeelSpherical,
            "brown_neel": Problem.BrownAndNeelEulerSpherical, "brown_neel_cartesian": Problem.BrownAndNeel,
            "neel_cubic": Problem.Neel}

# additions and multiplications of one particle-step (FMA = 2), transcendentals and noise left
# out; the implicit steps with the Newton iterations these ensembles take
FLOPS = {("neel", "em"): 131, ("neel", "heun"): 200, ("neel", "milstein"): 139,
         ("neel_spherical", "em"): 88, ("neel_spherical", "heun"): 150, ("neel_spherical", "milstein"): 95,
         ("brown_neel", "em"): 476, ("brown_neel", "heun"): 703, ("brown_neel", "milstein"): 492,
         ("brown_neel_cartesian", "heun"): 525, ("brown_neel_cartesian", "milstein"): 370,
         ("neel_cubic", "midpoint"): 7572, ("neel_cubic", "midpoint_exact"): 1600}

# time steps (s)
DT = {"neel": 1e-11, "neel_spherical": 1e-11, "brown_neel": 2.5e-12, "brown_neel_cartesian": 2.5e-12,
      "midpoint": 1e-10, "midpoint_exact": 1e-11, "serve": 2e-12}


def _case(name, call, model, solver, precision, n, steps, window, noise="philox", sets=1):
    case = {"call": call, "model": model, "solver": solver, "precision": precision, "n": n, "steps": steps,
            "window": window, "noise": noise, "sets": sets}
    return {"name": name, **case} if name else case


def listed():
    return [
        # a parameter scan's smallest call: one warp-pair of particles, a short run; the call's own cost counts
        _case("neel_heun_fp64_64", "simulate", "neel", "heun", "fp64", 64, 2000, 100),
        # the plain Neel relaxation of 1024 particles, too few to fill the GPU: the step's latency counts
        _case("neel_heun_fp64_1024", "simulate", "neel", "heun", "fp64", 1024, 12000, 100),
        # spherical Neel coordinates with the pole rotation, an odd particle count
        _case("neel_spherical_em_fp64_30011", "simulate", "neel_spherical", "em", "fp64", 30011, 2000, 500),
        # coupled Brown+Neel in Cartesian form, an ensemble that fills the GPU and leaves a ragged tile
        _case("brown_neel_cartesian_heun_fp64_100003", "simulate", "brown_neel_cartesian", "heun", "fp64", 100003,
              3000, 500),
        # the coupled Brown+Neel workload in its drop-in precision: full size, and a ragged mid-size ensemble
        _case("brown_neel_milstein_fp64_65536", "simulate", "brown_neel", "milstein", "fp64", 65536, 5000, 1000),
        _case("brown_neel_heun_fp64_20001", "resident", "brown_neel", "heun", "fp64", 20001, 4000, 500),
        # the same workload in single precision, full size and an ensemble four times larger
        _case("brown_neel_milstein_fp32_65536", "simulate", "brown_neel", "milstein", "fp32", 65536, 9000, 1000),
        _case("brown_neel_heun_fp32_262144", "simulate", "brown_neel", "heun", "fp32", 262144, 4000, 1000),
        # the stiff path: cubic anisotropy, implicit midpoint with the reference's Newton matrix, largest work
        _case("cubic_midpoint_fp64_262144", "simulate", "neel_cubic", "midpoint", "fp64", 262144, 400, 100),
        # the same step with the analytic Newton matrix
        _case("cubic_midpoint_exact_fp64_65537", "simulate", "neel_cubic", "midpoint_exact", "fp64", 65537, 1200, 100),
        # caller-supplied Wiener increments: a run compared path by path with another program
        _case("neel_heun_injected_fp64_16384", "simulate", "neel", "heun", "fp64", 16384, 300, 50, noise="injected"),
        # a batch of parameter sets of uneven sizes through the server
        _case("neel_batch_fp32_24", "serve", "neel", "heun", "fp32", 0, 4000, 1000, sets=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["neel", "neel", "neel_spherical", "brown_neel", "brown_neel", "brown_neel_cartesian",
                       "neel_cubic", "injected", "serve"])
    if kind == "serve":
        return _case("", "serve", "neel", "heun", rng.choice(["fp64", "fp32"]), 0, 1000 * rng.randint(2, 5), 1000,
                     sets=rng.randint(2, 24))
    if kind == "injected":
        n = _log(rng, 500, 16384)
        return _case("", "simulate", "neel", rng.choice(["em", "heun", "milstein"]), rng.choice(["fp64", "fp32"]), n,
                     50 * rng.randint(3, 6), 50, noise="injected")
    call = rng.choice(["simulate", "simulate", "resident"])
    if kind == "neel_cubic":
        return _case("", call, kind, rng.choice(["midpoint", "midpoint_exact"]), "fp64", _log(rng, 1000, 200000),
                     100 * rng.randint(2, 4), 100)
    precision = rng.choice(["fp64", "fp64", "fp32"])
    solver = rng.choice(["heun", "milstein"] if kind == "brown_neel_cartesian" else ["em", "heun", "milstein"])
    n = _log(rng, 64, 100000) if precision == "fp64" else _log(rng, 1000, 262144)
    window = rng.choice([100, 250, 500])
    return _case("", call, kind, solver, precision, n, window * rng.randint(3, 2000 // window), window)


# ------------------------------------------------------------------ the calls
def _specs(case, seed):
    seed = 0x5EED0000 + 7919 * int(seed)
    precision = Precision.FP32 if case["precision"] == "fp32" else Precision.FP64
    n, steps, window = case["n"], case["steps"], case["window"]
    common = dict(steps=steps, oversampling=window, precision=precision, seed=seed)
    if case["call"] == "serve":
        # sizes of the batched workload; every set runs `steps` steps
        sets = provider.batched_sets(case["sets"], seed=seed, precision=precision, step_scale=1e-9, oversampling=window)
        return [dataclasses.replace(s, number_of_steps=steps, timestep=DT["serve"]) for s in sets]
    model, solver = case["model"], SOLVERS[case["solver"]]
    if model == "neel_cubic":
        spec = provider.cubic_implicit(n, dt=DT[case["solver"]], **common)
        if case["solver"] == "midpoint_exact":
            spec = dataclasses.replace(spec, jacobian=Jacobian.Exact)
    elif model in ("neel", "neel_spherical"):
        spec = provider.neel_relaxation(n, solver=solver, dt=DT[model], **common)
        if model == "neel_spherical":
            spec = dataclasses.replace(spec, problem=Problem.NeelSpherical, use_coordinate_transformation=True,
                                       min_angle_before_transformation=math.pi / 36)
    else:
        spec = provider.brown_neel_relaxation(n, solver=solver, dt=DT[model], **common)
        if model == "brown_neel_cartesian":
            axis = provider.easy_axis(Problem.BrownAndNeel, spec.orientation)
            m0 = provider.along_axis_random_sign(np.random.default_rng(seed), axis)
            spec = dataclasses.replace(spec, problem=Problem.BrownAndNeel, magnetisation=m0,
                                       use_euler_coordinate_transformation=False,
                                       use_spherical_coordinate_transformation=False)
    if case["noise"] == "injected":
        spec = provider.with_injected_noise(spec, seed=seed + 1)
    return [spec]


def prepare(case, seed):
    ctx = sp.Context(0)
    state = {"case": case, "ctx": ctx, "specs": _specs(case, seed)}
    if case["call"] == "serve":
        state["server"] = ctx.server()
    return state


def _outputs(result, single):
    # the library hands every result over in double arrays; the single-precision form's window
    # means carry the accuracy of its 32-bit states and are kept as such
    mean = result.mean.astype(np.float32) if single else result.mean
    return {"mean": mean, "weight": result.weight, "time": result.time, "field": result.field}


def run(state):
    case, ctx, specs = state["case"], state["ctx"], state["specs"]
    single = case["precision"] == "fp32"
    if case["call"] == "serve":
        server = state["server"]
        results = [server.wait(rid)[0] for rid in server.submit_many(specs)]
        return [{"mean": o["mean"], "weight": o["weight"]} for o in (_outputs(r, single) for r in results)]
    if case["call"] == "resident":
        with ctx.ensemble(specs[0]) as ens:
            total = specs[0].integrated_steps
            done = total // 2 // case["window"] * case["window"]
            ens.advance(done)
            ens.advance(total - done)
            return [_outputs(ens.read(), single)]
    return [_outputs(ctx.simulate(specs[0]), single)]


def _work_sizes(case):
    """(particles, integrated steps) of every ensemble of the case."""
    if case["call"] != "serve":
        return [(case["n"], case["steps"] - case["window"])]
    # the batched workload draws n log-uniformly from 1e3 to 6.4e4: its mean
    n = (6.4e4 - 1e3) / math.log(64.0)
    return [(n, case["steps"] - case["window"])] * case["sets"]


def work(case):
    flops = FLOPS[case["model"], case["solver"]]
    outputs = 9 if case["model"] == "brown_neel" else 6 if case["model"] == "brown_neel_cartesian" else 3
    real = 8
    total = {"bytes": 0.0, "flops": 0.0}
    for n, steps in _work_sizes(case):
        total["flops"] += flops * float(n) * steps
        total["bytes"] += 13.0 * real * n + real * (case["steps"] // case["window"]) * (outputs + 4)
        if case["noise"] == "injected":
            total["bytes"] += 3.0 * real * n * steps
    return total


# ------------------------------------------------------------------ 64-bit restatement
# seconds of one particle-step of the restatement below, for the 20-second limit
_COST = {"neel": 5e-7, "neel_spherical": 8e-7, "brown_neel": 2e-6, "brown_neel_cartesian": 9e-7, "neel_cubic": 1.5e-5}


def exact(case, seed):
    spent = sum(steps * (max(n, 2000) * _COST[case["model"]]) for n, steps in _work_sizes(case))
    if spent > 15.0:
        return None
    kept = ("mean", "weight") if case["call"] == "serve" else ("mean", "weight", "time", "field")
    return [{k: v for k, v in _integrate(spec).items() if k in kept} for spec in _specs(case, seed)]


def _t(a):
    return torch.from_numpy(np.array(a, dtype=np.float64))


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def _lin(*terms):
    """sum of scalar * vector over (scalar, vector) pairs"""
    return tuple(sum(s * v[i] for s, v in terms) for i in range(3))


def _philox(counter, key):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF
    c, (k0, k1) = list(counter), key
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _normals(seed, n, step, m):
    pid = torch.arange(n, dtype=torch.int64)
    key = (seed & 0xFFFFFFFF, seed >> 32 & 0xFFFFFFFF)
    out = []
    for call in range(2 if m > 3 else 1):
        zero = torch.zeros_like(pid)
        w = _philox([zero + (step & 0xFFFFFFFF), zero + (step >> 32), pid, zero + (call << 24)], key)
        u = [(x.to(torch.float64) + 0.5) * 2.0 ** -32 for x in w]
        for a, b in ((0, 1), (2, 3)):
            r = torch.sqrt(-2.0 * torch.log(u[a]))
            out += [r * torch.cos(2.0 * math.pi * u[b]), r * torch.sin(2.0 * math.pi * u[b])]
    return out[:m]


def _euler_axes(e, brown):
    """body axes of the ZXZ Euler angles, as rows (Neel problems) or columns (coupled ones)"""
    (sf, st, ss), (cf, ct, cs) = [torch.sin(x) for x in e], [torch.cos(x) for x in e]
    m = [[cf * cs - ct * sf * ss, -sf * cs - ct * cf * ss, st * ss],
         [ct * sf * cs + cf * ss, ct * cf * cs - sf * ss, -st * cs],
         [st * sf, st * cf, ct]]
    return [tuple(m[j][i] for j in range(3)) for i in range(3)] if brown else [tuple(r) for r in m]


class _Physics:
    """Per-particle prefactors, derived from the particle properties in SI units."""

    def __init__(self, s):
        kb = 1.3806485279e-23
        full = lambda v: _t(np.broadcast_to(np.asarray(v, dtype=np.float64), (s.n,)))  # noqa: E731
        self.spec, self.dt = s, s.timestep
        r, ms, alpha, gamma = (full(v) for v in (s.magnetic_radius, s.saturation_magnetisation, s.damping_constant,
                                                 s.gyromagnetic_ratio))
        k = full(s.anisotropy_constant)
        volume = 4.0 / 3.0 * math.pi * r ** 3
        self.moment = volume * ms
        diff = 2.0 * alpha * kb * s.temperature / (gamma * self.moment)
        self.a = -gamma / (1.0 + alpha * alpha)
        self.b = self.a.abs() * alpha
        self.dn = torch.sqrt(diff)
        self.dp = -(self.a ** 2) * (1.0 + alpha * alpha) * diff
        self.twoalpha = 2.0 * alpha
        self.pf = -2.0 * k / ms
        self.euler = [_t(s.orientation[:, i]) for i in range(3)]
        self.mag = [_t(s.magnetisation[:, i]) for i in range(3)]
        if s.problem in (Problem.BrownAndNeel, Problem.BrownAndNeelEulerSpherical):
            friction = 6.0 * full(s.viscosity) * (4.0 / 3.0 * math.pi * full(s.hydrodynamic_radius) ** 3)
            c = 1.0 / friction
            self.cf = c * torch.sqrt(2.0 * kb * s.temperature * friction)
            self.d = c * self.moment
            self.bpd = self.b + self.d
            self.ct = c * (-2.0 * k * volume)

    def field(self, t):
        f = self.spec.field
        s = math.sin(2.0 * math.pi * f.frequency[0] * t + f.phase[0])
        return tuple(f.amplitude[i] * s + f.offset[i] for i in range(3))

    def weights(self, out):
        axis = self.spec.problem == Problem.BrownAndNeel
        return [torch.ones_like(self.moment) if axis and i < 3 else self.moment for i in range(out)]

    def heff(self, m, axes, B):
        x, y, z = axes
        if self.spec.anisotropy == Anisotropy.Uniaxial:
            h = _lin((self.pf * _dot(m, z), z))
        else:
            c = [_dot(m, v) for v in axes]
            h = _lin((self.pf * c[0] * (c[1] ** 2 + c[2] ** 2), x), (self.pf * c[1] * (c[0] ** 2 + c[2] ** 2), y),
                     (self.pf * c[2] * (c[0] ** 2 + c[1] ** 2), z))
        return tuple(h[i] + B[i] for i in range(3))


class _Neel(_Physics):
    noise, out = 3, 3

    def __init__(self, s):
        super().__init__(s)
        self.axes = _euler_axes(self.euler, False)
        norm = torch.sqrt(_dot(self.mag, self.mag))
        self.y = [m / norm for m in self.mag]

    def chart(self, y):
        return y, None

    def det(self, y, c, B):
        u = _cross(y, self.heff(y, self.axes, B))
        return _lin((self.a, u), (-self.b, _cross(y, u)))

    def drift(self, y, c):
        return [self.dp * v for v in y]

    def noise_term(self, y, c, w):
        return _lin((self.b * self.dn, w), (-self.b * self.dn * _dot(y, w), y), (self.a * self.dn, _cross(y, w)))

    def finish(self, y, c):
        return list(y)

    def output(self, y):
        return y

    def newton_matrix(self, m, B, w):
        """-I + dt/2 J_det + 1/2 J_sto at the midpoint m, [n][3][3]."""
        zero, n = torch.zeros_like(m[0]), self.spec.n

        def skew(v):
            return torch.stack([torch.stack([zero, -v[2], v[1]], -1), torch.stack([v[2], zero, -v[0]], -1),
                                torch.stack([-v[1], v[0], zero], -1)], -2)

        col = lambda v: v[:, None, None]  # noqa: E731
        h = self.heff(m, self.axes, B)
        eye = torch.eye(3, dtype=torch.float64).expand(n, 3, 3)
        mx, hx, wx = skew(m), skew(h), skew(w)
        exact = self.spec.jacobian == Jacobian.Exact
        if self.spec.anisotropy == Anisotropy.Uniaxial:
            z = torch.stack(self.axes[2], -1)
            jh = col(self.pf) * z[:, :, None] * z[:, None, :]
        elif not exact:
            jh = eye
        else:
            a = torch.stack([torch.stack(v, -1) for v in self.axes], -2)  # rows: body axes
            c = torch.stack([_dot(m, v) for v in self.axes], -1)
            g = 2.0 * c[:, :, None] * c[:, None, :]
            g = g - torch.diag_embed(torch.diagonal(g, dim1=1, dim2=2)) + torch.diag_embed((c * c).sum(-1, keepdim=True) - c * c)
            jh = col(self.pf) * (a.transpose(1, 2) @ g @ a)
        p1, p2 = col(self.a * self.dn), col(self.b * self.dn)
        if not exact:
            jd = col(self.a) * (mx @ jh - hx) - col(self.twoalpha / self.dt) * mx
            js = -p1 * wx
        else:
            ju = mx @ jh - hx
            jd = col(self.a) * ju - col(self.b) * (mx @ ju - skew(_cross(m, h)))
            mv, wv = torch.stack(m, -1), torch.stack(w, -1)
            js = -p2 * (col(_dot(m, w)) * eye + mv[:, :, None] * wv[:, None, :]) - p1 * wx
        return -eye + 0.5 * self.dt * jd + 0.5 * js


class _NeelSpherical(_Physics):
    noise, out = 3, 3

    def __init__(self, s):
        super().__init__(s)
        self.axes = _euler_axes(self.euler, False)
        self.y = [torch.acos(self.mag[2]), torch.atan2(self.mag[1], self.mag[0])]
        self.lo = s.min_angle_before_transformation if s.use_coordinate_transformation else -1.0

    def chart(self, y):
        rot = (y[0] < self.lo) | (y[0] > math.pi - self.lo) if self.lo >= 0 else torch.zeros_like(y[0], dtype=torch.bool)
        return _pole_rotate(y, rot), rot

    def _frame(self, y, rot):
        st, ct, sf, cf = torch.sin(y[0]), torch.cos(y[0]), torch.sin(y[1]), torch.cos(y[1])
        return st, ct, sf, cf, _spherical(st, ct, sf, cf, rot)

    def _project(self, st, ct, sf, cf, rot):
        zero = torch.zeros_like(st)
        pick = lambda a, b: tuple(torch.where(rot, p, q) for p, q in zip(a, b))  # noqa: E731
        eth = pick((st, ct * sf, ct * cf), (ct * cf, ct * sf, -st))
        eph = pick((zero, cf, -sf), (-sf, cf, zero))
        return (_lin((-self.a, eph), (self.b, eth)), _lin((self.a / st, eth), (self.b / st, eph)))

    def det(self, y, rot, B):
        st, ct, sf, cf, m = self._frame(y, rot)
        h = self.heff(m, self.axes, B)
        return [_dot(p, h) for p in self._project(st, ct, sf, cf, rot)]

    def drift(self, y, rot):
        return [-0.5 * self.dp * torch.cos(y[0]) / torch.sin(y[0]), torch.zeros_like(y[0])]

    def noise_term(self, y, rot, w):
        st, ct, sf, cf, _ = self._frame(y, rot)
        return [self.dn * _dot(p, w) for p in self._project(st, ct, sf, cf, rot)]

    def finish(self, y, rot):
        return _pole_unrotate(y, rot)

    def output(self, y):
        none = torch.zeros_like(y[0], dtype=torch.bool)
        return list(self._frame(y, none)[4])


def _spherical(st, ct, sf, cf, rot):
    return tuple(torch.where(rot, a, b) for a, b in ((-ct, st * cf), (st * sf, st * sf), (st * cf, ct)))


def _pole_rotate(y, rot):
    st, ct, sf, cf = torch.sin(y[0]), torch.cos(y[0]), torch.sin(y[1]), torch.cos(y[1])
    return [torch.where(rot, torch.acos(-cf * st), y[0]), torch.where(rot, torch.atan2(sf * st, ct), y[1])]


def _pole_unrotate(y, rot):
    st, ct, sf, cf = torch.sin(y[0]), torch.cos(y[0]), torch.sin(y[1]), torch.cos(y[1])
    return [torch.where(rot, torch.acos(cf * st), torch.fmod(y[0], 2.0 * math.pi)),
            torch.where(rot, torch.atan2(sf * st, -ct), torch.fmod(y[1], 2.0 * math.pi))]


class _BrownNeelEuler(_Physics):
    noise, out = 6, 9

    def __init__(self, s):
        super().__init__(s)
        self.y = [*self.euler, torch.acos(self.mag[2]), torch.atan2(self.mag[1], self.mag[0])]
        self.brown = s.brown_min_angle_before_transformation if s.use_euler_coordinate_transformation else -1.0
        self.neel = s.neel_min_angle_before_transformation if s.use_spherical_coordinate_transformation else -1.0

    def chart(self, y):
        tb, tn = y[1].abs(), y[3].abs()
        br = (tb < self.brown) | (tb > math.pi - self.brown)
        nr = (tn < self.neel) | (tn > math.pi - self.neel)
        (s0, s1, s2), (c0, c1, c2) = [torch.sin(v) for v in y[:3]], [torch.cos(v) for v in y[:3]]
        turned = [torch.atan2(-c2 * c0 + c1 * s0 * s2, s0 * c2 + c1 * c0 * s2), torch.acos(-s1 * s2),
                  torch.atan2(c1, c2 * s1)]
        return [torch.where(br, a, b) for a, b in zip(turned, y[:3])] + _pole_rotate(y[3:], nr), (br, nr)

    def finish(self, y, chart):
        br, nr = chart
        (s0, s1, s2), (c0, c1, c2) = [torch.sin(v) for v in y[:3]], [torch.cos(v) for v in y[:3]]
        turned = [torch.atan2(c0 * c2 - c1 * s0 * s2, -c2 * s0 - c1 * c0 * s2), torch.acos(s1 * s2),
                  torch.atan2(-c1, c2 * s1)]
        return [torch.where(br, a, torch.fmod(b, 2.0 * math.pi)) for a, b in zip(turned, y[:3])] + _pole_unrotate(y[3:], nr)

    def _trig(self, y):
        return [torch.sin(v) for v in y], [torch.cos(v) for v in y]

    def _euler_project(self, S, C, br, v):
        """Euler angle rates of the angular velocity v; a rotated chart has its polar axis along -x"""
        u = tuple(torch.where(br, p, q) for p, q in ((v[2], v[0]), (v[1], v[1]), (-v[0], v[2])))
        first = (S[2] * u[0] - C[2] * u[1]) / S[1]
        return [first, C[2] * u[0] + S[2] * u[1], u[2] - C[1] * first]

    def _sphere_project(self, S, C, nr, v):
        u = tuple(torch.where(nr, p, q) for p, q in ((v[2], v[0]), (v[1], v[1]), (-v[0], v[2])))
        return [C[4] * u[1] - S[4] * u[0], u[2] - (C[4] * u[0] + S[4] * u[1]) * C[3] / S[3]]

    def _moment_axes(self, S, C, chart):
        br, nr = chart
        m = _spherical(S[3], C[3], S[4], C[4], nr)
        sf, st, ss, cf, ct, cs = S[0], S[1], S[2], C[0], C[1], C[2]
        own = [(cf * cs - ct * sf * ss, ct * sf * cs + cf * ss, st * sf),
               (-sf * cs - ct * cf * ss, ct * cf * cs - sf * ss, st * cf), (st * ss, -st * cs, ct)]
        return m, [tuple(torch.where(br, p, q) for p, q in ((-v[2], v[0]), (v[1], v[1]), (v[0], v[2]))) for v in own]

    def det(self, y, chart, B):
        S, C = self._trig(y)
        m, axes = self._moment_axes(S, C, chart)
        h, z = self.heff(m, axes, B), axes[2]
        torque = _lin((self.ct * _dot(m, z), _cross(z, m)))
        mxh = _cross(m, h)
        return (self._euler_project(S, C, chart[0], _lin((1.0, torque), (self.d, mxh)))
                + self._sphere_project(S, C, chart[1], _lin((-self.a, h), (self.bpd, mxh), (1.0, torque))))

    def noise_term(self, y, chart, w):
        S, C = self._trig(y)
        m, _ = self._moment_axes(S, C, chart)
        wa, wb = w[:3], w[3:]
        mxw = _cross(m, wb)
        return (self._euler_project(S, C, chart[0], _lin((self.cf, wa), (self.d * self.dn, mxw)))
                + self._sphere_project(S, C, chart[1], _lin((self.cf, wa), (self.bpd * self.dn, mxw),
                                                             (-self.a * self.dn, wb))))

    def drift(self, y, chart):
        S, C = self._trig(y)
        br, nr = chart
        ct, cs, ss = C[1], C[2], S[2]
        cn, cp, sn, sf = C[3], C[4], S[3], S[4]
        csc = 1.0 / S[1]
        cot = csc * ct
        ad, dd = self.a * self.d * self.dn ** 2, 0.25 * (self.d * self.dn) ** 2
        half = 0.5 * self.cf ** 2
        s2n = 2.0 * sn * cn
        ch, sh = cp * cs + ss * sf, cs * sf - cp * ss
        s2, c2 = 2.0 * sh * ch, ch * ch - sh * sh
        same = [csc * sn * (ad * sh - 2.0 * dd * (cn * ch + cot * sn * s2)),
                half * cot - ad * ch * sn + dd * (0.5 * (3.0 + cn * cn - sn * sn + 2.0 * c2 * sn * sn) * cot - s2n * sh),
                -(ad * (cn + sn * cot * sh) - dd * sn * (2.0 * cn * cot * ch + (2.0 * csc * csc - 1.0) * sn * s2))]
        # one chart rotated and the other not: s = +1 (Brown) or -1 (Neel)
        s = torch.where(br, 1.0, -1.0).to(torch.float64)
        c2s, s2s, s2p = cs * cs - ss * ss, 2.0 * cs * ss, 2.0 * sf * cp
        p, q = sn * sf * cs, cn * ss
        mixed = [csc * (ad * (-s * q + p) + 2.0 * dd * (-s * c2s * cot * s2n * sf + cp * sn * (cn * cs + s * sn * sf * ss)
                                                         + cot * s2s * (cn * cn - sn * sn * sf * sf))),
                 half * cot + ad * (-s * cn * cs - ss * sn * sf)
                 + dd * (2.0 * cs * cs * cot * (cn * cn + cp * cp * sn * sn) + s * cs * sn * sn * s2p
                         + 2.0 * ss * (-sn * cn * cp + cot * sn * sn * ss) + s * cot * s2n * sf * s2s),
                 ad * (s * sn * cp - cot * p + s * cot * q)
                 - dd * (cn * cs + s * sn * sf * ss) * (2.0 * cp * cot * sn - (3.0 + c2s) * csc * csc * (p - s * q))]
        nd = half + 0.5 * (self.a ** 2 + self.bpd ** 2) * self.dn ** 2
        return [torch.where(br == nr, u, v) for u, v in zip(same, mixed)] + [nd * cn / sn, torch.zeros_like(cn)]

    def output(self, y):
        S, C = self._trig(y)
        none = torch.zeros_like(y[0], dtype=torch.bool)
        m, axes = self._moment_axes(S, C, (none, none))
        return [*axes[0], *axes[1], *m]


class _BrownNeelCartesian(_Physics):
    noise, out = 6, 6

    def __init__(self, s):
        super().__init__(s)
        (sa, sb, sg), (ca, cb, cg) = [torch.sin(v) for v in self.euler], [torch.cos(v) for v in self.euler]
        n = [ca * cg - sa * cb * sg, -ca * sg - sa * cb * cg, sa * sb]
        ln, lm = torch.sqrt(_dot(n, n)), torch.sqrt(_dot(self.mag, self.mag))
        self.y = [v / ln for v in n] + [v / lm for v in self.mag]

    def chart(self, y):
        return y, None

    def det(self, y, c, B):
        n, e = y[:3], y[3:]
        en = _dot(e, n)
        h = tuple(self.pf * en * n[i] + B[i] for i in range(3))
        torque = _lin((self.ct * en, _cross(n, e)))
        mxh = _cross(e, h)
        return [*_cross(_lin((1.0, torque), (self.d, mxh)), n),
                *_cross(_lin((-self.a, h), (self.bpd, mxh), (1.0, torque)), e)]

    def noise_term(self, y, c, w):
        n, e, wa, wb = y[:3], y[3:], w[:3], w[3:]
        ddn = self.d * self.dn
        return [*_lin((-self.cf, _cross(n, wa)), (ddn * _dot(n, e), wb), (-ddn * _dot(n, wb), e)),
                *_lin((-self.cf, _cross(e, wa)), (self.bpd * self.dn, wb), (-self.bpd * self.dn * _dot(e, wb), e),
                      (self.a * self.dn, _cross(e, wb)))]

    def drift(self, y, c):
        n, e = y[:3], y[3:]
        d2 = 0.5 * (self.d * self.dn) ** 2
        nd = self.cf ** 2 + (self.a ** 2 + self.bpd ** 2) * self.dn ** 2
        return [*_lin((-self.cf ** 2 - d2 * (_dot(e, e) - 1.0), n), (self.d * self.a * self.dn ** 2, _cross(n, e))),
                *[-nd * v for v in e]]

    def finish(self, y, c):
        return list(y)

    def output(self, y):
        return y


def _step(p, solver, y, B, w):
    dt = p.dt
    if solver == Solver.Implicit_Midpoint:
        yn, yj = y, list(y)
        open_ = torch.ones_like(y[0], dtype=torch.bool)
        for _ in range(p.spec.max_iteration):
            r = [0.5 * (u + v) for u, v in zip(yj, yn)]
            a, b = p.det(r, None, B), p.noise_term(r, None, w)
            rhs = torch.stack([-(r[i] + a[i] * dt + b[i] + 0.5 * yn[i] - 1.5 * yj[i]) for i in range(3)], -1)
            dx = torch.linalg.solve(p.newton_matrix(r, B, w), rhs)
            dx = torch.where(open_[:, None], dx, torch.zeros_like(dx))
            yj = [yj[i] + dx[:, i] for i in range(3)]
            open_ = open_ & ((dx * dx).sum(-1).sqrt() > p.spec.accuracy_goal)
            if not bool(open_.any()):
                break
        return yj
    y, chart = p.chart(y)
    a, d, b = p.det(y, chart, B), p.drift(y, chart), p.noise_term(y, chart, w)
    if solver == Solver.EulerMaruyama:
        y = [v + (a[i] + d[i]) * dt + b[i] for i, v in enumerate(y)]
    elif solver == Solver.Millstein:
        ww = sum(v * v for v in w)
        y = [v + a[i] * dt + b[i] + d[i] * ww for i, v in enumerate(y)]
    else:
        s = [v + (a[i] + d[i]) * dt + b[i] for i, v in enumerate(y)]
        a2, d2 = p.det(s, chart, B), p.drift(s, chart)
        y = [v + 0.5 * (a[i] + d[i] + a2[i] + d2[i]) * dt + b[i] for i, v in enumerate(y)]
    return p.finish(y, chart)


def _integrate(spec):
    """Results of one ensemble: mean, weight, time and field."""
    p = {Problem.Neel: _Neel, Problem.NeelSpherical: _NeelSpherical, Problem.BrownAndNeelEulerSpherical: _BrownNeelEuler,
         Problem.BrownAndNeel: _BrownNeelCartesian}[spec.problem](spec)
    window, samples = spec.oversampling, spec.number_of_steps // spec.oversampling
    weights = p.weights(p.out)
    total = np.array([float(w.sum()) for w in weights])
    mean = np.zeros((samples, p.out))
    y = p.y
    out = p.output(y)
    mean[0] = [float((w * o).sum()) for w, o in zip(weights, out)]
    half = 0.5 if spec.solver == Solver.Implicit_Midpoint else 0.0
    for k in range(1, samples):
        acc = [torch.zeros_like(p.moment) for _ in range(p.out)]
        for g in range((k - 1) * window, k * window):
            if spec.noise == Noise.Injected:
                w = [_t(v) for v in spec.injected_dw[g]]
            else:
                w = [math.sqrt(p.dt) * v for v in _normals(spec.seed, spec.n, g, p.noise)]
            y = _step(p, spec.solver, y, p.field(p.dt * (g + 1 + half)), w)
            acc = [s + o for s, o in zip(acc, p.output(y))]
        mean[k] = [float((w * s).sum()) / window for w, s in zip(weights, acc)]
    time, end = np.zeros(samples), 0.0
    field = np.zeros((samples, 3))
    field[0] = p.field(0.0)
    for k in range(1, samples):
        start = end + p.dt
        end = p.dt * (k * window) + start
        time[k] = (end - start) - 0.5 * p.dt * window
        field[k] = np.mean([p.field(p.dt * ((k - 1) * window + l + 1)) for l in range(window)], axis=0)
    return {"mean": mean / total, "weight": total, "time": time, "field": field}
