"""FP64 angle problems around the chart thresholds: particles that start on both sides of the
pole angle of each chart and cross it (a Neel angle moves by about 0.03 rad per step), so the
carried chart is entered, kept and left, alone and in every combination of the two charts.

Bars: the parity tests' 1e-9 per trajectory value, on the particles whose oracle run agrees
with its own long-double run to 1e-11 (at least half of them here).  The final angles are
compared as directions, whose components do not amplify the azimuth's 1/sin(theta)."""
import dataclasses
import math

import numpy as np
import pytest

import oracle
import stochasticphysics_b200 as sp
from stochasticphysics_b200 import provider
from stochasticphysics_b200._abi import Problem, Solver

from test_gpu_parity import LD_STRICT, REL_TRAJ, ld_spread, select_particles, small_spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sp.Context(0)
    yield c
    c.close()


def threshold_spec(problem, solver, n, steps=240, W=40, brown=True, neel=True, pole=math.pi / 36):
    rng = np.random.default_rng(n)
    spec = small_spec(problem, solver, n=n, steps=steps, W=W, seed=n)
    centre = rng.choice([pole, math.pi - pole, 0.5 * math.pi], size=(2, n))
    theta = np.clip(centre + rng.uniform(-0.03, 0.03, (2, n)), 0.02, math.pi - 0.02)
    phi = rng.uniform(0, 2 * math.pi, n)
    m0 = np.stack([np.sin(theta[1]) * np.cos(phi), np.sin(theta[1]) * np.sin(phi), np.cos(theta[1])], axis=1)
    euler = np.array(spec.orientation, copy=True)
    euler[:, 1] = theta[0]
    kw = dict(orientation=euler, magnetisation=m0)
    if problem == Problem.NeelSpherical:
        kw.update(use_coordinate_transformation=neel, min_angle_before_transformation=pole)
    else:
        kw.update(use_euler_coordinate_transformation=brown, use_spherical_coordinate_transformation=neel,
                  brown_min_angle_before_transformation=pole, neel_min_angle_before_transformation=pole)
    return dataclasses.replace(spec, **kw)


def directions(problem, y):
    t, p = y[:, -2], y[:, -1]
    out = [np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)]
    if problem == Problem.BrownAndNeelEulerSpherical:
        out += [c for a in provider.body_axes(problem, y[:, :3]) for c in a.T]
    return np.stack(out, axis=1)


CASES = [(Problem.NeelSpherical, s, n, False, True) for s in (Solver.EulerMaruyama, Solver.Heun_Strong, Solver.Millstein)
         for n in (1, 33, 257)]
CASES += [(Problem.BrownAndNeelEulerSpherical, s, n, b, m) for s in (Solver.EulerMaruyama, Solver.Heun_Strong, Solver.Millstein)
          for n, b, m in ((1, True, True), (31, True, True), (257, True, True), (65, True, False), (65, False, True))]
# a pole angle above pi / 2 turns the chart for every state, one of 0 for none
CASES += [(Problem.NeelSpherical, Solver.Heun_Strong, 64, False, True, 1.8),
          (Problem.BrownAndNeelEulerSpherical, Solver.Heun_Strong, 64, True, True, 0.0)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(getattr(v, "name", v)) for v in c))
def test_threshold_crossings_match_the_oracle(ctx, case):
    problem, solver, n, brown, neel = case[:5]
    spec = threshold_spec(problem, solver, n, brown=brown, neel=neel, **({"pole": case[5]} if len(case) > 5 else {}))
    spec = provider.with_injected_noise(spec, seed=n)
    spread, _ = ld_spread(spec, oracle.simulate(spec, trajectories=True))
    good = np.where(np.max(spread, axis=1) <= LD_STRICT)[0]
    assert 2 * len(good) >= n
    sub = select_particles(spec, good)
    gpu = ctx.simulate(sub, trajectories=True, final_state=True)
    ref = oracle.simulate(sub, trajectories=True, final_state=True)
    err = np.abs(gpu.trajectories - ref["trajectories"]) / np.maximum(np.abs(ref["trajectories"]), 1e-3)
    assert np.max(err) < REL_TRAJ
    assert np.max(np.abs(directions(problem, gpu.final_state) - directions(problem, ref["final_state"]))) < REL_TRAJ


@pytest.mark.parametrize("problem", [Problem.NeelSpherical, Problem.BrownAndNeelEulerSpherical])
def test_pieces_and_server_equal_one_run(ctx, problem):
    """The chart is kept across launches: any cut of the run gives the same bits."""
    spec = threshold_spec(problem, Solver.Heun_Strong, 300, steps=1600, W=40)
    whole = ctx.simulate(spec, final_state=True)
    with ctx.ensemble(spec, shape={"block": 32, "persistent": 0, "chunk_steps": 120}) as ens:
        for piece in (40, 200, 7, 1313):
            ens.advance(piece)
        cut = ens.read(final_state=True)
    with ctx.server(chunk_steps=80) as srv:
        served = srv.wait(srv.submit(spec))[0]
    np.testing.assert_array_equal(whole.mean, cut.mean)
    np.testing.assert_array_equal(whole.final_state, cut.final_state)
    np.testing.assert_array_equal(whole.mean, served.mean)
