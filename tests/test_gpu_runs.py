"""The step loop's runs: a run of steps ends at a window's end, at a stage's end (8 or 5 copied
steps, 4 or 2 drawn) and at a field tile's end (32 or 128 steps), and lanes past the ensemble's
end repeat the last particle.  Windows shorter than, equal to and longer than each, particle
counts on both sides of a warp and a tile, whatever draws the noise."""
import numpy as np
import pytest

import oracle
import stochasticphysics_b200 as sp
from stochasticphysics_b200 import provider
from stochasticphysics_b200._abi import Precision, Problem, Solver

from test_gpu_parity import ABS_MEAN, REL_TRAJ, small_spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = sp.Context(0)
    yield c
    c.close()


CASES = [(Problem.Neel, 1, 1), (Problem.Neel, 31, 3), (Problem.Neel, 33, 8), (Problem.Neel, 257, 37), (Problem.Neel, 64, 129),
         (Problem.NeelSpherical, 33, 5), (Problem.NeelSpherical, 100, 32), (Problem.BrownAndNeel, 65, 7),
         (Problem.BrownAndNeel, 31, 33), (Problem.BrownAndNeelEulerSpherical, 33, 2),
         (Problem.BrownAndNeelEulerSpherical, 129, 31)]


@pytest.mark.parametrize("precision", [Precision.FP64, Precision.FP32])
@pytest.mark.parametrize("problem,n,W", CASES)
def test_windows_of_every_length(ctx, problem, n, W, precision):
    """The same steps summed into windows of W and of one step: the window means are the means of
    the recorded steps.  A Kahan sum of at most 129 values of size 1 is within two ulps."""
    steps = max(3 * W, 40) // W * W + W
    spec = small_spec(problem, Solver.Heun_Strong, n=n, steps=steps, W=W, seed=n, timestep=1e-12, precision=precision)
    single = small_spec(problem, Solver.Heun_Strong, n=n, steps=steps - W + 1, W=1, seed=n, timestep=1e-12, precision=precision)
    eps = 2.3e-16 if precision == Precision.FP64 else 1.2e-7
    for injected in (False, True):
        a, b = (provider.with_injected_noise(s, seed=3) if injected else s for s in (spec, single))
        got = ctx.simulate(a, trajectories=True).trajectories[:, 1:]
        each = ctx.simulate(b, trajectories=True).trajectories[:, 1:]
        want = each.reshape(n, steps // W - 1, W, -1).mean(axis=2)
        assert np.max(np.abs(got - want)) <= 4 * eps


@pytest.mark.parametrize("problem,n,W", CASES)
def test_drawn_and_copied_agree_with_the_oracle(ctx, problem, n, W):
    steps = max(3 * W, 40) // W * W + W
    spec = small_spec(problem, Solver.Heun_Strong, n=n, steps=steps, W=W, seed=n, timestep=1e-12)
    alone = ctx.simulate(spec, trajectories=True)  # drawn before the chunk, copied
    with ctx.server() as srv:                      # drawn in the step kernel
        served = srv.wait(srv.submit(spec))[0]
    np.testing.assert_array_equal(alone.mean, served.mean)
    ref = oracle.simulate(spec, trajectories=True)
    err = np.abs(alone.trajectories - ref["trajectories"]) / np.maximum(np.abs(ref["trajectories"]), 1e-3)
    assert np.max(err) < REL_TRAJ
    assert np.max(np.abs(alone.mean - ref["mean"])) < ABS_MEAN
