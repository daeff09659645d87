"""Upload of caller-supplied increments: the pieces, the threads and the padded or converted
layouts.  A particle's path depends on its own increments only, so particles picked from a
large ensemble (several threads, several pieces each) and run in a small one (one thread, one
piece) have the same bits."""
import numpy as np
import pytest

import stochasticphysics_b200 as sp
from stochasticphysics_b200 import provider
from stochasticphysics_b200._abi import Precision, Problem, Solver

from test_gpu_parity import select_particles, small_spec

pytestmark = pytest.mark.gpu

# doubles: 2048 x 3 x 260 = 12.8 MB and 1001 x 6 x 520 = 25 MB, above four threads' threshold and
# more than two pieces per thread; 256 x 3 x 682 is just below it, 257 x 3 x 681 just above
CASES = [(2048, 260, Problem.Neel), (1001, 520, Problem.BrownAndNeel), (256, 682, Problem.Neel), (257, 682, Problem.Neel),
         (1, 100, Problem.Neel)]


@pytest.mark.parametrize("precision", [Precision.FP64, Precision.FP32])
@pytest.mark.parametrize("n,steps,problem", CASES)
def test_every_increment_arrives(n, steps, problem, precision):
    spec = small_spec(problem, Solver.Heun_Strong, n=n, steps=steps + 1, W=1, precision=precision, timestep=1e-12)
    spec = provider.with_injected_noise(spec, seed=n)
    idx = np.unique(np.linspace(0, n - 1, min(n, 40)).astype(int))
    with sp.Context(0) as ctx:
        for _ in range(2):  # the second upload reuses the pinned pieces
            large = ctx.simulate(spec, trajectories=True)
        small = ctx.simulate(select_particles(spec, idx), trajectories=True)
    assert large.trajectories.shape[1] == steps + 1
    np.testing.assert_array_equal(large.trajectories[idx], small.trajectories)
