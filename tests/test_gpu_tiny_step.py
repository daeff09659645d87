"""Time steps down to the smallest double: the FP64 increments underflow to nothing, not to NaN.
-2 dt ln u is subnormal below about 1e-298 s, which the kernels' square root need not take.  No
increment of these steps reaches a state of order one, so it stays as it began."""
import numpy as np
import pytest

import stochasticphysics_b200 as sp
from stochasticphysics_b200._abi import Problem, Solver

from test_gpu_parity import small_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 70000])  # drawn before the chunk, drawn in the step kernel
@pytest.mark.parametrize("problem", list(Problem))
@pytest.mark.parametrize("timestep", [1e-290, 1e-300, 5e-324])
def test_state_stays(problem, timestep, n):
    spec = small_spec(problem, Solver.Heun_Strong, n=n, steps=30, W=10, seed=4, timestep=timestep)
    with sp.Context(0) as ctx:
        out = ctx.simulate(spec)
    assert out.stats["nonfinite_particles"] == 0
    # the window mean divides a sum of ten equal values: one rounding each way
    np.testing.assert_allclose(out.mean, np.broadcast_to(out.mean[0], out.mean.shape), rtol=1e-14, atol=1e-15)
