"""Launch counts of runs with caller-supplied increments: the kernels that spread uploaded pieces
(2 MiB each) to the padded or single-precision layout are counted for the ensemble and for the
process.  Whole pieces in the device's own layout are copied without one."""
import pytest

import stochasticphysics_b200 as sp
from stochasticphysics_b200 import provider
from stochasticphysics_b200._abi import Precision, Problem, Solver
from stochasticphysics_b200.simulator import kernel_launch_count

from test_gpu_parity import small_spec

pytestmark = pytest.mark.gpu

PIECE = (2 << 20) // 8


@pytest.mark.parametrize("precision", [Precision.FP64, Precision.FP32])
@pytest.mark.parametrize("n,steps", [(256, 40), (255, 40), (257, 400), (256, 400)])
def test_spread_kernels_are_counted(n, steps, precision):
    spec = small_spec(Problem.Neel, Solver.Heun_Strong, n=n, steps=steps + 1, W=1, precision=precision, timestep=1e-12)
    spec = provider.with_injected_noise(spec, seed=n)
    doubles = spec.integrated_steps * 3 * n
    assert doubles * 8 < 4 << 20  # one thread
    direct = precision == Precision.FP64 and n % 256 == 0
    spread = 0 if direct else -(-doubles // PIECE)
    with sp.Context(0) as ctx:
        before = kernel_launch_count()
        launches = ctx.simulate(spec).stats["kernel_launches"]
        # three for the initial state, the target, four of the one chunk
        assert launches == 3 + 1 + 4 + spread
        assert kernel_launch_count() - before == launches
