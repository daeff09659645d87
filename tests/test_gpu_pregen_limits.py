"""Where the separate noise draw ends: the largest ensemble that takes it and the next one, for
every problem, solver and anisotropy with a limit of its own.  The launch count tells the two
apart (one kernel more per chunk); the server's groups always draw in the step kernel, and a
run has the same bits either way."""
import dataclasses

import numpy as np
import pytest
import torch

import stochasticphysics_b200 as sp
from stochasticphysics_b200._abi import Anisotropy, Problem, Solver

from test_gpu_parity import small_spec

pytestmark = pytest.mark.gpu

EM, HEUN, MIL = Solver.EulerMaruyama, Solver.Heun_Strong, Solver.Millstein
UNI, CUBIC, BOTH = Anisotropy.Uniaxial, Anisotropy.Cubic, Anisotropy.UniaxialCubic
SPH, BNE = Problem.NeelSpherical, Problem.BrownAndNeelEulerSpherical
# particles per SM
LIMITS = [(Problem.Neel, HEUN, UNI, 176), (Problem.Neel, EM, BOTH, 176), (Problem.Neel, HEUN, CUBIC, 152),
          (Problem.Neel, HEUN, BOTH, 152), (SPH, EM, CUBIC, 224), (SPH, HEUN, BOTH, 256), (BNE, MIL, UNI, 208),
          (BNE, HEUN, CUBIC, 256), (BNE, EM, BOTH, 256), (Problem.BrownAndNeel, HEUN, UNI, 56),
          (Problem.BrownAndNeel, HEUN, CUBIC, 72), (Problem.BrownAndNeel, EM, UNI, 76),
          (Problem.BrownAndNeel, EM, CUBIC, 168), (Problem.BrownAndNeel, MIL, UNI, 100),
          (Problem.BrownAndNeel, MIL, CUBIC, 168)]


@pytest.fixture(scope="module")
def ctx():
    c = sp.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("problem,solver,aniso,per_sm", LIMITS)
def test_both_sides_of_the_limit(ctx, problem, solver, aniso, per_sm):
    limit = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    launches = []
    for n in (limit, limit + 1):
        spec = small_spec(problem, solver, aniso=CUBIC if aniso == CUBIC else UNI, n=n, steps=60, W=20, seed=n)
        if aniso == BOTH:
            rng = np.random.default_rng(n)
            spec = dataclasses.replace(spec, anisotropy=BOTH, cubic_constant=np.full(n, -4e3),
                                       uniaxial_rotation=rng.uniform(0, 2 * np.pi, (n, 3)))
        alone = ctx.simulate(spec)
        with ctx.server() as srv:
            served = srv.wait(srv.submit(spec))[0]
        np.testing.assert_array_equal(alone.mean, served.mean)
        launches.append(alone.stats["kernel_launches"])
    assert launches[0] == launches[1] + 1
