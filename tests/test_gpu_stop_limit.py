"""The inner solves of one grid compare with the largest value that meets the criterion, found before the
first iteration; those of a batch form the criterion in every iteration.  Both stop at the same iteration
with the same error, bit for bit: at ordinary tolerances, at one so small that no such value is found, and
where the iteration cap ends the solve."""
import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(precision="fp64", criterion="recursive", tol=1e-32),
                                  dict(precision="fp64", criterion="recursive", tol=1e-7),
                                  dict(precision="fp64", criterion="recursive", tol=1e-200, itmax=40),
                                  dict(precision="fp64", criterion="recursive", tol=1e-32, itmax=7),
                                  dict(precision="fp64", criterion="true", tol=1e-12),
                                  dict(precision="mixed", criterion="true", tol=1e-10),
                                  dict(precision="mixed", criterion="true", tol=1e-10, inner_tol=0.03125)])
@pytest.mark.parametrize("dims", [(9, 7, 1), (20, 20, 20), (64, 31, 48)])
def test_same_stop(cuda_lib, dims, opts):
    prob = _problem(dims, (0, 0, 0))
    out = []
    for arg in (prob, [prob, prob]):
        with HeatFlow(arg, task_depth=4, **opts) as hf:
            hf.initial_evolve()
            steps = []
            for k in (1, 2, 3):
                st = hf.run(k, 1)
                n = 1 if arg is prob else 2
                steps.append((st["iterations"] // n, st["inner_iterations"] // n, st["unconverged"] // n,
                              st["last_err"], hf.get_state()[0][:prob.ncells].copy()))
            out.append(steps)
    for a, b in zip(*out):
        assert a[:4] == b[:4]
        assert np.array_equal(a[4], b[4])
