"""A context whose options change between steps runs each step as a context created with them would: the
criterion, the precision and the task depth pick kernels, grids of blocks and plans anew."""
import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

OPTS = [dict(precision="fp64", criterion="true", tol=1e-13), dict(precision="fp64", criterion="recursive", tol=1e-32),
        dict(precision="mixed", criterion="true", tol=1e-10, task_depth=32), dict(precision="mixed", criterion="true", tol=1e-10)]


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("dims", [[(25, 9, 3)], [(96, 70, 64)], [(40, 33, 20), (9, 8, 7)]])
def test_options_change_between_steps(cuda_lib, dims, use_graph):
    probs = [_problem(d, (0, 0, 0)) for d in dims]
    order = [0, 1, 0, 2, 3, 1, 3]
    with HeatFlow(probs, use_graph=use_graph, **OPTS[order[0]]) as hf:
        hf.initial_evolve()
        for k, which in enumerate(order):
            before = hf.get_state()
            hf.set_opts(use_graph=use_graph, **OPTS[which])
            hf.set_state(*before)
            hf.run(k + 1, 1)
            after = hf.get_state()
            with HeatFlow(probs, use_graph=use_graph, **OPTS[which]) as fresh:
                fresh.set_state(*before)
                fresh.run(k + 1, 1)
                assert np.array_equal(fresh.get_state()[0], after[0]), (k, which)
