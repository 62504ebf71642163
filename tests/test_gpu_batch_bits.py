"""A grid's field does not depend on the batch it is in where the caller gives the task depth: alone, in
two batches of different grids and next to a large one, bit for bit, for tasks of one plane and of many."""
import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

GRIDS = [((40, 33, 50), (1, 0, 1)), ((61, 17, 90), (0, 0, 0)), ((24, 70, 31), (0, 1, 0))]
LARGE = ((90, 96, 96), (0, 0, 0))


def _fields(grids, opts):
    probs = [_problem(*g) for g in grids]
    with HeatFlow(probs, **opts) as hf:
        hf.initial_evolve()
        assert hf.run(1, 3)["unconverged"] == 0
        return hf.split(hf.get_state()[0])


@pytest.mark.parametrize("depth", [4, 32, 64])
@pytest.mark.parametrize("precision,tol", [("mixed", 1e-10), ("fp64", 1e-13)])
def test_a_grid_in_any_batch(cuda_lib, precision, tol, depth):
    opts = dict(precision=precision, criterion="true", tol=tol, use_graph=1, task_depth=depth)
    alone = [_fields([g], opts)[0] for g in GRIDS]
    for batch in (GRIDS, [*GRIDS, LARGE, LARGE]):
        for a, b in zip(alone, _fields(batch, opts)):
            assert np.array_equal(a, b)
