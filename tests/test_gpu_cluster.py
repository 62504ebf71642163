"""The inner solve of a small grid on the chip: in one thread-block cluster (up to 16 FP64 or 32 FP32 tiles
of one plane) and in co-resident blocks with one task each, at the edges of those rules and of the blocks'
shares: one tile, 15 to 17, 30 to 34, tasks of one to three planes, wraps across blocks, padded rows, and
grids past both.  Bit for bit the solve of the same grid in a batch, whose blocks exchange everything
through memory."""
import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

WRAP, OPEN = (1, 1, 1), (0, 0, 0)
SIZES = [((25, 25, 1), OPEN), ((5, 3, 1), (1, 1, 0)), ((2, 2, 2), WRAP), ((33, 17, 4), WRAP), ((20, 20, 20), OPEN),
         ((64, 16, 15), WRAP), ((63, 16, 17), (0, 0, 1)), ((30, 14, 80), (1, 0, 1)), ((30, 14, 81), (1, 0, 1)),
         ((48, 48, 48), OPEN), ((65, 33, 24), WRAP), ((64, 16, 144), (1, 1, 0)), ((64, 16, 145), (1, 1, 0)),
         ((64, 16, 32), OPEN), ((64, 15, 33), WRAP)]
OPTS = [("fp64", "recursive", 1e-32), ("fp64", "true", 1e-13), ("mixed", "true", 1e-10)]


def _check(prob, copies, precision, criterion, tol):
    out = []
    for arg in (prob, [prob] * copies):
        with HeatFlow(arg, precision=precision, criterion=criterion, tol=tol, task_depth=4) as hf:
            hf.initial_evolve()
            st = hf.run(1, 3)
            out.append((hf.get_state()[0][:prob.ncells], st["unconverged"]))
    assert np.isfinite(out[0][0]).all()
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("precision,criterion,tol", OPTS)
@pytest.mark.parametrize("dims,periodic", SIZES)
def test_small_grid_equals_batch(cuda_lib, dims, periodic, precision, criterion, tol):
    _check(_problem(dims, periodic), 2, precision, criterion, tol)


@pytest.mark.parametrize("precision,criterion,tol", OPTS)
@pytest.mark.parametrize("ny,nz,periodic", [(16, 304, (0, 0, 1)), (15, 456, WRAP), (16, 608, OPEN)])
def test_deep_tasks_equal_batch(cuda_lib, ny, nz, periodic, precision, criterion, tol):
    """Two tiles side by side, tasks of 2, 3 and 4 planes (the last do not fit), in a batch of three of
    which the tasks are cut the same."""
    _check(_problem((128 if precision == "mixed" else 64, ny, nz), periodic), 3, precision, criterion, tol)
