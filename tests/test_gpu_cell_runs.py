"""The element-wise passes (right-hand side, first residual from the stored products, x update) at the edges
of their runs of cells, which are dealt to the tasks in pieces of 512: one cell short of a piece, a piece,
one past it, an odd number of cells, rows of which a pair of cells crosses the end, several groups of
tasks, wraps.  The field of four steps against the oracle's BiCG."""
import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from oracle.oracle import Oracle
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

SIZES = [((7, 73, 1), (0, 0, 0)), ((8, 8, 8), (0, 0, 1)), ((27, 19, 1), (0, 0, 0)), ((3, 11, 31), (1, 0, 0)),
         ((33, 31, 17), (1, 1, 0)), ((64, 9, 40), (0, 0, 0)), ((2, 65, 13), (0, 1, 0))]


@pytest.mark.parametrize("precision,criterion,tol,bound", [("fp64", "recursive", 1e-32, 1e-10), ("fp64", "true", 1e-13, 1e-10),
                                                           ("mixed", "true", 1e-10, 1e-9)])
@pytest.mark.parametrize("dims,periodic", SIZES)
def test_run_edges(cuda_lib, dims, periodic, precision, criterion, tol, bound):
    prob = _problem(dims, periodic)
    o = Oracle(prob)
    o.set_state(*prob.initial_state())
    rc, _ = o.run(4, itime0=1, mode=0, tol=1e-32, itmax=50000)
    assert rc == 0
    ref = o.get_state()[0]
    with HeatFlow(prob, precision=precision, criterion=criterion, tol=tol) as hf:
        hf.initial_evolve()
        st = hf.run(1, 4)
        got = hf.get_state()[0]
    assert st["unconverged"] == 0
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= bound
