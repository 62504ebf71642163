"""The residual sweep on planes whose tasks are runs of 256 consecutive columns instead of 32 x 8 tiles: row
ends and wraps inside a warp, a plane of exactly one run and of one column more, one row, narrow rows.  As
tests/test_gpu_cell_runs.py."""
import pytest

import test_gpu_cell_runs as runs

pytestmark = pytest.mark.gpu

SIZES = [((16, 16, 9), (1, 1, 0)), ((257, 1, 4), (1, 0, 0)), ((17, 15, 6), (1, 1, 1)), ((33, 8, 7), (0, 0, 0)),
         ((3, 86, 5), (1, 0, 1)), ((65, 19, 4), (1, 1, 0))]


@pytest.mark.parametrize("precision,criterion,tol,bound", [("fp64", "recursive", 1e-32, 1e-10), ("fp64", "true", 1e-13, 1e-10),
                                                           ("mixed", "true", 1e-10, 1e-9)])
@pytest.mark.parametrize("dims,periodic", SIZES)
def test_column_runs(cuda_lib, dims, periodic, precision, criterion, tol, bound):
    runs.test_run_edges(cuda_lib, dims, periodic, precision, criterion, tol, bound)
