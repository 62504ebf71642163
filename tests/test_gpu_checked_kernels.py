"""The index-checked build on the kernels that the smallest grids do not reach: the co-resident on-chip
solve, the general persistent solve and the plain launches, with wraps, padded rows, partial tiles and
tasks of one plane and of many, and a grid that takes the general solve by its size."""
import numpy as np
import pytest

from heatflow_gb300 import abi
from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem
from test_gpu_checked import checked_lib  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu

OPTS = {"recursive": dict(precision="fp64", criterion="recursive", tol=1e-32),
        "fp64": dict(precision="fp64", criterion="true", tol=1e-13), "mixed": dict(precision="mixed", criterion="true", tol=1e-10)}


def _check(lib, prob, first, kernel, **kw):
    out = []
    for library in (lib, abi.load_library()):
        with HeatFlow(prob, library=library, **kw) as hf:
            assert hf.inner_solver(first) == kernel
            hf.initial_evolve()
            hf.run(1, 3)
            out.append(hf.get_state())
            enabled, record = hf.index_checks()
            assert enabled == (library is lib) and record[0] == 0, record
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("opts", sorted(OPTS))
@pytest.mark.parametrize("kernel", ["resident", "general", "launches"])
@pytest.mark.parametrize("dims,periodic", [((2, 2, 2), (1, 1, 1)), ((33, 31, 17), (1, 1, 1)), ((66, 17, 9), (0, 1, 0)),
                                           ((7, 5, 30), (1, 0, 1))])
def test_no_index_fails(checked_lib, dims, periodic, kernel, opts):  # noqa: F811
    _check(checked_lib, _problem(dims, periodic), kernel, kernel, use_graph=0, **OPTS[opts])


@pytest.mark.parametrize("opts", sorted(OPTS))
def test_no_index_fails_in_deep_tasks(checked_lib, opts):  # noqa: F811
    """One task of 40 planes (of 20 in FP64)."""
    _check(checked_lib, _problem((9, 7, 40), (1, 0, 1)), "general", "general", use_graph=1, task_depth=80, **OPTS[opts])


@pytest.mark.parametrize("opts", ["fp64", "mixed"])
def test_no_index_fails_by_size(checked_lib, opts):  # noqa: F811
    _check(checked_lib, _problem((98, 97, 140), (1, 0, 0)), "auto", "general", use_graph=1, **OPTS[opts])
