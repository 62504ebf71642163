"""The bounded waits of every persistent solve run out without any GPU fault: a block of the on-chip or the
general solve of one grid, or of a batch's queue, leaves; the others give up after a short time limit, the
host reads HF_EDEVICE, and the next steps equal an untouched run."""
import ctypes as C

import numpy as np
import pytest

from heatflow_gb300 import abi
from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

SMALL, LARGE = ((40, 33, 20), (1, 0, 0)), ((90, 96, 96), (0, 0, 0))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("grids,kernel", [([SMALL], "resident"), ([SMALL], "general"), ([SMALL, SMALL], "general"),
                                          ([SMALL, LARGE, LARGE], "general")])
def test_waits_run_out(cuda_lib, grids, kernel, precision):
    probs = [_problem(*g) for g in grids]
    opts = dict(precision=precision, criterion="true", tol=1e-10, use_graph=1, task_depth=4)
    fields = []
    for leave in (True, False):
        with HeatFlow(probs, **opts) as hf:
            assert hf.inner_solver(kernel) == kernel
            hf.initial_evolve()
            hf.run(1, 2)
            if leave:
                status, seconds = C.c_int32(), C.c_double()
                lib = abi.load_library()
                assert lib.hf_check_barrier_timeout(hf.h, 200, C.byref(status), C.byref(seconds)) == abi.HF_OK
                assert status.value == abi.HF_EDEVICE
                assert 0.2 <= seconds.value < 3.0, seconds.value
            hf.run(3, 3)
            fields.append(hf.get_state())
    assert np.array_equal(fields[0][0], fields[1][0]) and np.array_equal(fields[0][1], fields[1][1])
