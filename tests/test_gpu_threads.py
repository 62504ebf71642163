"""Contexts of different sizes that step at the same time on threads of their own: each gives the bits it
gives alone.  The grids' inner solves run in one kernel with different amounts of shared memory, and
every set_opts captures the steps again."""
import threading

import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

DIMS = [(48, 48, 48), (64, 64, 96)]          # tasks of one plane and of three


def _steps(dims, opts, out):
    try:
        with HeatFlow(_problem(dims, (0, 0, 0)), **opts) as hf:
            hf.initial_evolve()
            for k in range(40):
                hf.set_opts(**opts)
                hf.run(1 + k, 1)
            out[dims] = hf.get_state()[0]
    except Exception as e:                   # noqa: BLE001 (reported by the caller)
        out[dims] = e


@pytest.mark.parametrize("use_graph", [0, 1])
def test_contexts_on_two_threads(cuda_lib, use_graph):
    opts = dict(precision="fp64", criterion="true", tol=1e-10, use_graph=use_graph)
    alone, together = {}, {}
    for dims in DIMS:
        _steps(dims, opts, alone)
    threads = [threading.Thread(target=_steps, args=(dims, opts, together)) for dims in DIMS]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for dims in DIMS:
        assert isinstance(together[dims], np.ndarray), together[dims]
        assert np.array_equal(together[dims], alone[dims])
