"""A right-hand-side probe between queued host-buffer steps is refused before it touches anything: the
queue ends as if it had not been asked."""
import numpy as np
import pytest

from heatflow_gb300 import abi
from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem
from test_gpu_host_async import _pinned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 1e-10)])
def test_probe_between_queued_steps(cuda_lib, precision, tol):
    prob = _problem((33, 17, 12), (1, 0, 0))
    fields, launches = [], []
    for probe in (False, True):
        bufs = [_pinned(prob.ncells, 300.0) for _ in range(3)]
        with HeatFlow(prob, precision=precision, criterion="true", tol=tol, use_graph=1) as hf:
            new, prev, free = bufs
            for k in range(5):
                hf.step_host_async(1 + k, new, prev, free)
                new, prev, free = free, new, prev
                if probe:
                    with pytest.raises(abi.HeatFlowError) as e:
                        hf.rhs(1 + k)
                    assert e.value.code == abi.HF_ESTATE
            launches.append(hf.host_sync()["kernel_launches"])
            fields.append(new.copy())
    assert np.array_equal(fields[0], fields[1]) and launches[0] == launches[1]
