"""Options that need more device memory than there is: set_opts says so and the context goes on with the
options it had.  The index-checked build refuses the first, second or third allocation of the new plan; no
memory is used up."""
import numpy as np
import pytest

from heatflow_gb300 import abi
from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem
from test_gpu_checked import checked_lib  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu

MIXED = dict(precision="mixed", criterion="true", tol=1e-10)
FP64 = dict(precision="fp64", criterion="true", tol=1e-13)       # twice the tiles: every table grows


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("which", [1, 2, 3])
def test_set_opts_refused(checked_lib, which, use_graph):  # noqa: F811
    prob = _problem((128, 64, 8), (1, 0, 0))
    fields = []
    for refuse in (False, True):
        with HeatFlow(prob, library=checked_lib, use_graph=use_graph, **MIXED) as hf:
            hf.initial_evolve()
            hf.run(1, 2)
            if refuse:
                hf.index_checks(probe=1 + which)
                with pytest.raises(abi.HeatFlowError) as e:
                    hf.set_opts(use_graph=use_graph, **FP64)
                assert e.value.code == abi.HF_ENOMEM
            hf.run(3, 2)
            fields.append(hf.get_state()[0])
            hf.set_opts(use_graph=use_graph, **FP64)
            hf.run(5, 2)
            fields.append(hf.get_state()[0])
            assert hf.index_checks()[1][0] == 0
    assert np.array_equal(fields[0], fields[2]) and np.array_equal(fields[1], fields[3])
