"""The persistent solve of several grids takes its tasks from one queue in which every grid advances
at its own pace: more grids than threads of a block, grids that end at different times, and a grid
that has no work at all (its right-hand side is NaN) give the host-polled kernels' bits."""
import numpy as np
import pytest

from heatflow_gb300 import abi
from heatflow_gb300.problem import point_source_cube, random_instance
from heatflow_gb300.solver import HeatFlow

pytestmark = pytest.mark.gpu

OPTS = [dict(precision="mixed", criterion="true", tol=1e-10),
        dict(precision="fp64", criterion="recursive", tol=1e-32)]


@pytest.mark.parametrize("opts", OPTS)
@pytest.mark.parametrize("count,lo,hi", [(2, 4, 40), (256, 2, 5), (257, 2, 5), (600, 2, 4)])
def test_queue_equals_host_loop(cuda_lib, opts, count, lo, hi):
    rng = np.random.default_rng(count)
    probs = [random_instance(rng, lo=lo, hi=hi) for _ in range(count)]
    out = []
    for g in (0, 1):
        with HeatFlow(probs, use_graph=g, **opts) as hf:
            hf.initial_evolve()
            st = hf.run(1, 3)
            out.append((hf.get_state(), {k: st[k] for k in ("iterations", "inner_iterations", "refinements",
                                                            "unconverged")}))
    assert out[0][1] == out[1][1]
    assert all(np.array_equal(a, b) for a, b in zip(out[0][0], out[1][0]))


def test_grid_without_work(cuda_lib):
    rng = np.random.default_rng(1)
    probs = [point_source_cube(9, icattaneo=0)] + [random_instance(rng, lo=4, hi=12) for _ in range(3)]
    tp = np.full(sum(p.ncells for p in probs), 300.0)
    tp[3] = np.nan
    out = []
    for g in (0, 1):
        with HeatFlow(probs, use_graph=g, **OPTS[0]) as hf:
            hf.set_state(tp, tp)
            with pytest.raises(abi.HeatFlowError) as e:
                hf.run(1, 3)
            assert e.value.code == abi.HF_ENAN_S
            out.append(hf.get_state())
    rest = slice(probs[0].ncells, None)
    for a, b in zip(*out):
        assert np.array_equal(a[rest], b[rest]) and np.isfinite(b[rest]).all()
