"""The rebuild's quotients are formed from shared reciprocals and must be the correctly rounded ones that
the set-up assembly's divisions give: cell lengths and conductivities of every magnitude, conductivities
whose products leave the range of the short form, and equal neighbours."""
import dataclasses

import numpy as np
import pytest

from heatflow_gb300.problem import Problem
from heatflow_gb300.solver import HeatFlow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,periodic,lengths", [((33, 20, 11), (0, 0, 0), (1.3e-9, 0.7e-9, 2.9e-9)),
                                                   ((16, 9, 24), (1, 1, 1), (3.1e-7, 1.1e-8, 1e-9)),
                                                   ((64, 3, 30), (0, 1, 0), (1e-9, 1e-9, 1e-9))])
def test_quotients_round_correctly(cuda_lib, dims, periodic, lengths):
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(n)
    values = np.concatenate([10.0 ** rng.uniform(-4, 4, 300) * rng.uniform(1, 2, 300), [149.0, 149.0, 1e-180, 3e-150]])
    tables = [np.array([[200.0, v, 2000.0, 700.0], [400.0, v, 2000.0, 700.0]]) for v in values]
    ct = rng.integers(0, len(tables), n).astype(np.int32)
    prob = Problem(nx=nx, ny=ny, nz=nz, lx=nx * lengths[0], ly=ny * lengths[1], lz=nz * lengths[2], kappa=100.0, rho=2000.0,
                   heat_capacity=700.0, tau=1e-12, em=0.0, iheater=0, power=None, time_step=1e-13, icattaneo=1,
                   kappa_bound=(149.0, 20.0, 60.0, 30.0, 50.0, 149.0), t_bath_face=(300.0,) * 6, t_bath=300.0,
                   periodic=periodic)
    with HeatFlow(prob, precision="fp64", criterion="true", tol=1e-12, use_graph=1) as hf:
        hf.set_property_tables(tables, ct)
        hf.initial_evolve()
        hf.run(1, 1)
        op = hf.operator()
    ref = dataclasses.replace(prob, kappa=values[ct], _keep=[])
    with HeatFlow(ref, precision="fp64", criterion="true", tol=1e-12) as hf0:
        op0 = hf0.operator()
    for key in ("diag", "cx", "cy", "cz"):
        assert np.array_equal(op[key], op0[key]), key
