"""The inner solve's passes on grids around the edges of their tiles (64 or 128 FP32, 32 or 64 FP64
cells wide, 16, 8 or 32 rows high, cut into parts along z): rows and columns one short of, equal to and
one past a tile, periodic faces that wrap across tiles and parts, one layer, padded rows.  The field of
three steps against the oracle's BiCG, on every step path bit for bit the same."""
import numpy as np
import pytest

from heatflow_gb300.problem import Problem
from heatflow_gb300.solver import HeatFlow
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SIZES = [((63, 17, 5), (0, 0, 0)), ((64, 16, 4), (1, 1, 1)), ((65, 15, 3), (1, 0, 1)), ((129, 9, 7), (1, 1, 0)),
         ((31, 33, 2), (0, 1, 1)), ((33, 32, 9), (1, 0, 0)), ((130, 7, 1), (1, 1, 0)), ((5, 65, 6), (0, 1, 0)),
         ((9, 5, 120), (0, 0, 1))]


def _problem(dims, periodic):
    nx, ny, nz = dims
    rng = np.random.default_rng(sum(dims))
    n = nx * ny * nz
    heat = np.zeros(n, np.int64)
    heat[rng.choice(n, 3, replace=False)] = 1
    return Problem(nx=nx, ny=ny, nz=nz, lx=nx * 1e-9, ly=ny * 1.2e-9, lz=nz * 0.9e-9, kappa=rng.uniform(20.0, 150.0, n),
                   rho=rng.uniform(1000, 3000, n), heat_capacity=700.0, tau=1e-12, em=0.0, iheater=heat,
                   power=np.where(heat > 0, 1e-6, 0.0), qdens_mode=1, time_step=1e-13, icattaneo=1,
                   periodic=periodic, kappa_bound=(149.0, 20.0, 60.0, 30.0, 50.0, 149.0),
                   t_bath_face=(300.0, 310.0, 295.0, 300.0, 305.0, 290.0), t_bath=300.0)


@pytest.mark.parametrize("precision,tol,bound", [("fp64", 1e-13, 1e-10), ("mixed", 1e-10, 1e-9)])
@pytest.mark.parametrize("dims,periodic", SIZES)
def test_tile_edges(cuda_lib, dims, periodic, precision, tol, bound):
    prob = _problem(dims, periodic)
    o = Oracle(prob)
    o.set_state(*prob.initial_state())
    rc, _ = o.run(3, itime0=1, mode=0, tol=1e-32, itmax=50000)
    assert rc == 0
    ref = o.get_state()[0]
    fields = []
    for g in (0, 1):
        with HeatFlow(prob, precision=precision, criterion="true", tol=tol, use_graph=g) as hf:
            hf.initial_evolve()
            st = hf.run(1, 3)
            fields.append(hf.get_state()[0])
        assert st["unconverged"] == 0
    assert np.array_equal(fields[0], fields[1])
    assert np.linalg.norm(fields[0] - ref) / np.linalg.norm(ref) <= bound
