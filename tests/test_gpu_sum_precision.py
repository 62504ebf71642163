"""The inner solve's FP32 sums cover 8192 cells at most; longer ones go on in FP64.

Values are chosen so that an FP32 sum over a whole deep task loses all but the first planes: in every
strip of four cells one is 1 in the first eight planes and 0 above, the others are 2^-13 everywhere.  The
first eight planes of a thread add up to 8, whose unit in FP32 is 2^-20, and those of each later group of
eight planes to 24 2^-26, less than half of it.  The operator is a multiple of the identity (the heat
capacity term is 1e12 times the conduction), so one CG iteration from zero solves the system, with
alpha = r.r / p.Ap = 1.  r.r comes from the residual sweep, whose threads own one column each and add
these values exactly; a p.Ap that loses the later planes is 3 (planes - 8) 2^-26 / 8 too small.

Left with the group of eight: 24 2^-26 of 8 (4.5e-8), and alpha's rounding to FP32 (6e-8); so 2^-22."""
import numpy as np
import pytest

from heatflow_gb300.problem import Problem
from heatflow_gb300.solver import HeatFlow

pytestmark = pytest.mark.gpu

EXP = 100                                     # rho c / dt = 2^EXP


@pytest.mark.parametrize("nz", [9, 16, 17, 64, 256])
def test_deep_sum(cuda_lib, nz):
    nx, ny = 32, 8
    n = nx * ny * nz
    prob = Problem(nx=nx, ny=ny, nz=nz, lx=nx * 1e-9, ly=ny * 1e-9, lz=nz * 1e-9, kappa=1.0, rho=2.0 ** 20,
                   heat_capacity=1.0, tau=0.0, em=0.0, iheater=np.zeros(n, np.int64), time_step=2.0 ** (20 - EXP),
                   icattaneo=0, kappa_bound=(1.0,) * 6, t_bath_face=(0.0,) * 6, t_bath=0.0)
    g = np.full((nz, ny, nx), 2.0 ** -13)
    g[:, :, ::4] = 0.0
    g[:8, :, ::4] = 1.0
    b = -g.reshape(-1) * 2.0 ** (EXP // 2)
    with HeatFlow(prob, precision="mixed", criterion="true", tol=1e-30, inner_itmax=1, max_refine=1,
                  task_depth=1024) as hf:
        x, _ = hf.linbcg(b, np.zeros(n))
    alpha = x.reshape(nz, ny, nx)[:8, :, ::4] * 2.0 ** (EXP // 2)
    assert np.abs(alpha - 1.0).max() <= 2.0 ** -22
