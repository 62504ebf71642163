"""The kernels that run the inner CG solves: which one a grid takes, on either side of each rule, and that
every one gives the bits of the plain launches (a kernel per pass, polled by the host; none of them waits
for another block): one thread-block cluster, co-resident blocks with their state on the chip, persistent
blocks with their state in memory, and the queue of a batch, whole-step and inner solves alone."""
import numpy as np
import pytest

from heatflow_gb300.solver import HeatFlow
from test_gpu_cg_tiles import _problem

pytestmark = pytest.mark.gpu

WRAP, OPEN = (1, 1, 1), (0, 0, 0)
RECURSIVE = dict(precision="fp64", criterion="recursive", tol=1e-32)
FP64 = dict(precision="fp64", criterion="true", tol=1e-13)
MIXED = dict(precision="mixed", criterion="true", tol=1e-10)
STATS = ("iterations", "inner_iterations", "refinements", "unconverged")


@pytest.mark.parametrize("opts,dims,kernel", [
    (MIXED, (64, 16, 32), "cluster"), (MIXED, (64, 16, 33), "resident"),        # 32 tasks of a plane, 33
    (FP64, (32, 16, 16), "cluster"), (FP64, (32, 16, 17), "resident"),          # 16, 17
    (RECURSIVE, (32, 16, 16), "cluster"), (RECURSIVE, (32, 16, 17), "resident"),
    (MIXED, (64, 16, 304), "resident"), (MIXED, (64, 16, 912), "resident"),     # 304 tasks of 1 and 3 planes:
    (MIXED, (64, 16, 913), "general"), (FP64, (32, 16, 913), "general"),        # two blocks an SM, not of 4
    (MIXED, (64, 16, 2432), "general"), (MIXED, (128, 128, 128), "general")])
def test_which_kernel(cuda_lib, opts, dims, kernel):
    prob = _problem(dims, OPEN)
    with HeatFlow(prob, **opts) as hf:
        assert hf.inner_solver() == kernel
        later = ("cluster", "resident", "general")
        for name in later[later.index(kernel):]:
            assert hf.inner_solver(name) == name
        assert hf.inner_solver("launches") == "launches"
        hf.set_opts(use_graph=1, **opts)
        assert hf.inner_solver() == "general"                # captured steps
        assert hf.inner_solver("auto") == kernel
    with HeatFlow([prob, prob], **opts) as hf:
        assert hf.inner_solver() == "general"


def _run(arg, steps, first, opts, **kw):
    with HeatFlow(arg, **dict(opts, **kw)) as hf:
        kernel = hf.inner_solver(first)
        hf.initial_evolve()
        st = hf.run(1, steps)
        return kernel, hf.get_state(), [st[k] for k in STATS]


def _equal(arg, opts, ways, steps=3, **kw):
    kernel, ref, stats = _run(arg, steps, "launches", opts, use_graph=0, **kw)
    assert kernel == "launches" and np.isfinite(ref[0]).all()
    for g, first in ways:
        _, got, st = _run(arg, steps, first, opts, use_graph=g, **kw)
        assert st == stats, (g, first)
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1]), (g, first)


@pytest.mark.parametrize("opts", [RECURSIVE, FP64, MIXED], ids=["recursive", "fp64", "mixed"])
@pytest.mark.parametrize("dims,periodic", [((3, 1, 1), OPEN), ((2, 2, 2), WRAP), ((25, 25, 1), OPEN), ((33, 17, 4), WRAP),
                                           ((63, 16, 17), (0, 0, 1)), ((30, 14, 81), (1, 0, 1)), ((65, 33, 24), WRAP),
                                           ((64, 16, 145), (1, 1, 0)), ((150, 97, 60), (0, 1, 0))])
def test_every_kernel_equals_the_launches(cuda_lib, dims, periodic, opts):
    _equal(_problem(dims, periodic), opts, [(g, f) for g in (0, 1) for f in ("auto", "resident", "general")] + [(2, "auto"), (3, "auto")])


@pytest.mark.parametrize("opts", [FP64, MIXED], ids=["fp64", "mixed"])
def test_large_grid_equals_the_launches(cuda_lib, opts):
    """Tasks of 14 (mixed) and 27 planes, rows of 161 cells."""
    _equal(_problem((161, 160, 160), (1, 0, 0)), opts, [(0, "auto"), (1, "auto")], steps=2)


@pytest.mark.parametrize("opts", [RECURSIVE, FP64, MIXED], ids=["recursive", "fp64", "mixed"])
@pytest.mark.parametrize("large", [False, True])
def test_batch_equals_the_launches(cuda_lib, large, opts):
    """Below and above the size from which a batch's solve is split into kernels."""
    grids = [((40, 33, 50), (1, 0, 1)), ((61, 17, 90), OPEN), ((3, 2, 1), (1, 1, 0)), ((24, 70, 31), (0, 1, 0))]
    if large:
        grids += [((90, 96, 96), OPEN), ((97, 61, 45), (0, 0, 1))]
    _equal([_problem(*g) for g in grids], opts, [(0, "auto"), (1, "auto"), (2, "auto")])


@pytest.mark.parametrize("check_every", [1, 7])
@pytest.mark.parametrize("opts", [dict(RECURSIVE, itmax=5), dict(MIXED, inner_itmax=3, max_refine=2)], ids=["fp64", "mixed"])
def test_limits_and_polls(cuda_lib, opts, check_every):
    """Solves that end at their limits, which are no multiples of the polls' distance."""
    _equal(_problem((33, 17, 4), WRAP), opts, [(0, "auto"), (1, "general")], check_every=check_every)


def test_linbcg_by_launches(cuda_lib):
    prob = _problem((33, 17, 4), OPEN)
    rng = np.random.default_rng(3)
    b = rng.uniform(-6e21, -4e21, prob.ncells)
    out = []
    for first in ("auto", "launches"):
        with HeatFlow(prob, **FP64) as hf:
            hf.inner_solver(first)
            out.append(hf.linbcg(b, np.zeros(prob.ncells))[0])
    assert np.array_equal(out[0], out[1])
