"""A wait between the blocks of the persistent GMRES solve that runs out: the
solve fails with EG_ERR_TIMEOUT, whatever its partition, reduction, precision
or direction, and the same solver then gives the bits it gave before.  The
wait limit is 1 poll (a word of another block takes longer than that to
arrive), so every block leaves by its own bound."""
import contextlib

import numpy as np
import pytest

from pdesolver_gb300 import abi, eulergpu, problems

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _solver(case, precision, grid):
    """a solver of 40 iterations and a right-hand side; closed in order"""
    if case.startswith("tet"):
        ms, opts, q = problems.config3(n=3, p=int(case[3]), seed=5)
        opts = dict(opts, Flux_name="RoeFlux", volume_integral_type=1)
    else:
        ms, opts, q = problems.config1(n=12, p=int(case[-1]), family=case[:-1], seed=8)
    with contextlib.ExitStack() as stack:
        def keep(x):
            stack.callback(x.close)
            return x
        g = keep(eulergpu.GPUMesh(ms, opts))
        lo = keep(eulergpu.LinearOperator(g, precision=precision))
        lo.calc(q)
        pc = keep(eulergpu.BlockJacobiPC(lo))
        pc.calc()
        ls = keep(eulergpu.LinearSolver(pc, lo, restart=30))
        ls.set_tolerances(reltol=0.0, abstol=0.0, itermax=40)
        ls.set_grid(grid)
        yield ls, np.random.default_rng(6).normal(size=q.shape)


def _run(ls, b, transpose, x0=0.0, polls=0):
    """status, solution and iterations of a solve"""
    x = np.full_like(b, x0)
    ls.set_wait_limit(polls)
    try:
        st = (ls.solve_transpose if transpose else ls.solve)(b, x)
    except eulergpu.EulerGPUError as e:
        return e.status, x, -1
    return abi.EG_OK, x, st.iters


@pytest.mark.parametrize("case", ["gamma3", "omega2", "tet2"])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("grid", [0, 20, 100])   # cluster or grid, one- and two-trip reductions
def test_a_wait_that_runs_out(gpu_lib, case, precision, grid):
    with _solver(case, precision, grid) as (ls, b):
        for transpose in (False, True):
            status, good, its = _run(ls, b, transpose)
            assert status == abi.EG_OK and its == 40
            for x0 in (0.0, 1.0):   # a nonzero guess: the first wait is the residual's gather
                assert _run(ls, b, transpose, x0, polls=1)[0] == abi.EG_ERR_TIMEOUT
                status, again, its = _run(ls, b, transpose)
                assert status == abi.EG_OK and its == 40
                assert np.array_equal(again, good)


def test_a_wait_that_runs_out_in_a_batched_launch(gpu_lib):
    with _solver("gamma3", 1, 0) as (ls, b):
        _, good, _ = _run(ls, b, False)
        eulergpu.set_gmres_batching(True)
        try:
            assert _run(ls, b, False, polls=1)[0] == abi.EG_ERR_TIMEOUT
            status, again, its = _run(ls, b, False)
        finally:
            eulergpu.set_gmres_batching(False)
        assert status == abi.EG_OK and np.array_equal(again, good)
