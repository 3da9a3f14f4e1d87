"""The persistent GMRES solve over what its data flow depends on: dense and
face-diagonal couplings, operators with and without interior nodes, block
partitions on both sides of the one- and two-trip reductions, restart lengths
at their limits, forward and transposed, zero and nonzero initial guesses.

The reference is the explicit Jacobian's own blocks applied on the host in
FP64 (conftest.block_apply); the solver stops on its true residual in its
own precision, so the FP64 residual may exceed the tolerance by the rounding
of one operator application: a factor 3, as for the other GMRES tests.
"""
import numpy as np
import pytest

from conftest import block_apply, block_apply_t
from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu


def _problem(case):
    if case.startswith("tet"):
        ms, opts, q = problems.config3(n=2, p=int(case[3]), seed=5)
        return ms, dict(opts, Flux_name="RoeFlux", volume_integral_type=1), q
    return problems.config1(n=6, p=int(case[-1]), family=case[:-1], seed=8)


@pytest.mark.parametrize("case", ["gamma1", "gamma2", "gamma3", "gamma4", "omega2", "omega4", "tet1", "tet2"])
@pytest.mark.parametrize("precision,tol", [(0, 1e-10), (1, 1e-4)])
def test_solution_for_every_partition(gpu_lib, case, precision, tol):
    ms, opts, q = _problem(case)
    g = eulergpu.GPUMesh(ms, opts)
    lo = eulergpu.LinearOperator(g, precision=0)
    lo.calc(q)
    d, c = lo.blocks()
    lo = eulergpu.LinearOperator(g, precision=precision)
    lo.calc(q)
    pc = eulergpu.BlockJacobiPC(lo)
    pc.calc()
    rng = np.random.default_rng(3)
    # a right-hand side of a known solution of O(1) entries
    for transpose, apply in ((False, block_apply), (True, block_apply_t)):
        b = apply(ms, d, c, rng.normal(size=q.shape))
        for grid, restart, guess in ((0, 30, False), (1, 31, True), (5, 29, False), (48, 30, True), (33, 7, False)):
            ls = eulergpu.LinearSolver(pc, lo, restart=restart)
            ls.set_tolerances(reltol=tol, abstol=0.0, itermax=6000)
            ls.set_grid(grid)
            x = rng.normal(size=q.shape) if guess else np.zeros_like(q)
            st = (ls.solve_transpose if transpose else ls.solve)(b, x)
            assert st.converged == 1, (transpose, grid, restart)
            r = b - apply(ms, d, c, x)
            assert np.linalg.norm(r) <= 3 * tol * np.linalg.norm(b), (transpose, grid, restart)
            ls.close()


def test_repeated_solves_of_one_solver(gpu_lib):
    """tags carry over from solve to solve, also between partitions and
    directions, and a repeated solve gives the same bits."""
    ms, opts, q = _problem("gamma3")
    g = eulergpu.GPUMesh(ms, opts)
    lo = eulergpu.LinearOperator(g, precision=1)
    lo.calc(q)
    pc = eulergpu.BlockJacobiPC(lo)
    pc.calc()
    ls = eulergpu.LinearSolver(pc, lo, restart=30)
    ls.set_tolerances(reltol=0.0, abstol=0.0, itermax=40)
    b = np.random.default_rng(4).normal(size=q.shape)
    first = {}
    for grid in (0, 64, 3, 64, 0, 3):
        ls.set_grid(grid)
        for transpose in (False, True):
            x = np.zeros_like(q)
            st = (ls.solve_transpose if transpose else ls.solve)(b, x)
            assert st.iters == 40
            ref = first.setdefault((grid, transpose), x)
            assert np.array_equal(ref, x), (grid, transpose)
