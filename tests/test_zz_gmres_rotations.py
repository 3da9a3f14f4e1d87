"""Hessenberg matrix and Givens rotations of the transposed FP32 solve are FP64
values.  On two elements whose interface flux is scaled by 1e-9, an iteration
lowers the residual by about that factor: after five the estimate is below the
range of FP32 (1e-45), after twelve (1e-108) within that of FP64.  With zero
tolerances the solve then takes its twelve iterations in one cycle; an
estimate that underflows to zero would end cycles early."""
import dataclasses

import numpy as np
import pytest

from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,p", [("gamma", 1), ("omega", 2), ("gamma", 3)])
@pytest.mark.parametrize("precision", [0, 1])
def test_transposed_rotations_in_fp64(gpu_lib, family, p, precision):
    ms, opts, q = problems.config1(n=1, p=p, family=family, seed=3)
    ms = dataclasses.replace(ms, nrm_face=ms.nrm_face * 1e-9)
    g = eulergpu.GPUMesh(ms, opts)
    lo = eulergpu.LinearOperator(g, precision=precision)
    lo.calc(q)
    pc = eulergpu.BlockJacobiPC(lo)
    pc.calc()
    ls = eulergpu.LinearSolver(pc, lo, restart=30)
    ls.set_tolerances(reltol=0.0, abstol=0.0, itermax=12)
    b = np.random.default_rng(2).normal(size=q.shape)
    st = ls.solve_transpose(b, np.zeros_like(b))
    assert (st.iters, st.restarts) == (12, 1)
    for x in (ls, pc, lo, g):
        x.close()
