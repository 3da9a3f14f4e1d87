"""Element-block inverses at the block sizes and element counts where the
tiles of the register Gauss-Jordan kernels end: M^-1 (D x) = x for the blocks
D of the operator.  An inverse with partial pivoting has a residual of about
cond(D) eps: the blocks of these operators have condition numbers of about
1e4, so 1e-11 (FP64) and 1e-2 (FP32) of the largest entry bound it; the FP64
solution of the same blocks on the host is the reference."""
import numpy as np
import pytest

from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(0, 1e-11), (1, 1e-2)])
@pytest.mark.parametrize("family,p,n", [("gamma", 1, 1), ("gamma", 1, 3), ("omega", 2, 3), ("gamma", 2, 3),
                                        ("omega", 3, 3), ("gamma", 3, 1), ("gamma", 3, 3), ("omega", 4, 3),
                                        ("gamma", 4, 3), ("diage", 1, 1), ("diage", 2, 1)])
def test_inverse_blocks(gpu_lib, family, p, n, precision, tol):
    if family == "diage":
        ms, opts, q = problems.config3(n=n, p=p, seed=2)
        opts = dict(opts, Flux_name="RoeFlux", volume_integral_type=1)
    else:
        ms, opts, q = problems.config1(n=n, p=p, family=family, seed=2)
    g = eulergpu.GPUMesh(ms, opts)
    exact = eulergpu.LinearOperator(g, precision=0)
    exact.calc(q)
    blocks = exact.blocks()[0].transpose(0, 2, 1)   # [E][row][col]
    lo = eulergpu.LinearOperator(g, precision=precision)
    lo.calc(q)
    pc = eulergpu.BlockJacobiPC(lo)
    pc.calc()
    b = np.random.default_rng(1).normal(size=q.shape)
    x = np.linalg.solve(blocks, b.reshape(blocks.shape[0], -1, 1)).reshape(q.shape)
    assert np.abs(pc.apply(b, np.zeros_like(b)) - x).max() <= tol * np.abs(x).max()
