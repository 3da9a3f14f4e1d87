"""The dense Jacobian kernels over every triangle operator (their block sizes,
face-node counts and thread counts differ), interior, periodic and boundary
interfaces, down to two elements, against the oracle's blocks.

Tolerance: the bounds of the other block tests, 1e-10 (FP64) and 1e-5 (FP32) of
the largest entry; an entry is a sum of DIM + 3 NF <= 17 products of rounding
2^-53 (2^-24) with the terms no larger than a few of the largest entries."""
import numpy as np
import pytest

from conftest import oracle_jacobian
from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fam", ["gamma", "omega", "wall"])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 3, 9])
def test_dense_blocks_match_oracle(gpu_lib, oracle, fam, p, n):
    if fam == "wall":
        ms, opts, q = problems.annulus_wall(n=n, p=p)
    else:
        ms, opts, q = problems.config1(n=n, p=p, family=fam, seed=23)
    g = eulergpu.GPUMesh(ms, opts)
    rd, rc = oracle_jacobian(oracle, g.desc, g.params, ms, q)
    scale = max(np.abs(rd).max(), np.abs(rc).max() if rc.size else 0.0)
    for prec, tol in ((0, 1e-10), (1, 1e-5)):
        lo = eulergpu.LinearOperator(g, precision=prec)
        lo.calc(q)
        d, c = lo.blocks()
        assert np.abs(d - rd).max() <= tol * scale
        assert not c.size or np.abs(c - rc).max() <= tol * scale
