"""Dense element Jacobians of operators with more nodes than the ones that come
with the package: the block beside face tables that do not fit in shared memory,
the block in the output beside face tables, and both outside.

The operator is the p = 4 Omega triangle with further interior nodes, copies of
its own with their own states and entries of Q, which in the wide form are on the
stencil of every face too: the kernels and the oracle take any operator, and the
Jacobian of its residual is defined as well.

Tolerance: that of the other dense-block tests, 1e-10 (FP64) and 1e-5 (FP32) of
the largest entry; an entry is a sum of at most DIM + 3 NF = 17 products."""
import dataclasses

import numpy as np
import pytest

from conftest import oracle_jacobian
from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu

LIMIT = 200 * 1024  # bytes of shared memory


def with_nodes(ms, q, Np, wide):
    op = ms.sbp
    own = op.numnodes
    rng = np.random.default_rng(Np)
    at = np.arange(Np) % own
    Q = rng.uniform(-1.0, 1.0, (op.dim, Np, Np)) * np.abs(op.Q).max()
    Q[:, :own, :own] = op.Q
    perm, interp = op.perm, op.interp
    if wide:
        new = np.tile(np.arange(own, Np, dtype=perm.dtype), (perm.shape[0], 1))
        perm = np.concatenate([perm, new], axis=1)
        interp = np.concatenate([interp, 0.005 * rng.uniform(-1.0, 1.0, interp.shape[:2] + (Np - own,))], axis=2)
    big = dataclasses.replace(op, nodes=op.nodes[at], w=op.w[at], Q=Q, perm=perm, interp=interp)
    mesh = dataclasses.replace(ms, sbp=big, coords=ms.coords[:, at], dxidx=ms.dxidx[:, at], jac=ms.jac[:, at])
    return mesh, np.ascontiguousarray(q[:, at] * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, (q.shape[0], Np, 1))))


@pytest.mark.parametrize("Np, wide, precision, in_global, tables",
                         [(35, False, 0, False, False), (40, False, 0, True, True), (64, False, 0, True, True),
                          (40, True, 0, True, False), (51, False, 1, False, False), (56, False, 1, True, True),
                          (56, True, 1, True, False)])
def test_large_dense_blocks_match_oracle(gpu_lib, oracle, Np, wide, precision, in_global, tables):
    ms, opts, q = problems.config1(n=1, p=4, family="omega", seed=29)
    ms, q = with_nodes(ms, q, Np, wide)
    # the route, from the shared memory of the block and of the face tables
    es, n, S, Nf = (8, 4)[precision], 4 * Np, ms.sbp.stencilsize, ms.sbp.numfacenodes
    fixed, block, faces = es * 2 * Np * (16 + Np), es * n * n, es * 3 * Nf * (S * S + 16)
    assert fixed <= LIMIT and (fixed + block > LIMIT) == in_global
    assert (fixed + (0 if in_global else block) + faces <= LIMIT) == tables
    g = eulergpu.GPUMesh(ms, opts)
    rd, rc = oracle_jacobian(oracle, g.desc, g.params, ms, q)
    scale = max(np.abs(rd).max(), np.abs(rc).max() if rc.size else 0.0)
    lo = eulergpu.LinearOperator(g, precision=precision)
    lo.calc(q)
    d, c = lo.blocks()
    tol = (1e-10, 1e-5)[precision]
    assert np.abs(d - rd).max() <= tol * scale
    assert not c.size or np.abs(c - rc).max() <= tol * scale
