"""A metric or Q entry that is not finite makes the split-form residual not
finite where it enters, as in the oracle, and a Newton solve ends with an
error."""
import dataclasses

import numpy as np
import pytest

from conftest import oracle_residual
from pdesolver_gb300 import abi, eulergpu, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["metric", "Q"])
@pytest.mark.parametrize("p", [1, 2, 3])
def test_not_finite_in_not_finite_out(gpu_lib, oracle, value, where, p):
    ms, opts, q = problems.config3(n=2, p=p, seed=4)
    if where == "metric":
        dxidx = ms.dxidx.copy()
        dxidx[3, 2, 1, 0] = value
        bad = dataclasses.replace(ms, dxidx=dxidx)
    else:
        Q = ms.sbp.Q.copy()
        Q[1, 0, 2] = value
        bad = dataclasses.replace(ms, sbp=dataclasses.replace(ms.sbp, Q=Q))
    g = eulergpu.GPUMesh(bad, opts)
    res = g.eval_residual(q, np.zeros_like(q))
    ref = oracle_residual(oracle, g.desc, g.params, q)
    finite = np.isfinite(ref)
    assert np.array_equal(np.isfinite(res), finite)
    assert not finite.all() and (where == "Q" or finite.any())
    ok = eulergpu.GPUMesh(ms, opts)
    good = ok.eval_residual(q, np.zeros_like(q))
    assert np.abs(np.where(finite, res - good, 0.0)).max() <= 1e-12 * np.abs(good).max()
    status = abi.EG_OK
    try:
        g.newton(q.copy(), {"itermax": 2}, precision=0)
    except eulergpu.EulerGPUError as e:
        status = e.status
    assert status == abi.EG_ERR_NONFINITE
    g.close()
    ok.close()
