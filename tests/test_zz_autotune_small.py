"""On a mesh whose built-in configuration is the one-launch residual, the
autotuner times that configuration beside the explicit ones, and keeps it when
it is the fastest."""
import numpy as np
import pytest

from conftest import oracle_residual
from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,own", [(3, True), (16, True), (28, True), (29, False)])
def test_builtin_configuration_is_a_candidate(gpu_lib, oracle, n, own):
    import torch
    ms, opts, q = problems.config1(n=n, p=2, family="omega", seed=4)
    g = eulergpu.GPUMesh(ms, opts)
    g.set_launch_config(2, False)      # a setting of the caller's does not hide it
    table = g.autotune(torch.from_numpy(q).cuda(), reps=5)
    builtin = {"elements_per_cta": 0, "volume_mma": False}
    assert any(c == builtin for c, _ in table) == own
    assert g.launch_config() == min(table, key=lambda t: t[1])[0]
    ref = oracle_residual(oracle, g.desc, g.params, q)
    assert np.abs(g.eval_residual(q, np.zeros_like(q)) - ref).max() <= 1e-12 * np.abs(ref).max()
    g.close()
