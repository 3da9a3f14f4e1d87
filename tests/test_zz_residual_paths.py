"""The residual's paths against each other and the oracle: the one-launch
form of small meshes gives the bits of the two-kernel form (the same
arithmetic in the same order), and the split form's fixed-point pair
directions hold on metrics and states far from uniform.

Split-form tolerance: the oracle and the kernel sum the same terms in another
order, Np pairs and a few face nodes of rounding 2^-53 each, relative to the
largest term of the element: 1e-12 of the element's largest residual entry
where the terms do not cancel (metrics scaled by element do not)."""
import dataclasses

import numpy as np
import pytest

from conftest import oracle_residual
from pdesolver_gb300 import eulergpu, problems

pytestmark = pytest.mark.gpu


def _weak(case):
    kind, p, n = case
    if kind == "tet":
        ms, opts, q = problems.config3(n=n, p=p, seed=4)
        return ms, dict(opts, Flux_name="RoeFlux", volume_integral_type=1), q
    if kind == "tetIR":
        ms, opts, q = problems.config3(n=n, p=p, seed=4)
        return ms, dict(opts, volume_integral_type=1), q
    if kind == "wall":
        return problems.annulus_wall(n=n, p=p)
    return problems.config1(n=n, p=p, family=kind, seed=4)


@pytest.mark.parametrize("case", [("gamma", 1, 1), ("gamma", 2, 9), ("gamma", 3, 13), ("gamma", 4, 28), ("omega", 2, 16),
                                  ("omega", 4, 3), ("tet", 1, 5), ("tet", 2, 3), ("tet", 3, 2), ("tetIR", 2, 2),
                                  ("wall", 2, 5)])
def test_small_mesh_form_gives_the_two_kernel_bits(gpu_lib, oracle, case):
    ms, opts, q = _weak(case)
    g = eulergpu.GPUMesh(ms, opts)
    small = g.eval_residual(q, np.zeros_like(q))
    g.set_launch_config(2, False)   # an explicit configuration keeps to the two kernels
    two = g.eval_residual(q, np.zeros_like(q))
    g.set_launch_config(0, False)
    assert np.array_equal(small, two)
    ref = oracle_residual(oracle, g.desc, g.params, q)
    assert np.abs(small - ref).max() <= 1e-12 * np.abs(ref).max()
    # a residual written over its own state
    import torch
    x = torch.from_numpy(q.copy()).cuda()
    g.eval_residual(x, x)
    assert np.array_equal(x.cpu().numpy(), small)
    # an unphysical state is reported, and the next call is clean
    bad = q.copy()
    bad[-1, -1, 0] = -1.0
    with pytest.raises(eulergpu.EulerGPUError):
        g.eval_residual(bad, np.zeros_like(q))
    assert np.array_equal(g.eval_residual(q, np.zeros_like(q)), small)


# (jumps only where face nodes are volume nodes: interpolated to the faces of the
# other operators they are no physical states, and the reference is NaN)
@pytest.mark.parametrize("dim,family,p,jump", [(3, "diage", 1, False), (3, "diage", 2, False), (3, "diage", 3, False),
                                               (3, "diage", 1, True), (3, "diage", 2, True), (3, "diage", 3, True),
                                               (2, "omega", 2, False), (2, "gamma", 2, False)])
def test_split_form_on_uneven_metrics_and_states(gpu_lib, oracle, dim, family, p, jump):
    rng = np.random.default_rng(9)
    if dim == 3:
        ms, opts, q = problems.config3(n=2, p=p, seed=4)
    else:
        ms, opts, q = problems.config1(n=3, p=p, family=family, seed=4)
        opts = dict(opts, Flux_name="IRFlux", volume_integral_type=2, Volume_flux_name="IRFlux")
    E = ms.numEl
    # elements from 2^-30 to 2^30 times their size, stretched in one direction
    scale = np.ldexp(1.0, rng.integers(-30, 31, size=E))[:, None, None, None]
    stretch = np.ones((E, 1, dim, 1))
    stretch[:, 0, 0, 0] = 10.0 ** rng.uniform(-4, 0, size=E)
    ms = dataclasses.replace(ms, dxidx=ms.dxidx * scale * stretch)
    if jump:
        # density and energy by factors up to 5 from node to node: logarithmic means
        f = rng.uniform(0.4, 2.0, size=q.shape[:2] + (1,))
        q = q * f
    g = eulergpu.GPUMesh(ms, opts)
    res = g.eval_residual(q, np.zeros_like(q))
    ref = oracle_residual(oracle, g.desc, g.params, np.ascontiguousarray(q))
    err = np.abs(res - ref).reshape(E, -1).max(1)
    assert np.all(err <= 1e-12 * np.abs(ref).reshape(E, -1).max(1))


# blocks of the narrow, the middle and the widest build of the split kernel, and
# the thread counts on both sides of each edge
@pytest.mark.parametrize("dim,p,epbs", [(3, 1, (1, 50, 73, 74, 100, 146)), (3, 2, (1, 22, 23, 24, 32, 33, 44)),
                                        (2, 2, (1, 73, 74, 109, 110, 146))])
def test_split_form_runs_at_every_block_width(gpu_lib, oracle, dim, p, epbs):
    if dim == 3:
        ms, opts, q = problems.config3(n=4, p=p, seed=4)
    else:
        ms, opts, q = problems.config1(n=12, p=p, family="gamma", seed=4)
        opts = dict(opts, Flux_name="IRFlux", volume_integral_type=2, Volume_flux_name="IRFlux")
    g = eulergpu.GPUMesh(ms, opts)
    ref = oracle_residual(oracle, g.desc, g.params, q)
    widths = set()
    for epb in epbs:
        if epb * ms.sbp.numnodes > 1024:
            continue
        try:
            g.set_launch_config(epb, False)
        except eulergpu.EulerGPUError:
            continue                         # refused for its shared memory
        widths.add(epb * ms.sbp.numnodes)
        r = g.eval_residual(q, np.zeros_like(q))
        assert np.abs(r - ref).max() <= 1e-12 * np.abs(ref).max(), epb
    assert len(widths) >= 4 and max(widths) > 512
