"""The split form's pair directions on stretched elements, each residual
component against its own terms in extended precision.

With velocity along one axis only, the mass and energy equations and that
momentum equation take the direction's own metrics and no others; the metrics
of that direction are made small beside the others (a thin element), so an
error relative to the element's largest metric would dominate them.  The face
normals are scaled to nothing, so the residual is the volume term.

Bound: component c of node j is a sum over its pairs k of F_c(d) n_jk[d].  In
FP64 a term carries the roundings of n_jk (2 DIM products and as many sums), of
the averages and the flux (about 40 operations with condition numbers near 1)
and of the sum (Np): 100 roundings of 2^-53 of sum |n| |F|, with |n| formed of
absolute values."""
import dataclasses

import numpy as np
import pytest

from conftest import oracle_residual
from pdesolver_gb300 import eulergpu, problems

X = np.longdouble


def _logavg(a, b):
    f = (a - b) / (a + b)
    u = f * f
    series = 1 + u * (X(1) / 3 + u * (X(1) / 5 + u * (X(1) / 7 + u * (X(1) / 9))))
    with np.errstate(invalid="ignore", divide="ignore"):
        F = np.where(u < X(1e-3), series, np.log(a / b) / 2 / f)
    return (a + b) / (2 * F)


def split_volume(ms, gamma, q):
    """sum_k -+F_IR(q_j, q_k; n_jk) of every node in extended precision, and
    the same sum of absolute values"""
    d, Np = ms.dim, ms.sbp.numnodes
    q, Q, dx = q.astype(X), ms.sbp.Q.astype(X), ms.dxidx.astype(X)
    g, g1 = X(gamma), X(gamma) - 1
    rho, vel = q[..., 0], q[..., 1:1 + d] / q[..., :1]
    p = g1 * (q[..., -1] - (q[..., 1:1 + d] ** 2).sum(-1) / (2 * rho))
    z1, zp = np.sqrt(rho / p), np.sqrt(rho * p)
    res, mag = np.zeros_like(q), np.zeros_like(q)
    for j in range(Np):
        for k in range(j):
            s1 = z1[:, j] + z1[:, k]
            lp, l1 = _logavg(zp[:, j], zp[:, k]), _logavg(z1[:, j], z1[:, k])
            rh = s1 * lp / 2
            u = (z1[:, j, None] * vel[:, j] + z1[:, k, None] * vel[:, k]) / s1[:, None]
            p1 = (zp[:, j] + zp[:, k]) / s1
            p2 = (g + 1) / (2 * g) * lp / l1 + g1 / (2 * g) * p1
            h = g * p2 / (rh * g1) + (u * u).sum(-1) / 2
            F = np.zeros((d,) + q[:, j].shape, dtype=X)   # unit directions
            for i in range(d):
                F[i, :, 0] = rh * u[:, i]
                F[i, :, 1:1 + d] = (rh * u[:, i])[:, None] * u
                F[i, :, 1 + i] += p1
                F[i, :, -1] = rh * u[:, i] * h
            n = dx[:, j] @ Q[:, j, k] - dx[:, k] @ Q[:, k, j]
            a = np.abs(dx[:, j]) @ np.abs(Q[:, j, k]) + np.abs(dx[:, k]) @ np.abs(Q[:, k, j])
            G, A = np.einsum("ei,iec->ec", n, F), np.einsum("ei,iec->ec", a, np.abs(F))
            res[:, j] -= G
            res[:, k] += G
            mag[:, j] += A
            mag[:, k] += A
    return res, mag


def _case(dim, family, p, thin, axis):
    """a mesh with the metrics of one direction scaled by 10^thin and a state
    moving along it"""
    if dim == 3:
        ms, opts, q = problems.config3(n=2, p=p, seed=4)
    else:
        ms, opts, q = problems.config1(n=3, p=p, family=family, seed=4)
        opts = dict(opts, Flux_name="IRFlux", volume_integral_type=2, Volume_flux_name="IRFlux")
    rng = np.random.default_rng(11)
    rho, c = rng.uniform(0.9, 1.2, size=q.shape[:2]), rng.uniform(0.2, 0.6, size=q.shape[:2])
    q = np.zeros_like(q)
    q[..., 0] = rho
    q[..., 1 + axis] = rho * c
    q[..., -1] = rng.uniform(0.6, 0.8, size=q.shape[:2]) / 0.4 + 0.5 * rho * c * c
    scale = np.ones((1, 1, dim, 1))
    scale[0, 0, axis, 0] = 10.0 ** thin
    size = np.ldexp(1.0, rng.integers(-40, 41, size=ms.numEl))[:, None, None, None]
    tiny = 2.0 ** -300
    return dataclasses.replace(ms, dxidx=ms.dxidx * scale * size, nrm_face=ms.nrm_face * tiny,
                               nrm_bndry=ms.nrm_bndry * tiny), opts, q


CASES = [(3, "diage", 1), (3, "diage", 2), (3, "diage", 3), (2, "omega", 2), (2, "gamma", 3)]


def _within(res, ms, opts, q):
    ref, mag = split_volume(ms, opts["gamma"], q)
    return np.all(np.abs(res - ref) <= 100 * X(2.0) ** -53 * mag)


@pytest.mark.parametrize("dim,family,p", CASES)
def test_reference_and_oracle_agree(oracle, dim, family, p):
    """the FP64 oracle is within the bound of the extended-precision sum"""
    ms, opts, q = _case(dim, family, p, -7.0, 0)
    desc, params = eulergpu.abi.MeshDesc(ms), eulergpu.params_from_opts(opts)
    assert _within(oracle_residual(oracle, desc, params, q), ms, opts, q)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,family,p", CASES)
@pytest.mark.parametrize("thin", [0.0, -3.0, -7.0, -12.0])
def test_thin_direction_keeps_fp64_accuracy(gpu_lib, dim, family, p, thin):
    for axis in range(dim):
        ms, opts, q = _case(dim, family, p, thin, axis)
        g = eulergpu.GPUMesh(ms, opts)
        res = g.eval_residual(q, np.zeros_like(q))
        g.close()
        assert _within(res, ms, opts, q), axis
