"""The work that is timed: what a user of the Euler solver has it do.

A pass goes through the public entry points of ``eulergpu`` on device arrays:

* ``residual``   one ``evalResidual`` (checked, as RK and Newton drivers of a
                 host code call it);
* ``rk4``        explicit time steps;
* ``linearise``  what one Newton iteration sets up: the explicit Jacobian, the
                 block-Jacobi inverses, and one application of each;
* ``gmres``      a fixed number of GMRES(30) iterations on the Newton system;
* ``adjoint``    the same on the transposed system;
* ``steady``     a whole steady solve with p-continuation.

Geometries are the quarter annulus (triangles, isentropic vortex data) and
the warped unit cube (tetrahedra, free-stream data) of ``problems.py``.
``precision`` 0 is plain FP64; 1 holds Jacobian, preconditioner and Krylov
vectors in FP32.
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
from pdesolver_gb300 import eulergpu, mesh, problems, sbp  # noqa: E402

GAMMA = 1.4
MACH = 0.5
RESTART = 30
# options of the steady solves (bench.py and the serving stream use the same)
NEWTON = {"res_abstol": 1e-10, "res_reltol": 1e-14, "itermax": 200, "krylov_reltol": 1e-2,
          "newton_globalize_euler": True, "euler_tau": 5.0}
LEVEL_TOL = 1e-4


# --------------------------------------------------------------------- cases
def _case(do, dim, family, p, n, form="weak", precision=0, **more):
    return {"do": do, "dim": dim, "family": family, "p": p, "n": n, "form": form,
            "precision": precision, **more}


def listed():
    return [
        # the vortex verification case: launches and latency are all it is
        dict(_case("residual", 2, "omega", 2, 16), name="residual_annulus16_omega2"),
        # residual of the steady annulus solve
        dict(_case("residual", 2, "gamma", 3, 64), name="residual_annulus64_gamma3"),
        # entropy-stable residual of the explicit 3-D run, the largest mesh
        dict(_case("residual", 3, "diage", 2, 24, "split"), name="residual_cube24_split2"),
        # explicit vortex run: 100 steps of a small mesh
        dict(_case("rk4", 2, "omega", 2, 16, steps=100), name="rk4_annulus16_omega2"),
        # entropy-stable explicit steps on a mesh of odd size
        dict(_case("rk4", 3, "diage", 1, 11, "split", steps=10), name="rk4_cube11_split1"),
        # Newton set-up, plain FP64, 2-D
        dict(_case("linearise", 2, "gamma", 3, 64), name="linearise_annulus64_gamma3_f64"),
        # Newton set-up of a served 3-D request (115-unknown blocks)
        dict(_case("linearise", 3, "diage", 2, 12, precision=1), name="linearise_cube12_p2_f32"),
        # the Krylov solve of the steady annulus problem
        dict(_case("gmres", 2, "gamma", 3, 64, precision=1, its=60), name="gmres_annulus64_gamma3_f32"),
        # the Krylov solve of a served 3-D request
        dict(_case("gmres", 3, "diage", 2, 12, precision=1, its=60), name="gmres_cube12_p2_f32"),
        # adjoint solve of a mid-size annulus, plain FP64
        dict(_case("adjoint", 2, "gamma", 2, 24, its=60), name="adjoint_annulus24_gamma2_f64"),
        # small steady solve of the batched and served mix
        dict(_case("steady", 2, "gamma", 2, 13, precision=1, mach=0.42), name="steady_annulus13_gamma2_f32"),
        # the headline steady solve
        dict(_case("steady", 2, "gamma", 3, 64, precision=1, mach=0.5), name="steady_annulus64_gamma3_f32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["residual", "residual", "rk4", "linearise", "gmres", "gmres", "adjoint", "steady"])
    precision = rng.randint(0, 1)
    if do in ("residual", "rk4"):
        more = {"steps": rng.randint(3, 30)} if do == "rk4" else {}
        if rng.random() < 0.6:
            return _case(do, 2, rng.choice(["omega", "gamma"]), rng.randint(1, 4), _log_int(rng, 8, 96), **more)
        p = rng.randint(1, 3)
        return _case(do, 3, "diage", p, _log_int(rng, 3, {1: 20, 2: 14, 3: 8}[p]),
                     rng.choice(["weak", "split"]), **more)
    if do == "steady":
        mach = round(rng.uniform(0.3, 0.7), 3)
        if rng.random() < 0.75:
            p = rng.randint(1, 4)
            most = {1: (20, 64), 2: (18, 56), 3: (14, 48), 4: (10, 36)}[p][precision]
            return _case(do, 2, "gamma", p, _log_int(rng, 8, most), precision=precision, mach=mach)
        return _case(do, 3, "diage", rng.randint(1, 2), rng.randint(3, 6), precision=precision, mach=mach)
    more = {} if do == "linearise" else {"its": rng.randint(20, 60)}
    if rng.random() < 0.7:
        # SBP-Omega is the family of the FP64 verification runs
        family = "omega" if not precision and rng.random() < 0.4 else "gamma"
        return _case(do, 2, family, rng.randint(1, 4), _log_int(rng, 8, 56), precision=precision, **more)
    form = rng.choice(["weak", "split"]) if do == "linearise" else "weak"
    return _case(do, 3, "diage", rng.randint(1, 2), _log_int(rng, 3, 10), form, precision=precision, **more)


# ------------------------------------------------------------------ geometry
@functools.lru_cache(maxsize=6)
def _mesh(dim, family, p, n):
    op = sbp.get_operator(dim, family, p)
    if dim == 2:
        return mesh.annulus(op, n, n, bc=mesh.BC_VORTEX)
    return mesh.cube(op, n, warp=0.05, seed=3, bc=mesh.BC_FREESTREAM)


def _opts(case):
    opts = {"gamma": GAMMA, "Ma": case.get("mach", MACH), "aoa": 0.0, "Flux_name": "RoeFlux",
            "volume_integral_type": 1}
    if case["dim"] == 2:
        opts["vortex_M_in"] = case.get("mach", MACH)
    if case["form"] == "split":
        opts.update(Flux_name="IRFlux", volume_integral_type=2, Volume_flux_name="IRFlux")
    return opts


def _degrees(case):
    """degrees of the continuation levels"""
    return (1, case["p"]) if case["do"] == "steady" and case["p"] > 1 else (case["p"],)


def _start(case, ms, seed):
    """the state a run starts from: the vortex with 0.1 % noise, the cube's
    free stream with 1 % noise, or (steady) the free stream with 1 % noise"""
    rng = np.random.default_rng(seed)
    mach = case.get("mach", MACH)
    if case["do"] == "steady":
        q = problems.free_stream(case["dim"], ms.coords.shape[:2], Ma=mach)
        return q * (1.0 + rng.uniform(-0.01, 0.01, size=q.shape))
    if case["dim"] == 2:
        q = problems.vortex_state(ms.coords, M_in=mach)
        return q * (1.0 + rng.normal(0.0, 1e-3, size=q.shape))
    q = problems.free_stream(3, ms.coords.shape[:2], Ma=mach)
    q[..., 0] *= 1.0 + rng.normal(0.0, 0.01, size=q.shape[:2])
    return q


def _operand(ms, seed):
    """a vector of O(1) entries (right-hand side, operand of an apply)"""
    shape = ms.coords.shape[:2] + (ms.dim + 2,)
    return np.random.default_rng([seed, 1]).normal(size=shape)


def _time_step(case):
    """0.1 node spacings per unit wave speed, from the mesh size alone"""
    return 0.05 / (case["n"] * case["p"] ** 2)


# ------------------------------------------------------------- prepare / run
class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    s.stream = torch.cuda.Stream()
    meshes = [_mesh(case["dim"], case["family"], p, case["n"]) for p in _degrees(case)]
    s.levels = [eulergpu.GPUMesh(ms, _opts(case)) for ms in meshes]
    for g in s.levels:
        g.set_stream(s.stream.cuda_stream)
    s.g = s.levels[-1]
    with torch.cuda.stream(s.stream):
        s.q = torch.from_numpy(np.ascontiguousarray(_start(case, meshes[0], seed))).cuda()
        if case["do"] == "residual":
            s.res = torch.empty_like(s.q)
        elif case["do"] in ("linearise", "gmres", "adjoint"):
            s.lo = eulergpu.LinearOperator(s.g, precision=case["precision"])
            s.pc = eulergpu.BlockJacobiPC(s.lo)
            s.b = torch.from_numpy(_operand(meshes[0], seed)).cuda()
            if case["do"] == "linearise":
                s.b = s.b.to(torch.float32 if case["precision"] else torch.float64)
                s.y, s.z = torch.empty_like(s.b), torch.empty_like(s.b)
            else:
                s.ls = eulergpu.LinearSolver(s.pc, s.lo, restart=RESTART)
                s.ls.set_tolerances(reltol=0.0, abstol=0.0, itermax=case["its"])
                s.lo.calc(s.q)
                s.pc.calc()
                if case["precision"]:
                    s.b = s.b.to(torch.float32).to(torch.float64)
                s.x = torch.empty_like(s.b)
    s.stream.synchronize()
    return s


def run(s):
    case, do = s.case, s.case["do"]
    with torch.cuda.stream(s.stream):
        if do == "residual":
            s.g.eval_residual(s.q, s.res)
            return s.res
        if do == "rk4":
            q = s.q.clone()
            h = _time_step(case)
            s.g.rk4(q, h, case["steps"] * h)
            return q
        if do == "linearise":
            s.lo.calc(s.q)
            s.pc.calc()
            s.lo.apply_native(s.b, s.y)
            s.pc.apply_native(s.b, s.z)
            return s.y, s.z
        if do in ("gmres", "adjoint"):
            s.x.zero_()
            (s.ls.solve if do == "gmres" else s.ls.solve_transpose)(s.b, s.x)
            # the values are the solver's own precision
            return s.x.to(torch.float32) if case["precision"] else s.x
        q, _ = eulergpu.solve_steady(s.levels, s.q.clone(), NEWTON, precision=case["precision"],
                                     level_tol=LEVEL_TOL)
        return q


# ---------------------------------------------------------------------- work
def _counts(case, p):
    """(elements, nodes, stencil nodes, face nodes, interfaces, boundary faces)"""
    n = case["n"]
    if case["dim"] == 2:
        nodes = {"omega": (3, 6, 10, 15), "gamma": (3, 7, 12, 18)}[case["family"]][p - 1]
        return 2 * n * n, nodes, nodes if case["family"] == "omega" else p + 1, p + 1, 3 * n * n - 2 * n, 4 * n
    nodes, nf = ((6, 3), (23, 9), (45, 15))[p - 1]
    return 6 * n**3, nodes, nf, nf, 12 * n**3 - 6 * n * n, 12 * n * n


def _residual_work(case, p):
    """q, metrics, normals and indices read once, the residual written; flops
    of the contraction or the node pairs, the face interpolation and fluxes"""
    E, Np, S, Nf, I, B = _counts(case, p)
    d = case["dim"]
    nv = d + 2
    by = 8 * (2 * E * Np * nv + E * Np * (d * d + 1) + I * Nf * d + 2 * B * Nf * d) + 4 * (5 * I + 2 * B)
    face = (I + B) * Nf * (130 + (4 * S * nv if d == 2 else 0)) + 2 * (d + 1) * E * Nf * nv * (S if d == 2 else 1)
    if case["form"] == "split":
        fl = E * Np * (Np - 1) // 2 * 96
    else:
        fl = E * Np * d * 14 + 2 * d * Np * Np * nv * E
    return by, fl + face


def _operator_values(case, p):
    """values of the element blocks and of the interface coupling blocks"""
    E, Np, S, _, I, _ = _counts(case, p)
    nv = case["dim"] + 2
    return E * (Np * nv) ** 2, 2 * I * ((S * nv) ** 2 if case["dim"] == 2 else S * nv * nv)


def _krylov_work(case, p, its):
    """one read of the preconditioned operator (element inverses and
    couplings) for each iteration"""
    E, Np, _, _, _, _ = _counts(case, p)
    N = E * Np * (case["dim"] + 2)
    es = 4 if case["precision"] else 8
    values = sum(_operator_values(case, p))
    return its * es * values + 2 * 8 * N, its * (2 * values + 4 * N * min(its, RESTART) / 2)


def _setup_work(case, p):
    """state and metrics read, element blocks, couplings and inverses written"""
    E, Np, _, _, _, _ = _counts(case, p)
    n = Np * (case["dim"] + 2)
    es = 4 if case["precision"] else 8
    diag, cpl = _operator_values(case, p)
    by, fl = _residual_work(case, p)
    return by + es * (2 * diag + cpl), fl + 2 * E * n**3 + 2 * case["dim"] * diag


def work(case):
    do, p = case["do"], case["p"]
    if do == "residual":
        by, fl = _residual_work(case, p)
    elif do == "rk4":
        by, fl = (4 * case["steps"] * v for v in _residual_work(case, p))
    elif do == "linearise":
        by, fl = _setup_work(case, p)
    elif do in ("gmres", "adjoint"):
        by, fl = _krylov_work(case, p, case["its"])
    else:
        # about 20 Newton iterations a level, each of about 5 n Krylov iterations
        by = fl = 0
        for lv in _degrees(case):
            for b, f in (_setup_work(case, lv), _krylov_work(case, lv, 5 * case["n"])):
                by, fl = by + 20 * b, fl + 20 * f
    return {"bytes": by, "flops": fl}


# --------------------------------------------------- the same in 64 bits
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pressure(q):
    m2 = (q[..., 1:-1] ** 2).sum(-1)
    return (GAMMA - 1.0) * (q[..., -1] - 0.5 * m2 / q[..., 0])


def _euler_flux(q, n):
    p = _pressure(q)
    un = (q[..., 1:-1] * n).sum(-1) / q[..., 0]
    return torch.cat([(q[..., 0] * un)[..., None], q[..., 1:-1] * un[..., None] + p[..., None] * n,
                      ((q[..., -1] + p) * un)[..., None]], -1)


def _roe_flux(q, qg, n):
    """Euler flux of q along n plus the Roe dissipation against qg, with the
    eigenvalue floor 0.025 of the spectral radius"""
    def prim(s):
        u = s[..., 1:-1] / s[..., :1]
        return u, (s[..., -1] + _pressure(s)) / s[..., 0]
    uL, hL = prim(q)
    uR, hR = prim(qg)
    sL, sR = q[..., 0].sqrt(), qg[..., 0].sqrt()
    f = 1.0 / (sL + sR)
    u = (sL[..., None] * uL + sR[..., None] * uR) * f[..., None]
    h = (sL * hL + sR * hR) * f
    phi = 0.5 * (u * u).sum(-1)
    area = (n * n).sum(-1).sqrt()
    a = ((GAMMA - 1.0) * (h - phi)).sqrt()
    un = (u * n).sum(-1)
    floor = 0.025 * (un.abs() + area * a)
    l1, l2, l3 = (0.5 * (torch.maximum(v.abs(), floor) - v) for v in (un + area * a, un - area * a, un))
    dq = q - qg
    de = phi * dq[..., 0] - (u * dq[..., 1:-1]).sum(-1) + dq[..., -1]
    dn = (n * dq[..., 1:-1]).sum(-1) - un * dq[..., 0]
    t1 = 0.5 * (l1 + l2) - l3
    t4 = 0.5 * (l1 - l2) / (area * a)
    c1 = t1 * (GAMMA - 1.0) / a**2 * de + t4 * dn
    c2 = t1 / area**2 * dn + t4 * (GAMMA - 1.0) * de
    one, zero = torch.ones_like(un)[..., None], torch.zeros_like(un)[..., None]
    return (_euler_flux(q, n) + l3[..., None] * dq + c1[..., None] * torch.cat([one, u, h[..., None]], -1)
            + c2[..., None] * torch.cat([zero, n, un[..., None]], -1))


def _log_mean(a, b):
    f = (a - b) / (a + b)
    u = f * f
    small = u < 1e-2
    us = torch.where(small, u, torch.zeros_like(u))
    series = torch.zeros_like(us)
    for k in range(10, -1, -1):
        series = series * us + 1.0 / (2 * k + 1)
    fl = torch.where(small, torch.full_like(f, 0.5), f)
    return (a + b) / (2.0 * torch.where(small, series, torch.atanh(fl) / fl))


def _ir_flux(q, qg, n):
    """Ismail-Roe flux along n"""
    pL, pR = _pressure(q), _pressure(qg)
    z1L, z1R = (q[..., 0] / pL).sqrt(), (qg[..., 0] / pR).sqrt()
    z5L, z5R = (q[..., 0] * pL).sqrt(), (qg[..., 0] * pR).sqrt()
    s1 = z1L + z1R
    u = (z1L[..., None] * q[..., 1:-1] / q[..., :1] + z1R[..., None] * qg[..., 1:-1] / qg[..., :1]) / s1[..., None]
    z5 = _log_mean(z5L, z5R)
    rho = 0.5 * s1 * z5
    p1 = (z5L + z5R) / s1
    p2 = (GAMMA + 1.0) / (2.0 * GAMMA) * z5 / _log_mean(z1L, z1R) + (GAMMA - 1.0) / (2.0 * GAMMA) * p1
    h = GAMMA * p2 / (rho * (GAMMA - 1.0)) + 0.5 * (u * u).sum(-1)
    m = rho * (u * n).sum(-1)
    return torch.cat([m[..., None], m[..., None] * u + p1[..., None] * n, (m * h)[..., None]], -1)


class _Exact:
    """R(q_own, q_nbr): the residual with the elements' own state and the
    state that their neighbours show them told apart, in 64 bits."""

    def __init__(self, case):
        self.case = case
        ms = _mesh(case["dim"], case["family"], case["p"], case["n"])
        op, dev = ms.sbp, _device()
        f64 = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        i64 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int64, device=dev)  # noqa: E731
        self.ms, self.split = ms, case["form"] == "split"
        self.Q, self.dxidx, self.wface, self.interp = f64(op.Q), f64(ms.dxidx), f64(op.wface), f64(op.interp)
        self.perm, self.nrm_face, self.nrm_bndry = i64(op.perm), f64(ms.nrm_face), f64(ms.nrm_bndry)
        itf, bf, nbr = i64(ms.interfaces), i64(ms.bndryfaces), i64(ms.nbrperm)
        self.eL, self.eR, self.eB = itf[:, 0], itf[:, 1], bf[:, 0]
        at = torch.arange(itf.shape[0], device=dev)[:, None]
        # interpolation rows of both sides in the order of elementL's face nodes
        self.wL, self.wR = self.interp[itf[:, 2]], self.interp[itf[:, 3]][at, nbr[itf[:, 4]]]
        self.pL, self.pR = self.perm[itf[:, 2]], self.perm[itf[:, 3]]
        self.wB, self.pB = self.interp[bf[:, 1]], self.perm[bf[:, 1]]
        self.qB = self._boundary(f64(ms.coords_bndry))

    def _boundary(self, x):
        if self.case["dim"] == 3:
            q = torch.zeros(x.shape[:-1] + (5,), dtype=x.dtype, device=x.device)
            q[..., 0], q[..., 1] = 1.0, MACH
            q[..., 4] = 1.0 / (GAMMA * (GAMMA - 1.0)) + 0.5 * MACH**2
            return q
        r2 = (x * x).sum(-1)
        k = 0.5 * (GAMMA - 1.0)
        rho = 2.0 * (1.0 + k * MACH**2 * (1.0 - 1.0 / r2)) ** (1.0 / (GAMMA - 1.0))
        p = (rho / 2.0) ** GAMMA / GAMMA
        m2 = ((2.0 / rho) ** (GAMMA - 1.0) * (1.0 + k * MACH**2) - 1.0) / k
        speed = (m2 * GAMMA * p / rho).sqrt()
        r = r2.sqrt()
        return torch.stack([rho, rho * speed * x[..., 1] / r, -rho * speed * x[..., 0] / r,
                            p / (GAMMA - 1.0) + 0.5 * rho * speed**2], -1)

    @staticmethod
    def _at(q, e, w, p):
        return torch.einsum("fis,fsc->fic", w, q[e[:, None], p])

    def _lift(self, res, e, w, p, flux):
        E, Np, nv = res.shape
        add = torch.einsum("fis,i,fic->fsc", w, self.wface, flux)
        at = (e[:, None] * Np + p).reshape(-1)
        return res.reshape(E * Np, nv).index_add(0, at, add.reshape(-1, nv)).reshape(E, Np, nv)

    def _volume(self, q, dx):
        if not self.split:
            return sum(torch.einsum("ij,eic->ejc", self.Q[k], _euler_flux(q, dx[..., k]))
                       for k in range(self.case["dim"]))
        Np = q.shape[1]
        j, k = torch.tril_indices(Np, Np, -1, device=q.device)
        n = sum(dx[:, j][..., m] * self.Q[m][j, k][:, None] - dx[:, k][..., m] * self.Q[m][k, j][:, None]
                for m in range(self.case["dim"]))
        G = _ir_flux(q[:, j], q[:, k], n)
        return torch.zeros_like(q).index_add(1, j, -G).index_add(1, k, G)

    def __call__(self, own, nbr=None):
        nbr = own if nbr is None else nbr
        step = max(1, 2_000_000 // own.shape[1] ** 2)
        res = torch.cat([self._volume(own[a:a + step], self.dxidx[a:a + step])
                         for a in range(0, own.shape[0], step)])
        flux = _ir_flux if self.split else _roe_flux
        fL = flux(self._at(own, self.eL, self.wL, self.pL), self._at(nbr, self.eR, self.wR, self.pR), self.nrm_face)
        fR = flux(self._at(nbr, self.eL, self.wL, self.pL), self._at(own, self.eR, self.wR, self.pR), self.nrm_face)
        fB = _roe_flux(self._at(own, self.eB, self.wB, self.pB), self.qB, self.nrm_bndry)
        res = self._lift(res, self.eL, self.wL, self.pL, -fL)
        res = self._lift(res, self.eR, self.wR, self.pR, fR)
        return self._lift(res, self.eB, self.wB, self.pB, -fB)

    # Jacobian at q: coupling C z, its transpose, and the element blocks
    def at(self, q):
        self.q = q
        E, Np, nv = q.shape
        n = Np * nv
        D = torch.empty(E, n, n, dtype=q.dtype, device=q.device)
        for c in range(n):
            v = torch.zeros(E, n, dtype=q.dtype, device=q.device)
            v[:, c] = 1.0
            D[:, :, c] = torch.func.jvp(lambda s: self(s, q), (q,), (v.reshape(q.shape),))[1].reshape(E, n)
        self.D = D
        self.lu = torch.linalg.lu_factor(D)
        self.back = torch.func.vjp(lambda s: self(q, s), q)[1]
        return self

    def couple(self, z, transpose):
        if transpose:
            return self.back(z)[0]
        return torch.func.jvp(lambda s: self(self.q, s), (self.q,), (z,))[1]

    def block(self, z, transpose=False):
        D = self.D.mT if transpose else self.D
        return (D @ z.reshape(z.shape[0], -1, 1)).reshape(z.shape)

    def block_solve(self, z, transpose=False):
        b = z.reshape(z.shape[0], -1, 1)
        return torch.linalg.lu_solve(*self.lu, b, adjoint=transpose).reshape(z.shape)


def _gmres(A, b, its, transpose):
    """`its` iterations of right-preconditioned GMRES(RESTART) from zero"""
    x = torch.zeros_like(b)
    while its > 0:
        r = b - A.block(x, transpose) - A.couple(x, transpose)
        V = [r / r.norm()]
        m = min(RESTART, its)
        H = torch.zeros(m + 1, m, dtype=b.dtype)
        for j in range(m):
            w = V[j] + A.couple(A.block_solve(V[j], transpose), transpose)
            for _ in range(2):
                for k, v in enumerate(V):
                    h = (v * w).sum()
                    w = w - h * v
                    H[k, j] += h.cpu()
            H[j + 1, j] = w.norm().cpu()
            V.append(w / w.norm())
        g = torch.zeros(m + 1, 1, dtype=b.dtype)
        g[0] = r.norm().cpu()
        y = torch.linalg.lstsq(H, g, driver="gelsd").solution[:, 0].tolist()
        x = x + A.block_solve(sum(c * v for c, v in zip(y, V)), transpose)
        its -= m
    return x


def exact(case, seed):
    if case["do"] == "steady":
        return None  # a Newton solve in plain torch takes minutes
    A = _Exact(case)
    q = torch.tensor(_start(case, A.ms, seed), device=_device())
    if case["do"] == "residual":
        return A(q)
    if case["do"] == "rk4":
        h = _time_step(case)
        Minv = torch.tensor(1.0 / A.ms.M, device=q.device)[..., None]
        for _ in range(case["steps"]):
            k1 = Minv * A(q)
            k2 = Minv * A(q + 0.5 * h * k1)
            k3 = Minv * A(q + 0.5 * h * k2)
            k4 = Minv * A(q + h * k3)
            q = q + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        return q
    b = torch.tensor(_operand(A.ms, seed), device=q.device)
    if case["precision"]:
        b = b.to(torch.float32).to(torch.float64)
    A.at(q)
    if case["do"] == "linearise":
        return A.block(b) + A.couple(b, False), A.block_solve(b)
    return _gmres(A, b, case["its"], case["do"] == "adjoint")
