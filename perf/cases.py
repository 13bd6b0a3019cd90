"""Performance cases: what a user of this framework has it do, through its public entry points.

A case's ``kind`` names the call:

* ``step``    one time step of :class:`FlowSolver` from a given state, the state read back (the call of a
              host program that drives the simulation): 3 nonlinear iterations of ElmGMR + memLS solve;
* ``newton``  one nonlinear iteration on the device: ``ElmGMR.device`` + ``MemLS.solflow_device``;
* ``adjoint`` the preconditioner of one adjoint iteration: the transposed memLS solve;
* ``vjp``     the exact vector-Jacobian product of the residual (backward of the assembly);
* ``asm``     ElmGMR residual + tangent, ``res`` the residual alone;
* ``sclr``    ElmGMRSclr residual + tangent of an advected scalar;
* ``spmv``    the 4x4 block product on the assembled pattern.

Meshes are the repository's own synthetic ones: ``cylinder`` (a x a cross-section, b layers, c outlets),
``bifurcation`` (grid spacing 2 / a) and ``lattice`` (a^3 cells).  A mesh is kept for the life of the
process, as a program that runs several solvers on one geometry keeps it; every ``prepare`` builds its own
solver objects and a new state from the seed.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from crimsonflowsolver_b200 import RCR, FlowParams, _native as N, mesh, solver
from crimsonflowsolver_b200.solver import FlowSolver

DEV = "cuda"


def _case(kind, geo, a, b=0, outlets=0, precision="fp64", name=None):
    c = {"kind": kind, "geo": geo, "a": a, "b": b, "outlets": outlets, "precision": precision}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest simulation anybody runs (a smoke test, a 0D-coupling study): launches and latency
        _case("step", "cylinder", 6, 6, 1, name="step_1k_fp64"),
        # the plain CPU-runnable workload, 107,520 tets
        _case("step", "cylinder", 24, 40, 1, name="step_108k_fp64"),
        # an ordinary bifurcation with two outlets in the mixed mode
        _case("step", "bifurcation", 27, 0, 2, "mixed", name="step_ybif_mixed"),
        # three outlets, mixed mode with the FP32 quadrature of the tangent, odd sizes
        _case("step", "cylinder", 37, 101, 3, "mixed_f32_tangent", name="step_657k_f32tangent"),
        # the headline workload: 4.0M tets, mixed
        _case("step", "cylinder", 80, 133, 1, "mixed", name="step_4m_mixed"),
        # the same mesh in plain FP64, one nonlinear iteration
        _case("newton", "cylinder", 80, 133, 1, name="newton_4m_fp64"),
        # the adjoint's preconditioner on a mid-size multi-outlet cylinder
        _case("adjoint", "cylinder", 24, 61, 3, name="adjoint_164k"),
        # the adjoint's exact residual derivative on the 1M-tet 3-outlet cylinder
        _case("vjp", "cylinder", 40, 133, 3, name="vjp_1m"),
        # the assembly microbenchmark at 6M tets
        _case("asm", "lattice", 100, name="asm_6m"),
        # residual evaluations (line searches, the primal of the adjoint), ragged size
        _case("res", "cylinder", 31, 47, 1, name="res_210k"),
        # transport of a scalar on an ordinary mesh
        _case("sclr", "lattice", 64, name="sclr_1.6m"),
        # block SpMV, plain arithmetic
        _case("spmv", "lattice", 83, name="spmv_3.4m_fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["step", "step", "newton", "adjoint", "vjp", "asm", "res", "sclr", "spmv"])
    if kind == "step":
        geo = rng.choice(["cylinder", "cylinder", "bifurcation"])
        prec = rng.choice(["fp64", "mixed", "mixed_f32_tangent"])
        if geo == "bifurcation":
            return _case(kind, geo, _log(rng, 8, 36), 0, 2, prec)
        return _case(kind, geo, _log(rng, 5, 48), _log(rng, 6, 120), rng.randint(1, 4), prec)
    if kind in ("newton", "adjoint"):
        prec = rng.choice(["fp64", "mixed"])
        return _case(kind, "cylinder", _log(rng, 5, 48), _log(rng, 6, 120), rng.randint(0, 3), prec)
    if kind == "vjp":
        return _case(kind, "cylinder", _log(rng, 5, 40), _log(rng, 6, 133), rng.randint(1, 4))
    if kind == "spmv":
        return _case(kind, "lattice", _log(rng, 12, 90), precision=rng.choice(["fp64", "mixed"]))
    if rng.random() < 0.5:
        return _case(kind, "lattice", _log(rng, 6, 95), precision="fp64")
    return _case(kind, "cylinder", _log(rng, 5, 48), _log(rng, 6, 120), rng.randint(1, 4))


_MESHES = {}


def _mesh(case):
    key = (case["geo"], case["a"], case["b"], case["outlets"])
    if key not in _MESHES:
        if len(_MESHES) > 3:
            _MESHES.clear()
        if case["geo"] == "lattice":
            m = mesh.lattice(case["a"])
        elif case["geo"] == "bifurcation":
            m = mesh.bifurcation(h=2.0 / case["a"])
        else:
            m = mesh.cylinder(ncross=case["a"], naxial=case["b"], n_outlets=max(1, case["outlets"]))
        _MESHES[key] = m
    return _MESHES[key]


def _params(case, m, rng):
    """Nominal RCR values +-20%; no outlet model where the case has no coupled outlets."""
    rcr = []
    if case["outlets"]:
        for s in m.outlets:
            f = rng.uniform(0.8, 1.2, 3)
            rcr.append(RCR(srfid=s, Rp=100.0 * f[0], C=1e-4 * f[1], Rd=1000.0 * f[2]))
    return FlowParams(rcr=rcr, precision=case["precision"] if case["kind"] not in ("spmv",) else "fp64")


def _state(m, rng):
    """A flow state: N(0, 1) nodal values on the lattice; on a tube the parabolic profile of its inlet (scaled
    to the seed's speed) with 2% perturbations off the prescribed nodes, and a few per cent of it as acceleration."""
    n = m.nshg
    if m.inlet_nodes is None:
        return rng.standard_normal((n, 4)), rng.standard_normal((n, 4))
    u0 = rng.uniform(8.0, 12.0)
    y = np.zeros((n, 4))
    # where along the tube's axis the profile applies: the first 4 cm (straight in every geometry)
    prof = 2.0 * u0 * np.clip(1.0 - m.x[:, 0] ** 2 - m.x[:, 1] ** 2, 0.0, None)
    y[:, 2] = prof * np.clip(5.0 - m.x[:, 2], 0.0, 1.0)
    y[:, :3] += 0.02 * u0 * rng.standard_normal((n, 3))
    y[:, 3] = 50.0 * (m.x[:, 2].max() - m.x[:, 2]) + 5.0 * rng.standard_normal(n)
    ac = np.zeros((n, 4))
    ac[:, :3] = 0.05 * u0 * rng.standard_normal((n, 3))
    full = ((m.iBC >> 3) & 7) == 7
    y[full, :3] = 0.0
    ac[full, :3] = 0.0
    y[m.inlet_nodes, :3] = m.inlet_profile * u0
    return y, ac


def _inputs(case, seed):
    """(mesh, parameters, y, ac, coef1, coef2) of a case: everything that does not need the GPU."""
    m = _mesh(case)
    rng = np.random.default_rng([seed, 17])
    P = _params(case, m, rng)
    y, ac = _state(m, rng)
    nc = len(P.rcr)
    return m, P, y, ac, rng.uniform(100.0, 200.0, nc), rng.uniform(-5.0, 5.0, nc)


def _randn(seed, *shape, dtype=torch.float64):
    return torch.randn(shape, dtype=dtype, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


def _memls(m, P, elm):
    ms = solver.MemLS(P, 1 + len(P.rcr), ctx=elm)
    ms.bc_create(1, *_face(solver.dirichlet_face(m), 0))
    for k, r in enumerate(P.rcr):
        ms.bc_create(2 + k, *_face(solver.neumann_face(m, r.srfid), 1))
    return ms


def _face(nodes_val, bctype):
    return nodes_val[0], 3, bctype, nodes_val[1]


class _State:
    """What a program holds between calls: the solver objects and its buffers."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        if torch is None:  # the interpreter is shutting down
            return
        # an lhs is freed before the context it borrows from
        for k in ("F", "ms", "elm"):
            obj = self.__dict__.get(k)
            if obj is not None:
                torch.cuda.synchronize()
                obj.close()


def prepare(case, seed):
    kind = case["kind"]
    m, P, y, ac, c1, c2 = _inputs(case, seed)
    if kind == "step":
        rng = np.random.default_rng([seed, 23])
        u0 = rng.uniform(8.0, 12.0)
        F = FlowSolver(m, P, inflow=lambda t: u0 + 5.0 * np.sin(2.0 * np.pi * t / 0.8))
        nc = len(P.rcr)
        return _State(kind=kind, F=F, y=np.asfortranarray(y), ac=np.asfortranarray(ac), Pn=rng.uniform(0.0, 100.0, nc),
                      Qn=rng.uniform(5.0, 15.0, nc))
    elm = solver.ElmGMR(m, P)
    n, nnz = m.nshg, elm._nnz()
    st = _State(kind=kind, elm=elm, P=P, nnz=nnz, y=torch.tensor(y, device=DEV), ac=torch.tensor(ac, device=DEV), c1=c1,
                c2=c2)
    new = lambda *s: torch.empty(s, dtype=torch.float64, device=DEV)  # noqa: E731
    if kind in ("asm", "newton", "adjoint"):
        st.lhsK, st.lhsP = new(nnz, 9), new(nnz, 4)
    if kind in ("asm", "res", "newton", "adjoint", "vjp"):
        st.res = new(n, 4)
    if kind in ("newton", "adjoint"):
        st.ms, st.sol = _memls(m, P, elm), new(n, 4)
        st.faceRes = np.concatenate([[0.0], c1 * P.alfi * P.gami * P.Delt])
    if kind == "adjoint":
        # the tangent of the step that is reversed, and a unit-norm cotangent on the free rows
        elm.device(st.y, st.ac, st.res, st.lhsK, st.lhsP, c1, c2)
        torch.cuda.synchronize()
        st.rhs = st.res / torch.linalg.norm(st.res)
    if kind == "vjp":
        st.lam, st.ybar, st.abar = _randn(seed, n, 4), new(n, 4), new(n, 4)
    if kind == "sclr":
        st.s, st.sdot = _randn(seed, n), _randn(seed + 1, n)
        st.res, st.lhsS = new(n), new(nnz)
    if kind == "spmv":
        dt = torch.float64 if case["precision"] == "fp64" else torch.float32
        val = _randn(seed, nnz, 16, dtype=dt)
        st.u = _randn(seed + 1, n, 4, dtype=dt)
        st.ku = torch.empty_like(st.u)
        torch.cuda.synchronize()
        N.check(N.lib().crimson_spmv4_prepare(elm.h, 0 if dt == torch.float64 else 1, val.data_ptr()), "spmv4_prepare")
    torch.cuda.synchronize()
    return st


def run(st):
    L = N.lib()
    if st.kind == "step":
        F = st.F
        F.istep = 0
        F.set_state(st.y, st.ac)
        nc = len(st.Pn)
        if nc:
            N.check(L.crimson_rcr_state(F.elm.h, nc, N.dp(st.Pn.copy()), N.dp(st.Qn.copy()), 1), "crimson_rcr_state")
        s = F.step()
        y, ac = F.state()
        return {"y": y, "ac": ac, "q": np.array(s.q_out[:nc]), "p": np.array(s.p_out[:nc])}
    if st.kind == "newton":
        st.elm.device(st.y, st.ac, st.res, st.lhsK, st.lhsP, st.c1, st.c2)
        st.ms.solflow_device(st.elm, st.res, st.lhsK, st.lhsP, st.faceRes, st.sol)
        return {"res": st.res, "sol": st.sol}
    if st.kind == "adjoint":
        ls, inc = N.LsStats(), np.ones(len(st.faceRes), dtype=np.int32)
        N.check(L.crimson_solflow_device_transposed(st.elm.h, st.ms.lhs, st.ms.ls, st.rhs.data_ptr(), st.lhsK.data_ptr(),
                                                    st.lhsP.data_ptr(), N.ip(inc), N.dp(st.faceRes), st.sol.data_ptr(),
                                                    ctypes.byref(ls)), "crimson_solflow_device_transposed")
        return {"sol": st.sol}
    if st.kind == "vjp":
        nc = len(st.c1)
        mub, c1b, c2b = ctypes.c_double(), np.zeros(max(nc, 1)), np.zeros(max(nc, 1))
        N.check(L.crimson_elmgmr_vjp(st.elm.h, st.y.data_ptr(), st.ac.data_ptr(), N.dp(st.c1), N.dp(st.c2),
                                     st.lam.data_ptr(), st.res.data_ptr(), st.ybar.data_ptr(), st.abar.data_ptr(),
                                     ctypes.byref(mub), N.dp(c1b), N.dp(c2b)), "crimson_elmgmr_vjp")
        return {"res": st.res, "ybar": st.ybar, "abar": st.abar, "mubar": mub.value, "c1bar": c1b[:nc], "c2bar": c2b[:nc]}
    if st.kind == "asm":
        st.elm.device(st.y, st.ac, st.res, st.lhsK, st.lhsP, st.c1, st.c2)
        return {"res": st.res, "lhsK": st.lhsK, "lhsP": st.lhsP}
    if st.kind == "res":
        st.elm.device(st.y, st.ac, st.res, None, None, st.c1, st.c2, lhs=False)
        return {"res": st.res}
    if st.kind == "sclr":
        st.elm.sclr_device(st.y, st.s, st.sdot, st.res, st.lhsS, isclr=1, diffus=0.1)
        return {"res": st.res, "lhsS": st.lhsS}
    N.check(L.crimson_spmv4_apply(st.elm.h, st.u.data_ptr(), st.ku.data_ptr()), "crimson_spmv4_apply")
    return {"ku": st.ku}


def _sizes(case):
    """(elements, nodes, blocks) from the construction alone: 6 tets per cell, about 15 blocks per node."""
    a, b = case["a"], case["b"]
    if case["geo"] == "lattice":
        cells, n = a ** 3, (a + 1) ** 3
    elif case["geo"] == "bifurcation":
        cells = int((np.pi * 5.2 + 2 * np.pi * 0.49 * 4.6) * (a / 2.0) ** 3)
        n = cells * 1.06
    else:
        cells, n = int(np.pi / 4 * a * a) * b, int(np.pi / 4 * (a + 1.3) ** 2) * (b + 1)
    return 6.0 * cells, float(n), 14.6 * n


def work(case):
    """Compulsory bytes (each input read once, each output written once) and operations of one pass.  A solve
    reads the assembled matrix at least once and its operations are counted for one product with it: how
    many an iterative solve needs is not known beforehand."""
    ne, n, nnz = _sizes(case)
    kind = case["kind"]
    mesh_b, state_b = 16 * ne + 24 * n, 56 * n
    lhs_b = 104 * nnz
    if kind == "step":
        return {"bytes": 2 * 64 * n + mesh_b + 3 * lhs_b, "flops": 3 * (2600 * ne + 40 * nnz)}
    if kind == "newton":
        return {"bytes": state_b + mesh_b + 64 * n + lhs_b, "flops": 2600 * ne + 40 * nnz}
    if kind == "adjoint":
        return {"bytes": 64 * n + lhs_b, "flops": 40 * nnz}
    if kind == "vjp":
        return {"bytes": state_b + mesh_b + 32 * n + 96 * n, "flops": 4000 * ne}
    if kind == "asm":
        return {"bytes": state_b + mesh_b + 32 * n + lhs_b, "flops": 2600 * ne}
    if kind == "res":
        return {"bytes": state_b + mesh_b + 32 * n, "flops": 1200 * ne}
    if kind == "sclr":
        return {"bytes": mesh_b + 40 * n + 8 * n + 8 * nnz, "flops": 1100 * ne}
    size = 8 if case["precision"] == "fp64" else 4
    return {"bytes": (16 * size + 4) * nnz + 8 * size * n, "flops": 32 * nnz}


# ---------------------------------------------------------------------------------------------
# exact(): the same quantities in plain torch, 64 bits, element by element as the formulation
# is written (SUPG/PSPG on linear tets, 4-point rule), scattered with index_add.
# ---------------------------------------------------------------------------------------------
_A4, _B4 = 0.5854101966249685, 0.1381966011250150
_B3, _C3, _A3 = 0.666666666666667, 0.166666666666667, 0.333333333333333


def _interior_rule():
    r = torch.full((4, 4), _B4, dtype=torch.float64, device=DEV)
    r[0, 0] = r[1, 1] = r[2, 2] = _A4
    r[:, 3] = 1.0 - r[:, 0] - r[:, 1] - r[:, 2]
    return r  # [point][node]


class _Geometry:
    """Element metrics of a set of tets: shape gradients, weight and metric tensor."""

    def __init__(self, x, ien):
        xe = x[ien]                                             # (e, 4, 3)
        d = 0.5 * (xe[:, :3] - xe[:, 3:]).transpose(1, 2)       # d x_i / d xi_j
        dxi = torch.linalg.inv(d)                               # d xi_i / d x_j
        self.W = torch.linalg.det(d) / 3.0
        self.g = torch.cat([0.5 * dxi, -0.5 * dxi.sum(1, keepdim=True)], 1)   # grad N_a (e, 4, 3)
        c1, c2 = 1.259921049894873, 0.6299605249474365
        C = torch.full((3, 3), c2, dtype=torch.float64, device=DEV) + (c1 - c2) * torch.eye(3, dtype=torch.float64, device=DEV)
        self.G = dxi.transpose(1, 2) @ (C @ dxi)


def _scatter(ien, v, n):
    return torch.zeros((n,) + v.shape[2:], dtype=torch.float64, device=DEV).index_add(0, ien.reshape(-1), v.reshape((-1,) + v.shape[2:]))


def _slots(ien, n):
    """Unique (row, column) pairs of the node graph in row order and the slot of each element pair."""
    key = (ien[:, :, None] * n + ien[:, None, :]).reshape(-1)
    u, inv = torch.unique(key, return_inverse=True)
    return u.numel(), inv.reshape(-1, 4, 4)


def _points(P, geo, yl, al, divq, mu):
    """Per quadrature point: u, acceleration, pressure, strong residual, tauM, tauC, tauBar, uBar."""
    rho = P.rho
    gy = torch.einsum("eak,ead->ekd", geo.g, yl)                # d y_d / d x_k; y = (u, v, w, p)
    gg = (geo.G * geo.G).sum((1, 2))
    tr = geo.G.diagonal(dim1=1, dim2=2).sum(1)
    dts = 2.0 / P.Delt * P.dtsfct
    for N_ in _interior_rule():
        u, a, p = torch.einsum("a,eai->ei", N_, yl[..., :3]), torch.einsum("a,eai->ei", N_, al), yl[..., 3] @ N_
        L_ = rho * (a + torch.einsum("ek,eki->ei", u, gy[..., :3])) + gy[..., 3] - divq
        fact = torch.sqrt(dts ** 2 + torch.einsum("ei,eij,ej->e", u, geo.G, u) + 36.0 * (mu / rho) ** 2 * gg)
        tb = torch.einsum("ei,eij,ej->e", L_, geo.G, L_)
        tM = 1.0 / fact
        tB = torch.where(tb != 0, tM / torch.sqrt(torch.where(tb != 0, tb, torch.ones_like(tb))), tb)
        yield N_, u, a, p, gy, L_, tM, rho * 0.125 * fact / tr * (P.taucfct / P.dtsfct), tB, u - tM[:, None] * L_ / rho


def _projection(geo, ien, y, mu, n):
    """Lumped projection of the viscous flux mu (grad u + grad u^T): (n, 3, 3)."""
    gu = torch.einsum("eak,eai->eki", geo.g, y[ien][..., :3])
    q = mu * (gu + gu.transpose(1, 2))
    SN = _interior_rule().sum(0)
    w = geo.W[:, None] * SN
    return _scatter(ien, w[:, :, None, None] * q[:, None], n) / _scatter(ien, w, n)[:, None, None]


def _residual(m, P, y, ac, mu, c1, c2):
    """res (n, 4) with projection, boundary faces, outlet coupling and the prescribed rows zeroed."""
    n, rho = m.nshg, P.rho
    x = torch.tensor(m.x, device=DEV)
    ien = torch.tensor(m.ien.astype(np.int64), device=DEV)
    geo = _Geometry(x, ien)
    yl, al = y[ien], ac[ien][..., :3]
    divq = torch.einsum("eaj,eaji->ei", geo.g, _projection(geo, ien, y, mu, n)[ien])
    rl = 0.0
    for N_, u, a, p, gy, L_, tM, tC, tB, ub in _points(P, geo, yl, al, divq, mu):
        gu = gy[..., :3]
        rN = rho * (a + torch.einsum("ek,eki->ei", ub, gu))
        div = gu.diagonal(dim1=1, dim2=2).sum(1)
        S = mu * (gu + gu.transpose(1, 2)) + (tC * div - p)[:, None, None] * torch.eye(3, dtype=torch.float64, device=DEV)
        S = S + (tM[:, None] * L_)[:, :, None] * u[:, None, :]
        S = S + (tB[:, None] * torch.einsum("ek,eki->ei", L_, gu))[:, :, None] * L_[:, None, :]
        mom = N_[None, :, None] * rN[:, None, :] + torch.einsum("eaj,eij->eai", geo.g, S)
        rl = rl + torch.cat([-mom, torch.einsum("eai,ei->ea", geo.g, ub)[..., None]], -1) * geo.W[:, None, None]
    res = _scatter(ien, rl, n)
    if m.ienb is not None and len(m.ienb):
        ienb = torch.tensor(m.ienb.astype(np.int64), device=DEV)
        res = res + _boundary(m, P, x, ienb, y, mu, n)
    for k, r in enumerate(P.rcr):
        nodes = torch.tensor(np.nonzero(m.ndsurf == r.srfid)[0], device=DEV)
        nabi = torch.tensor(m.NABI[nodes.cpu().numpy()], device=DEV)
        Q = (nabi * y[nodes][:, :3]).sum()
        res = res.index_add(0, nodes, torch.cat([-(Q * c1[k] + c2[k]) * nabi, torch.zeros_like(nabi[:, :1])], 1))
    vel = torch.tensor(((m.iBC >> 3) & 7) == 7, device=DEV)
    pre = torch.tensor(((m.iBC >> 2) & 1) == 1, device=DEV)
    keep = torch.stack([~vel, ~vel, ~vel, ~pre], 1)
    return torch.where(keep, res, torch.zeros_like(res))


def _boundary(m, P, x, ienb, y, mu, n):
    """Traction, pressure and influx stabilisation of the boundary faces (rigid wall, zero natural pressure)."""
    geo, xb, yl = _Geometry(x, ienb), x[ienb], y[ienb]
    nrm = torch.linalg.cross(xb[:, 1] - xb[:, 0], xb[:, 2] - xb[:, 0])
    area2 = torch.linalg.norm(nrm, dim=1)
    nrm, Wb = nrm / area2[:, None], 2.0 * _A3 * area2 / 4.0
    gu = torch.einsum("eak,eai->eki", geo.g, yl[..., :3])
    tau = torch.einsum("ek,eki->ei", nrm, mu * (gu + gu.transpose(1, 2)))
    tn = (nrm * tau).sum(1)
    natural = torch.tensor(((m.iBCB[:, 0] >> 1) & 1) == 1, device=DEV)
    out = 0.0
    for q in range(3):
        Nb = torch.full((3,), _C3, dtype=torch.float64, device=DEV)
        Nb[q] = _B3
        u, p = torch.einsum("a,eai->ei", Nb, yl[:, :3, :3]), yl[:, :3, 3] @ Nb
        un = (nrm * u).sum(1)
        p = torch.where(natural, torch.zeros_like(p), p - tn)
        back = torch.where(natural & (un < 0), un, torch.zeros_like(un))
        f = -(tau - nrm * tn[:, None]) + nrm * p[:, None] - P.stabflux_coeff * P.rho * back[:, None] * u
        f = torch.cat([f, un[:, None]], 1) * Wb[:, None]
        out = out - Nb[None, :, None] * f[:, None, :]
    return _scatter(ienb[:, :3], out, n)


def _tangent(m, P, y, ac, mu):
    """lhsK (nnz, 9) and lhsP (nnz, 4) as the formulation's approximate Jacobian."""
    n, rho = m.nshg, P.rho
    ien = torch.tensor(m.ien.astype(np.int64), device=DEV)
    geo = _Geometry(torch.tensor(m.x, device=DEV), ien)
    divq = torch.einsum("eaj,eaji->ei", geo.g, _projection(geo, ien, y, mu, n)[ien])
    nnz, slot = _slots(ien, n)
    lf, W, g = P.alfi * P.gami * P.Delt, geo.W, geo.g
    gab = torch.einsum("eai,ebi->eab", g, g)
    Kd, tc, tm = 0.0, 0.0, 0.0
    for N_, u, a, p, gy, L_, tM, tC, tB, ub in _points(P, geo, y[ien], ac[ien][..., :3], divq, mu):
        ug, Lg, bg = torch.einsum("ei,eai->ea", u, g), torch.einsum("ei,eai->ea", L_, g), torch.einsum("ei,eai->ea", ub, g)
        Kd = Kd + P.almi * rho * N_[:, None] * N_[None, :] + lf * (
            rho * N_[None, :, None] * bg[:, None, :] + mu * gab + rho * tM[:, None, None] * ug[:, :, None] * ug[:, None, :]
            + tB[:, None, None] * Lg[:, :, None] * Lg[:, None, :])
        tc, tm = tc + tC, tm + tM
    SN, eye = _interior_rule().sum(0), torch.eye(3, dtype=torch.float64, device=DEV)
    K = torch.zeros((nnz, 9), dtype=torch.float64, device=DEV)
    Pm = torch.zeros((nnz, 4), dtype=torch.float64, device=DEV)
    for i in range(4):
        for j in range(4):
            si, sj = g[:, i], g[:, j]
            blk = (W * Kd[:, i, j])[:, None, None] * eye + (lf * W)[:, None, None] * (
                tc[:, None, None] * sj[:, :, None] * si[:, None, :] + 4.0 * mu * si[:, :, None] * sj[:, None, :])
            K.index_add_(0, slot[:, i, j], blk.reshape(-1, 9))
            G = (lf * W * SN[i])[:, None] * sj
            C = lf * W / rho * tm * gab[:, i, j]
            Pm.index_add_(0, slot[:, i, j], torch.cat([G, C[:, None]], 1))
    # rows and columns of prescribed velocities stay: the solver scales them out
    return K, Pm


def _scalar(m, P, y, s, sdot, diffus):
    """res (n) and lhsS (nnz) of the advection-diffusion equation (SUPG), without boundary data on the lattice."""
    n = m.nshg
    ien = torch.tensor(m.ien.astype(np.int64), device=DEV)
    geo = _Geometry(torch.tensor(m.x, device=DEV), ien)
    W, g, lf = geo.W, geo.g, P.alfi * P.gami * P.Delt
    ul, sl, dl = y[ien][..., :3], s[ien], sdot[ien]
    gS = torch.einsum("eai,ea->ei", g, sl)
    w = W[:, None] * _interior_rule().sum(0)
    q = _scatter(ien, w[..., None] * (diffus * gS)[:, None], n) / _scatter(ien, w, n)[:, None]
    divS = torch.einsum("eai,eai->e", g, q[ien])
    gab = torch.einsum("eai,ebi->eab", g, g)
    gg = (geo.G * geo.G).sum((1, 2))
    rl, xS = 0.0, 0.0
    for N_ in _interior_rule():
        u, sd = torch.einsum("a,eai->ei", N_, ul), dl @ N_
        conv = (u * gS).sum(1)
        tau = 1.0 / torch.sqrt((2.0 / P.Delt * P.dtsfct) ** 2 + torch.einsum("ei,eij,ej->e", u, geo.G, u) + 9.0 * diffus ** 2 * gg)
        ug = torch.einsum("ei,eai->ea", u, g)
        r = N_[None, :] * (sd + conv)[:, None] + diffus * torch.einsum("eai,ei->ea", g, gS) + (tau * (sd + conv - divS))[:, None] * ug
        rl = rl - W[:, None] * r
        # the SUPG mass term carries no time-integration factor in this formulation
        xS = xS + W[:, None, None] * (P.almi * N_[:, None] * N_[None, :] + lf * N_[None, :, None] * ug[:, None, :]
                                      + tau[:, None, None] * ug[:, :, None] * N_[None, None, :]
                                      + lf * (diffus * gab + tau[:, None, None] * ug[:, :, None] * ug[:, None, :]))
    nnz, slot = _slots(ien, n)
    S = torch.zeros(nnz, dtype=torch.float64, device=DEV).index_add(0, slot.reshape(-1), xS.reshape(-1))
    return _scatter(ien, rl, n), S


def exact(case, seed):
    """64-bit values of the assemblies, the derivative and the product.  The solves and time steps stop at a
    tolerance of 1e-5 of an iterative method, so no independent value has their digits: None."""
    kind = case["kind"]
    if kind in ("step", "newton", "adjoint"):
        return None
    m, P, yh, ah, c1, c2 = _inputs(case, seed)
    y, ac = torch.tensor(yh, device=DEV), torch.tensor(ah, device=DEV)
    n = m.nshg
    mu = torch.tensor(P.mu, dtype=torch.float64, device=DEV)
    if kind in ("asm", "res"):
        out = {"res": _residual(m, P, y, ac, mu, c1, c2)}
        if kind == "asm":
            out["lhsK"], out["lhsP"] = _tangent(m, P, y, ac, mu)
        return out
    if kind == "vjp":
        lam = _randn(seed, n, 4)
        c1t, c2t = (torch.tensor(c, device=DEV, requires_grad=True) for c in (c1, c2))
        for t in (y, ac, mu):
            t.requires_grad_(True)
        res = _residual(m, P, y, ac, mu, c1t, c2t)
        gy, ga, gm, g1, g2 = torch.autograd.grad((res * lam).sum(), [y, ac, mu, c1t, c2t])
        return {"res": res.detach(), "ybar": gy, "abar": ga, "mubar": float(gm), "c1bar": g1, "c2bar": g2}
    if kind == "sclr":
        if case["geo"] != "lattice":
            return None
        res, S = _scalar(m, P, y, _randn(seed, n), _randn(seed + 1, n), 0.1)
        return {"res": res, "lhsS": S}
    dt = torch.float64 if case["precision"] == "fp64" else torch.float32
    ien = torch.tensor(m.ien.astype(np.int64), device=DEV)
    key = torch.unique((ien[:, :, None] * n + ien[:, None, :]).reshape(-1))
    val, u = _randn(seed, key.numel(), 16, dtype=dt), _randn(seed + 1, n, 4, dtype=dt)
    ku = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    for c in torch.arange(key.numel(), device=DEV).split(4_000_000):
        prod = torch.einsum("kij,kj->ki", val[c].double().view(-1, 4, 4), u[key[c] % n].double())
        ku.index_add_(0, torch.div(key[c], n, rounding_mode="floor"), prod)
    return {"ku": ku}
