"""The forms of the persistent GMRES kernel (values per thread in registers: 1,
2, 4, 8, or the running vector in memory), with no, one and several coupled
faces (which share rim nodes), against independent paths.

* Restarts: a Krylov dimension of 4 forces several cycles per call; iteration
  counts and solution against the CPU oracle's memLS (1e-10, the bound of the
  other memLS parity tests).
* Forms: one nonlinear iteration with a Krylov dimension of 65, for which the
  solver takes the launch-per-step path, and with 50; neither restarts on these
  systems, so both do the same arithmetic up to the order of sums: the same
  iteration counts, solutions equal to 1e-9 (GMRES and CG stop at 1e-4, which
  multiplies a difference of 1e-15 per product by the number of products).
"""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from oracle import pyoracle as po
from tests.conftest import relerr
from tests.linsys import first_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncross,naxial", [(2, 1), (4, 3), (8, 10)])
def test_restarts_match_oracle(ncross, naxial):
    m = mesh.cylinder(ncross=ncross, naxial=naxial)
    m.set_inflow(10.0)
    P = FlowParams(rcr=[RCR(srfid=3)], kspace=4)
    colm, rowp = po.genadj(m.ien, m.nshg)
    F, Res4, Val4, faceRes, _, _ = first_system(m, P, colm, rowp)
    osol, ost = F.memls.solve(Res4, Val4.copy(), faceRes)
    ms = solver.MemLS(P, 2, nshg=m.nshg, colm=colm, rowp=rowp)
    try:
        nodes, sv = solver.dirichlet_face(m)
        ms.bc_create(1, nodes, 3, 0, sv)
        nn, vv = solver.neumann_face(m, 3)
        ms.bc_create(2, nn, 3, 1, vv)
        sol, st = ms.solve(Res4, Val4.copy(), faceRes)
    finally:
        ms.close()
    assert (st.RI.itr, st.GM.itr, st.CG.itr) == (ost.RI.itr, ost.GM.itr, ost.CG.itr)
    assert relerr(sol, osol) < 1e-10, relerr(sol, osol)


@pytest.mark.parametrize("ncross,naxial,outlets", [(12, 13, 3), (24, 40, 1), (32, 47, 4), (46, 57, 0), (58, 71, 2)])
def test_forms_match_launch_per_step(ncross, naxial, outlets):
    m = mesh.cylinder(ncross=ncross, naxial=naxial, n_outlets=max(1, outlets))
    out = []
    for kspace in (50, 65):
        P = FlowParams(rcr=[RCR(srfid=s) for s in m.outlets] if outlets else [], kspace=kspace, nitr=1)
        F = solver.FlowSolver(m, P, inflow=lambda t: 10.0)
        try:
            st = F.step()
            out.append((F.state()[0], (st.ri_itr[0], st.gm_itr[0], st.cg_itr[0])))
        finally:
            F.close()
    assert out[0][1] == out[1][1]
    assert relerr(out[0][0], out[1][0]) < 1e-9, relerr(out[0][0], out[1][0])
