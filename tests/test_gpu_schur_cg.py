"""CGRAD on the explicitly formed Schur operator at the sizes where its kernel
changes form: one slice, a last slice with missing rows, a block with several
warps per slice, operators that stay in shared memory and operators that are
streamed, no, one and several coupled faces.

* Small meshes: a memLS solve to a tight tolerance against the sparse direct
  solution (the bound of the other direct-solve tests, 1e-7 normwise).
* Larger meshes: one time step against the same mesh with randomly renumbered
  nodes, whose column offsets exceed 16 bits, so that CGRAD multiplies by the
  two products there: states equal to 1e-8 normwise (both stop at the solver's
  1e-5 on slightly different iterates), the same outer iteration counts.
"""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from oracle import pyoracle as po
from tests.conftest import relerr
from tests.linsys import direct_solve, first_system
from tests.test_gpu_cg_layout import _renumber

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncross,naxial", [(2, 1), (2, 2), (3, 5), (5, 7), (8, 9)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_small_meshes_match_direct_solve(ncross, naxial, precision):
    m = mesh.cylinder(ncross=ncross, naxial=naxial)
    m.set_inflow(10.0)
    P = FlowParams(rcr=[RCR(srfid=3)], precision=precision, max_refine=8, refine_tol=1e-10, epstol_mom=1e-9,
                   epstol_cont=1e-9, epstol_ns=1e-6, explicit_schur=1)
    colm, rowp = po.genadj(m.ien, m.nshg)
    _, Res4, Val4, faceRes, _, _ = first_system(m, P, colm, rowp)
    xd, _, _ = direct_solve(m, colm, rowp, Res4, Val4, faceRes)
    ms = solver.MemLS(P, 2, nshg=m.nshg, colm=colm, rowp=rowp)
    try:
        nodes, sv = solver.dirichlet_face(m)
        ms.bc_create(1, nodes, 3, 0, sv)
        nn, vv = solver.neumann_face(m, 3)
        ms.bc_create(2, nn, 3, 1, vv)
        sol, _ = ms.solve(Res4, Val4.copy(), faceRes)
        again, _ = ms.solve(Res4, Val4.copy(), faceRes)
        assert ms.schur_info()[0] == 1
    finally:
        ms.close()
    assert np.array_equal(sol, again)
    # FP64 stops at the outer tolerance, the mixed solve at its FP64 defect
    assert relerr(sol, xd) < (1e-4 if precision == "fp64" else 1e-7), relerr(sol, xd)


@pytest.mark.parametrize("ncross,naxial,n_outlets,precision", [
    (32, 47, 0, "fp64"),     # resident, no coupled face
    (32, 47, 3, "mixed"),    # resident, several faces
    (41, 57, 1, "fp64"),     # streamed
    (41, 57, 4, "fp64"),
    (55, 61, 1, "mixed"),
])
def test_forms_agree_with_two_products(ncross, naxial, n_outlets, precision):
    m = mesh.cylinder(ncross=ncross, naxial=naxial, n_outlets=max(1, n_outlets))
    assert m.nshg > 32768
    mr, perm = _renumber(m)
    out = []
    for mm in (m, mr):
        P = FlowParams(rcr=[RCR(srfid=s) for s in mm.outlets] if n_outlets else [], precision=precision, nitr=1,
                       explicit_schur=1)
        F = solver.FlowSolver(mm, P, inflow=lambda t: 10.0)
        try:
            st = F.step()
            out.append((F.state()[0], st.ri_itr[0], F.memls.schur_info()[0]))
        finally:
            F.close()
    (y0, r0, s0), (y1, r1, s1) = out
    assert (s0, s1) == (1, -1)
    assert r0 == r1
    assert relerr(y1[perm], y0) < 1e-8, relerr(y1[perm], y0)
