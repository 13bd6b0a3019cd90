"""CGRAD with two products (two_products=True) and on the explicit operator:
the kernel that each choice runs, at the sizes where it changes form, and the
same solutions.

* Small meshes, a memLS solve with CG to 1e-9: the same outer iterations,
  solutions equal to 1e-9 normwise (about a hundred CG iterations times the
  operator's condition, 1e4, times the rounding of a product, 1e-16, with a
  factor 10).  On the smallest the oracle's memLS reports a singular
  least-squares system (its first directions already solve it), and so do the
  two products.
* Larger meshes, one nonlinear iteration: states equal to 1e-8 normwise (both
  stop at the solver's 1e-5 on slightly different iterates), the same outer
  iteration counts.  At 324k nodes the FP64 operator's kernel keeps no vector
  in shared memory and marks the operator's lines to leave the L2 first.
* Own-ring offsets within 16 bits and 2-ring offsets beyond: the explicit
  operator does not apply and the default solve is the two-product one, bit
  for bit.
"""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from oracle import pyoracle as po
from tests.conftest import relerr
from tests.linsys import first_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncross,naxial", [(2, 1), (3, 5), (5, 7), (8, 9)])
def test_small_meshes_agree(ncross, naxial):
    m = mesh.cylinder(ncross=ncross, naxial=naxial)
    m.set_inflow(10.0)
    par = dict(rcr=[RCR(srfid=3)], epstol_mom=1e-9, epstol_cont=1e-9, epstol_ns=1e-6)
    colm, rowp = po.genadj(m.ien, m.nshg)
    F, Res4, Val4, faceRes, _, _ = first_system(m, FlowParams(**par), colm, rowp)
    try:
        F.memls.solve(Res4, Val4.copy(), faceRes)
        singular = False
    except RuntimeError:
        singular = True
    nodes, sv = solver.dirichlet_face(m)
    nn, vv = solver.neumann_face(m, 3)
    out = []
    for two in (False, True):
        ms = solver.MemLS(FlowParams(two_products=two, explicit_schur=1, **par), 2, nshg=m.nshg, colm=colm, rowp=rowp)
        try:
            assert ms.cg_form() == ("none", "none")
            ms.bc_create(1, nodes, 3, 0, sv)
            ms.bc_create(2, nn, 3, 1, vv)
            if two and singular:
                with pytest.raises(RuntimeError, match="SINGULAR"):
                    ms.solve(Res4, Val4.copy(), faceRes)
                return
            sol, st = ms.solve(Res4, Val4.copy(), faceRes)
            out.append((sol, st.RI.itr, ms.cg_form()))
        finally:
            ms.close()
    (s0, r0, f0), (s1, r1, f1) = out
    assert (f0, f1) == (("schur_resident", "none"), ("products_resident", "none"))
    assert r0 == r1
    assert relerr(s1, s0) < 1e-9, relerr(s1, s0)


def _step(m, n_outlets, **par):
    P = FlowParams(rcr=[RCR(srfid=s) for s in m.outlets] if n_outlets else [], nitr=1, **par)
    F = solver.FlowSolver(m, P, inflow=lambda t: 10.0)
    try:
        st = F.step()
        return F.state()[0], st.ri_itr[0], F.memls.cg_form()[0 if P.precision == "fp64" else 1]
    finally:
        F.close()


@pytest.mark.parametrize("ncross,naxial,n_outlets,precision,form", [
    (12, 13, 0, "fp64", "schur_resident"),
    (24, 40, 3, "fp64", "schur_resident"),
    (24, 40, 4, "mixed", "schur_resident"),
    (41, 57, 0, "fp64", "schur"),
    (41, 57, 1, "fp64", "schur"),
    (41, 57, 4, "fp64", "schur"),
    (55, 61, 2, "mixed", "schur"),
    (66, 90, 1, "fp64", "schur"),
    (66, 90, 3, "mixed", "schur"),
])
def test_forms_agree_on_one_numbering(ncross, naxial, n_outlets, precision, form):
    m = mesh.cylinder(ncross=ncross, naxial=naxial, n_outlets=max(1, n_outlets))
    (y0, r0, f0), (y1, r1, f1) = (_step(m, n_outlets, precision=precision, two_products=t) for t in (False, True))
    assert (f0, f1) == (form, "products_resident")
    assert r0 == r1
    assert relerr(y1, y0) < 1e-8, relerr(y1, y0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_wide_second_ring_takes_two_products(precision):
    m = mesh.cylinder(ncross=150, naxial=2)
    (y0, r0, f0), (y1, r1, f1) = (_step(m, 1, precision=precision, two_products=t) for t in (False, True))
    assert f0 == f1 == "products_resident"
    assert r0 == r1 and np.array_equal(y0, y1)


def test_f32_tangent_choices():
    m = mesh.cylinder(ncross=8, naxial=9)
    forms = [_step(m, 1, precision="mixed_f32_tangent", **kw)[2]
             for kw in ({}, {"explicit_schur": 1}, {"explicit_schur": 1, "two_products": True})]
    assert forms == ["products_resident", "schur_resident", "products_resident"]
