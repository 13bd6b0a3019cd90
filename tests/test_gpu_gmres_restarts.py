"""Restarts of the persistent GMRES kernel in its larger forms (2, 4 and 8
values per thread in registers, the running vector in memory), with no, one and
several coupled faces: a Krylov dimension of 4, four cycles per call and a
tolerance that none of them reaches, so that every call restarts three times.

* FP64 against the CPU oracle's time stepper: the same counts of outer, GMRES
  and CG iterations, states equal to 1e-9 (the bound of the other form tests).
* Mixed against FP64: the same GMRES counts, states equal to 1e-4 (FP32
  rounding, 6e-8, of matrices and basis over 40 products, times the condition
  of the scaled momentum block, below 100 here, with a margin of 4).
"""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from oracle import pyoracle as po
from tests.conftest import relerr

pytestmark = pytest.mark.gpu


def _inflow(t):
    return 10.0


def _params(m, outlets, precision="fp64"):
    return FlowParams(rcr=[RCR(srfid=s) for s in m.outlets] if outlets else [], nitr=1, kspace=4, ngmres=4, nprjs=2,
                      epstol_mom=1e-12, epstol_cont=1e-2, precision=precision, max_refine=1)


def _step(m, P):
    F = solver.FlowSolver(m, P, inflow=_inflow)
    try:
        st = F.step()
        return F.state()[0], (st.ri_itr[0], st.gm_itr[0], st.cg_itr[0])
    finally:
        F.close()


@pytest.mark.parametrize("ncross,naxial,outlets", [(24, 40, 1), (32, 47, 4), (46, 57, 0), (58, 71, 2)])
def test_restarts_match_oracle(ncross, naxial, outlets):
    m = mesh.cylinder(ncross=ncross, naxial=naxial, n_outlets=max(1, outlets))
    P = _params(m, outlets)
    y, its = _step(m, P)
    O = po.OracleFlow(m, P, nthreads=8, inflow=_inflow)
    O.step()
    assert its == tuple(O.stats[0][:3])
    # two outer iterations, two calls each, four cycles of four and three restarts' residuals
    assert its[:2] == (2, 2 * 2 * (4 * 4 + 3))
    assert relerr(y, O.y) < 1e-9, relerr(y, O.y)


@pytest.mark.parametrize("ncross,naxial,outlets", [(24, 40, 3), (58, 71, 0)])
def test_mixed_restarts_match_fp64(ncross, naxial, outlets):
    m = mesh.cylinder(ncross=ncross, naxial=naxial, n_outlets=max(1, outlets))
    (y0, i0), (y1, i1) = (_step(m, _params(m, outlets, p)) for p in ("fp64", "mixed"))
    assert i0[:2] == i1[:2]
    assert np.isfinite(y1).all() and relerr(y1, y0) < 1e-4, relerr(y1, y0)
