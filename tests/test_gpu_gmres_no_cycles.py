"""A memLS solve that allows GMRES no cycle (ngmres = 0): GMRES then returns
X = 0, so the momentum column of NSSOLVER's least-squares system is zero and
the solve reports it as singular, also on an lhs whose work space still holds
the vectors of an earlier solve."""
import ctypes

import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from crimsonflowsolver_b200 import _native as N
from oracle import pyoracle as po
from tests.linsys import first_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_gmres_cycle_is_singular(precision):
    m = mesh.cylinder(ncross=4, naxial=3)
    m.set_inflow(10.0)
    P = FlowParams(rcr=[RCR(srfid=3)], precision=precision)
    colm, rowp = po.genadj(m.ien, m.nshg)
    _, Res4, Val4, faceRes, _, _ = first_system(m, P, colm, rowp)
    ms = solver.MemLS(P, 2, nshg=m.nshg, colm=colm, rowp=rowp)
    none = solver.MemLS(FlowParams(rcr=P.rcr, precision=precision, ngmres=0), 2, nshg=m.nshg, colm=colm, rowp=rowp)
    try:
        nodes, sv = solver.dirichlet_face(m)
        ms.bc_create(1, nodes, 3, 0, sv)
        nn, vv = solver.neumann_face(m, 3)
        ms.bc_create(2, nn, 3, 1, vv)
        sol, _ = ms.solve(Res4, Val4.copy(), faceRes)
        Ri, Val, inc, st = np.ascontiguousarray(Res4), Val4.copy(), np.ones(2, dtype=np.int32), N.LsStats()
        rc = N.lib().crimson_memls_solve(ms.lhs, none.ls, 4, N.dp(Ri.copy()), N.dp(Val), N.ip(inc),
                                         N.dp(np.asarray(faceRes, dtype=np.float64)), ctypes.byref(st))
        assert N.ERRORS.get(rc) == "SINGULAR", rc
        again, _ = ms.solve(Res4, Val4.copy(), faceRes)
        assert np.array_equal(sol, again)
    finally:
        none.close()
        ms.close()
