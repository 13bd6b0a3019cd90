"""A coupled face created again on an lhs that has solved with it, with fewer,
then with more nodes: the solve uses the new nodes, bit for bit as a fresh lhs
does."""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from oracle import pyoracle as po
from tests.linsys import first_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_f32_tangent"])
def test_recreated_face_takes_its_new_nodes(precision):
    m = mesh.cylinder(ncross=8, naxial=6)
    m.set_inflow(10.0)
    P = FlowParams(rcr=[RCR(srfid=3)], precision=precision, nprjs=3)
    colm, rowp = po.genadj(m.ien, m.nshg)
    _, Res4, Val4, faceRes, _, _ = first_system(m, P, colm, rowp)
    nodes, sv = solver.dirichlet_face(m)
    nn, vv = solver.neumann_face(m, 3)

    def lhs():
        ms = solver.MemLS(P, 2, nshg=m.nshg, colm=colm, rowp=rowp)
        ms.bc_create(1, nodes, 3, 0, sv)
        return ms

    kept = lhs()
    try:
        for part in (slice(0, len(nn) // 2), slice(len(nn) // 3, len(nn) // 3 + 5), slice(0, len(nn))):
            sols = []
            fresh = lhs()
            try:
                for ms in (kept, fresh):
                    ms.bc_create(2, nn[part], 3, 1, vv[part])
                    sols.append(ms.solve(Res4, Val4.copy(), faceRes)[0])
            finally:
                fresh.close()
            assert np.array_equal(*sols), part
    finally:
        kept.close()
