"""Assembly at the edges of its kernels: fewer tets than a warp's element
groups, edge and node counts with a remainder of a warp, edges whose lower node
is the later one in its tets, against the CPU oracle.  Tolerance as in
test_gpu_parity: rounding of sums in another order, 1e-12 normwise."""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from oracle import pyoracle as po
from tests.conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncross,naxial,idiff", [(2, 1, 1), (2, 2, 0), (3, 2, 1), (4, 5, 1), (7, 11, 0)])
def test_elm_edges(ncross, naxial, idiff):
    m = mesh.cylinder(ncross=ncross, naxial=naxial)
    rng = np.random.default_rng(10 * ncross + naxial)
    even = np.array([[0, 1, 2, 3], [1, 0, 3, 2], [2, 3, 0, 1], [3, 2, 1, 0], [1, 2, 0, 3], [0, 3, 1, 2]])
    m.ien[:] = np.take_along_axis(m.ien, even[rng.integers(0, len(even), size=len(m.ien))], axis=1)
    P = FlowParams(rcr=[RCR(srfid=3)], idiff=idiff)
    y, ac = 10.0 * rng.standard_normal((m.nshg, 4)), rng.standard_normal((m.nshg, 4))
    with solver.ElmGMR(m, P) as elm:
        colm, rowp = elm.genadj()
        g, r = elm(y, ac, [110.0], [-2.0]), elm(y, ac, [110.0], [-2.0], lhs=False)
    o = po.Elm(m, P, colm, rowp)(y, ac, srflist=[3], coef1=[110.0], coef2=[-2.0])
    for k in ("res", "lhsK", "lhsP"):
        assert relerr(g[k], o[k]) < 1e-12, (k, relerr(g[k], o[k]))
    assert relerr(r["res"], o["res"]) < 1e-12
