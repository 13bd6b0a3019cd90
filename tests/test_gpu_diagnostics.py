"""Reports on an lhs only read it: they launch no kernel."""
import ctypes

import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from crimsonflowsolver_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,column", [("fp64", 0), ("mixed", 1), ("mixed_f32_tangent", 1)])
def test_reports_launch_nothing(precision, column):
    m = mesh.cylinder(ncross=8, naxial=10)
    L = N.lib()
    r, nb = (ctypes.c_int(), ctypes.c_int()), ctypes.c_longlong()
    F = solver.FlowSolver(m, FlowParams(rcr=[RCR(srfid=3)], precision=precision), inflow=lambda t: 10.0)
    try:
        layout = lambda: L.crimson_memls_cg_layout(F.memls.lhs, *map(ctypes.byref, r), ctypes.byref(nb))  # noqa: E731
        assert N.ERRORS[layout()] == "STATE"   # nothing solved yet
        F.step()
        before = L.crimson_launch_count()
        assert layout() == N.OK
        F.memls.schur_info()
        assert L.crimson_launch_count() == before
        assert r[column].value == 1 and r[1 - column].value == 0 and nb.value > 0
    finally:
        F.close()
