"""crimson_elmgmr_vjp into 8-byte aligned outputs (a view that starts at an odd
double of its buffer): the same cotangents as into aligned buffers.  acbar bit
for bit; ybar to 1e-13 normwise, because the boundary faces' terms are added
with atomics, in any order."""
import ctypes

import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from crimsonflowsolver_b200 import _native as N
from tests.conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncross,naxial,idiff", [(2, 1, 0), (3, 2, 1), (7, 11, 1)])
def test_vjp_outputs_need_8_byte_alignment(ncross, naxial, idiff):
    import torch

    m = mesh.cylinder(ncross=ncross, naxial=naxial)
    P = FlowParams(rcr=[RCR(srfid=3)], idiff=idiff)
    rng = np.random.default_rng(ncross)
    y, ac, lam = (torch.tensor(s * rng.standard_normal((m.nshg, 4)), device="cuda") for s in (10.0, 5.0, 1.0))
    c1, c2 = np.array([110.0]), np.array([-2.0])
    out = []
    with solver.ElmGMR(m, P) as elm:
        for off in (0, 1):
            # doubles off .. off + 4 n of a buffer with a guard value on either side
            buf = [torch.full((4 * m.nshg + 2,), 7.0, dtype=torch.float64, device="cuda") for _ in range(2)]
            yb, ab = (b[off:off + 4 * m.nshg] for b in buf)
            assert yb.data_ptr() % 16 == 8 * off
            mub, c1b, c2b = ctypes.c_double(), np.zeros(1), np.zeros(1)
            torch.cuda.synchronize()
            N.check(N.lib().crimson_elmgmr_vjp(elm.h, y.data_ptr(), ac.data_ptr(), N.dp(c1), N.dp(c2), lam.data_ptr(),
                                               None, yb.data_ptr(), ab.data_ptr(), ctypes.byref(mub), N.dp(c1b),
                                               N.dp(c2b)), "vjp")
            torch.cuda.synchronize()
            for b in buf:
                g = b.cpu().numpy()
                assert np.all(g[:off] == 7.0) and np.all(g[off + 4 * m.nshg:] == 7.0)
            out.append((yb.cpu().numpy(), ab.cpu().numpy(), mub.value, c1b[0], c2b[0]))
    (y0, a0, *s0), (y1, a1, *s1) = out
    assert np.array_equal(a0, a1) and s0 == s1
    assert relerr(y1, y0) < 1e-13, relerr(y1, y0)
