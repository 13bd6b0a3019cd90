"""crimson_elmgmr_vjp at the edges of its kernels: fewer tets than a block's
element groups, remainders of a warp of nodes, with and without the viscous
flux projection, every boundary flag (bits 0, 1, 2, 4) and no coupled outlet,
against central differences of the production residual.

Bound: 1e-6 of the derivative (truncation, as the other difference tests) plus
the rounding of the quotient, eps sum|lambda res| / h with a factor 10."""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver
from tests.test_gpu_adjoint import _res, _vjp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncross,naxial,outlets,idiff", [(2, 1, 0, 1), (2, 1, 1, 0), (3, 2, 1, 1), (4, 5, 2, 0),
                                                         (7, 11, 3, 1)])
def test_vjp_edges(ncross, naxial, outlets, idiff):
    import torch

    m = mesh.cylinder(ncross=ncross, naxial=naxial, n_outlets=max(1, outlets))
    rng = np.random.default_rng(ncross * 100 + naxial)
    # natural pressure, normal velocity, traction and bit 4 flags on random faces, with their values
    m.iBCB[:, 0] |= rng.choice([0, 1, 2, 3, 4, 6, 7, 16, 18], size=len(m.iBCB)).astype(np.int32)
    m.BCB[:] = rng.standard_normal(m.BCB.shape)
    P = FlowParams(rcr=[RCR(srfid=s) for s in m.outlets] if outlets else [], idiff=idiff)
    nc = len(P.rcr)
    c1, c2 = list(rng.uniform(80.0, 120.0, nc)), list(rng.uniform(-3.0, 3.0, nc))
    t = lambda s: torch.tensor(s * rng.standard_normal((m.nshg, 4)), device="cuda")
    y, ac, lam = t(10.0), t(5.0), t(1.0)
    with solver.ElmGMR(m, P) as elm:
        _, yb, ab, _, _, _ = _vjp(elm, y, ac, c1, c2, lam)
        scale = float((lam * _res(elm, y, ac, c1, c2)).abs().sum())
        for _ in range(2):
            dy, da, h = t(10.0), t(5.0), 1e-6
            da[:, 3] = 0.0
            fd = float((lam * (_res(elm, y + h * dy, ac + h * da, c1, c2)
                               - _res(elm, y - h * dy, ac - h * da, c1, c2))).sum()) / (2 * h)
            an = float((yb * dy).sum() + (ab * da).sum())
            assert abs(fd - an) <= 1e-6 * abs(an) + 10 * 2.2e-16 * scale / h, (fd, an)
