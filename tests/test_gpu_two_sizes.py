"""Two solvers of different sizes in one process, stepped in turn, in the mode
whose CG kernel sizes its shared memory by the mesh: the larger one's columns
take more than 48 KB per block, the smaller one's fewer.  The larger one steps
after the smaller one as it does alone, bit for bit."""
import numpy as np
import pytest

from crimsonflowsolver_b200 import FlowParams, RCR, mesh, solver

pytestmark = pytest.mark.gpu


def test_larger_solver_steps_after_smaller_one():
    P = FlowParams(rcr=[RCR(srfid=3)], precision="mixed_f32_tangent", nitr=1, nprjs=1, max_refine=1, maxiters=3)
    big, small = mesh.cylinder(ncross=72, naxial=110), mesh.cylinder(ncross=4, naxial=3)
    make = lambda m: solver.FlowSolver(m, P, inflow=lambda t: 10.0)  # noqa: E731
    states = []
    for interleaved in (False, True):
        F = [make(big)] + ([make(small)] if interleaved else [])
        try:
            for _ in range(2):
                for f in F:
                    f.step()
            states.append(F[0].state()[0])
        finally:
            for f in F:
                f.close()
    assert np.array_equal(*states)
