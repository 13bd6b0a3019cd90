"""CPU: bench.py counts the bytes of the CG kernel that ran, in every mode."""
import inspect
import os
import sys

import pytest

from crimsonflowsolver_b200 import _native as N

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize("mbytes", [4, 8])
def test_model_follows_the_kernel(mbytes):
    import bench

    nnz, nnz2, n, nface = 1000, 4000, 100, 2
    model = {f: bench.cg_iter_model(f, nnz, nnz2, n, nface, mbytes) for f in bench.CG_KERNELS}
    assert set(model) == set(N.CG_FORMS[1:])
    byt = {f: v[2] for f, v in model.items()}
    assert byt["schur"] == bench.cg_schur_iter_bytes(nnz2, n, nface, mbytes)
    assert byt["schur"] - byt["schur_resident"] == nnz2 * (mbytes + 2)
    assert byt["products"] == bench.cg_iter_bytes(nnz, n, mbytes, nface)
    assert byt["products_resident"] == bench.cg_iter_bytes(nnz, n, mbytes, nface, resident=True)
    for f, (kernel, _, _) in model.items():
        assert kernel.startswith("k_cg_schur" if f.startswith("schur") else "k_cg_persistent")
        assert {4: "<float>", 8: "<double>"}[mbytes] in kernel


def test_every_mode_uses_the_model():
    import bench

    for run in (bench.run_ours, bench.run_scale):
        src = inspect.getsource(run)
        assert "cg_iter_model(" in src and "cg_iter_bytes(" not in src and "cg_schur_iter_bytes(" not in src, run
