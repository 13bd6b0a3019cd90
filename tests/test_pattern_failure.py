"""CPU: an allocation that fails while the pattern is built leaves it marked as
not built.  Under a preloaded CUDA runtime without a GPU (fake_cudart.c), each
allocation of crimson_genadj is made to fail in turn: the call returns an
error, and the next assembly on the same context builds the whole pattern (its
edge pass gets its list of slots) and succeeds."""
import ctypes
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = "/usr/local/cuda/include"


@pytest.mark.skipif(shutil.which("gcc") is None or not os.path.isdir(CUDA_INC), reason="gcc or the CUDA headers missing")
def test_failed_allocation_leaves_pattern_unbuilt(tmp_path):
    so = tmp_path / "libfake_cudart.so"
    cc = subprocess.run(["gcc", "-std=gnu99", "-Wall", "-shared", "-fPIC", "-I", CUDA_INC,
                         os.path.join(HERE, "fake_cudart.c"), "-o", str(so)], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    run = subprocess.run([sys.executable, os.path.abspath(__file__), str(so)], capture_output=True, text=True,
                         timeout=120, env=dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT))
    assert run.returncode == 0, run.stdout + run.stderr


def _child(fake_path):
    import numpy as np

    from crimsonflowsolver_b200 import _native as N
    from crimsonflowsolver_b200 import mesh

    fake, L = ctypes.CDLL(fake_path), N.lib()
    m = mesh.cylinder(ncross=2, naxial=1)
    i, j = np.repeat(m.ien, 4, axis=1), np.tile(m.ien, (1, 4))
    nnz = len(np.unique(np.stack([i.ravel(), j.ravel()]), axis=1).T)
    ien = np.asfortranarray(m.ien + 1, dtype=np.int32)
    x = np.asfortranarray(m.x)
    p = N.Params(rho=1.06, mu=0.04, Dtgl=1e3, Delt=1e-3, dtsfct=1.0, taucfct=1.0, almi=1.0, alfi=1.0, gami=1.0, idiff=1,
                 iconvflow=2, ndofBC=7)
    vec = [np.zeros((m.nshg, 4)) for _ in range(3)]
    K, P = np.zeros((nnz, 9)), np.zeros((nnz, 4))

    def context():
        h = ctypes.c_void_p()
        fake.fake_reset(-1, nnz, 0)
        N.check(L.crimson_ctx_create(ctypes.byref(h), ctypes.byref(p), m.nshg, m.nshg, len(m.ien), N.ip(ien), N.dp(x)),
                "ctx")
        return h

    def genadj(h):
        total = ctypes.c_longlong()
        return L.crimson_genadj(h, None, None, 0, ctypes.byref(total)), total.value

    h = context()
    fake.fake_reset(-1, nnz, 0)
    assert genadj(h) == (0, nnz)
    allocations = fake.fake_mallocs()
    L.crimson_ctx_destroy(h)
    assert allocations >= 10
    for k in range(allocations):
        h = context()
        fake.fake_reset(k, nnz, 0)
        rc, _ = genadj(h)
        assert rc != 0, k
        fake.fake_reset(-1, nnz, 0)
        rc = L.crimson_elmgmr_device(h, vec[0].ctypes.data, vec[1].ctypes.data, None, None, vec[2].ctypes.data,
                                     K.ctypes.data, P.ctypes.data, 1)
        assert fake.fake_null_edge_lists() == 0, k
        assert (rc, fake.fake_edge_passes()) == (0, 1), (k, rc)
        assert genadj(h) == (0, nnz), k
        L.crimson_ctx_destroy(h)


if __name__ == "__main__":
    _child(sys.argv[1])
