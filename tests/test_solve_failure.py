"""CPU: an allocation that fails in a memLS solve or in the block product's
preparation leaves the handle usable.  Under a preloaded CUDA runtime without a
GPU (fake_cudart.c), whose kernels do nothing and whose products are all one, so
that a solve ends with a singular least-squares system, each device, pinned or
event allocation is made to fail in turn: the call returns an error, and the next
one on the same handle ends as on a fresh one, with the same device memory and
the same CG kernel."""
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
@pytest.mark.parametrize("what", ["fp64", "mixed", "mixed_f32_tangent", "two_products", "spmv4"])
def test_failed_allocation_leaves_handle_usable(tmp_path, what):
    so = tmp_path / "libfake_cudart.so"
    cc = subprocess.run(["gcc", "-std=gnu99", "-Wall", "-shared", "-fPIC", "-I", CUDA_INC,
                         os.path.join(HERE, "fake_cudart.c"), "-o", str(so)], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    run = subprocess.run([sys.executable, os.path.abspath(__file__), str(so), what], capture_output=True, text=True,
                         timeout=120, env=dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT))
    assert run.returncode == 0, run.stdout + run.stderr


def _child(fake_path, what):
    import numpy as np

    from crimsonflowsolver_b200 import _native as N
    from crimsonflowsolver_b200 import mesh

    fake, L = ctypes.CDLL(fake_path), N.lib()
    fake.fake_live.restype = ctypes.c_size_t
    m = mesh.cylinder(ncross=3, naxial=2)
    n = m.nshg
    i, j = np.repeat(m.ien, 4, axis=1).ravel(), np.tile(m.ien, (1, 4)).ravel()
    rows, cols = np.unique(np.stack([i, j]), axis=1)
    colm = np.concatenate([[1], 1 + np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    rowp, nnz = (cols + 1).astype(np.int32), len(cols)
    gn = np.arange(1, n + 1, dtype=np.int32)

    class Solve:
        def __init__(self):
            self.ls, self.lhs = ctypes.c_void_p(), ctypes.c_void_p()
            N.check(L.crimson_memls_ls_create(ctypes.byref(self.ls), 3, 0, 0.0, 0.0, 0, 0, None, None, None), "ls")
            N.check(L.crimson_memls_ls_set_precision(self.ls, {"mixed": 1, "mixed_f32_tangent": 2}.get(what, 0), 2, 0.0),
                    "precision")
            N.check(L.crimson_memls_ls_set_two_products(self.ls, int(what == "two_products")), "two_products")
            N.check(L.crimson_memls_lhs_create(ctypes.byref(self.lhs), n, n, nnz, N.ip(gn), N.ip(colm), N.ip(rowp), 1),
                    "lhs")
            val = np.ones((4, 3))
            N.check(L.crimson_memls_bc_create(self.lhs, 1, 4, 3, 1, N.ip(gn[:4].copy()), N.dp(val)), "bc")

        def __call__(self):
            R, V = np.ones((n, 4)), np.ones((nnz, 16))
            st = N.LsStats()
            return L.crimson_memls_solve(self.lhs, self.ls, 4, N.dp(R), N.dp(V), N.ip(np.ones(1, dtype=np.int32)),
                                         N.dp(np.array([2.0])), ctypes.byref(st))

        def state(self):
            f64, f32 = ctypes.c_int(), ctypes.c_int()
            L.crimson_memls_cg_form(self.lhs, ctypes.byref(f64), ctypes.byref(f32))
            return f64.value, f32.value

        def close(self):
            L.crimson_memls_lhs_free(self.lhs)
            L.crimson_memls_ls_free(self.ls)

    class Spmv:
        def __init__(self):
            self.h = ctypes.c_void_p()
            p = N.Params(rho=1.06, mu=0.04, Dtgl=1e3, Delt=1e-3, dtsfct=1.0, taucfct=1.0, almi=1.0, alfi=1.0, gami=1.0,
                         idiff=1, iconvflow=2, ndofBC=7)
            ien, x = np.asfortranarray(m.ien + 1, dtype=np.int32), np.asfortranarray(m.x)
            N.check(L.crimson_ctx_create(ctypes.byref(self.h), ctypes.byref(p), n, n, len(m.ien), N.ip(ien), N.dp(x)), "ctx")
            fake.fake_rows(n, nnz // n)
            fake.fake_reset(-1, nnz, 0)
            total = ctypes.c_longlong()
            N.check(L.crimson_genadj(self.h, None, None, 0, ctypes.byref(total)), "genadj")

        def __call__(self):
            val, u = np.ones((nnz, 16)), np.ones((n, 4))
            rc = L.crimson_spmv4_prepare(self.h, 0, val.ctypes.data)
            if rc:   # nothing to multiply with
                assert N.ERRORS[L.crimson_spmv4_apply(self.h, u.ctypes.data, u.ctypes.data)] == "STATE"
                return rc
            return L.crimson_spmv4_apply(self.h, u.ctypes.data, u.ctypes.data)

        def state(self):
            return ()

        def close(self):
            L.crimson_ctx_destroy(self.h)

    make = Spmv if what == "spmv4" else Solve

    def fresh(fail_at):
        base = fake.fake_live()
        c = make()
        fake.fake_reset(fail_at, 0, 0)
        return c, c(), fake.fake_live() - base, base

    c, end, memory, _ = fresh(-1)
    expected = "OK" if what == "spmv4" else "SINGULAR"
    assert N.ERRORS.get(end, "OK") == expected, (N.ERRORS.get(end), L.crimson_last_error())
    allocations, state = fake.fake_mallocs(), c.state()
    c.close()
    assert allocations >= (3 if what == "spmv4" else 40)
    for k in range(allocations):
        c, rc, _, base = fresh(k)
        assert rc not in (0, end), (k, rc)
        fake.fake_reset(-1, 0, 0)
        rc = c()
        assert (rc, c.state(), fake.fake_live() - base) == (end, state, memory), k
        c.close()


if __name__ == "__main__":
    _child(*sys.argv[1:])
