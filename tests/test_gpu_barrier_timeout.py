"""A barrier wait that runs out: every later call of the block's loop reports
it too, none of them waits again, and the context stays usable."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_one_wait_runs_out_once(tmp_path):
    exe = tmp_path / "gridred_timeout"
    cc = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                         "-DCRIMSON_GR_WAIT_CLOCKS=20000000LL", "-I",
                         os.path.join(ROOT, "crimsonflowsolver_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                         os.path.join(HERE, "gridred_timeout.cu"), "-o", str(exe)], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
    reported, calls, clocks, limit = map(int, run.stdout.split())
    assert reported == calls
    assert limit <= clocks < 2 * limit, (clocks, limit)
