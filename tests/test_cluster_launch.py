"""Host check of the one-cluster launch's fallbacks (axia-fem_gb300/csrc/solver.cuh)
with faked CUDA calls: no GPU is needed."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_refused_cluster_leaves_no_error(tmp_path):
    nvcc = shutil.which("nvcc")
    if not nvcc:
        pytest.skip("no nvcc")
    exe = str(tmp_path / "cluster_check")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    os.path.join(HERE, "host", "cluster_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
