"""The register pass kernels' shared-memory index maps, on the host: for every
variant each point is loaded once from where TMA put it, the exchange between
the phases is consistent and stays within the warp that owns its slots, the
output lands where the TMA store reads it, and nothing has bank conflicts
(tests/reg_layout_check.cu, compiled with nvcc, run without a GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_reg_index_maps(tmp_path):
    if not (os.path.exists(NVCC) or shutil.which(NVCC)):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "reg_layout_check")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17",
                    "--expt-relaxed-constexpr", "-o", exe, os.path.join(HERE, "reg_layout_check.cu")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.count("\n") == r.stdout.count("ok ")
