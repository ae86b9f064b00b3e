"""The tcgen05 GEMM compiles for sm_100a with each of its build options."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
NVCC = NVCC if os.path.exists(NVCC) else shutil.which("nvcc")


@pytest.mark.skipif(not NVCC, reason="needs nvcc")
@pytest.mark.parametrize("options", [["-DTNX_TMEM_ACC=4"], ["-DTNX_TMEM_ACC=4", "-DTNX_EPI_WARPS=4"]])
def test_gemm_tc_options_compile(tmp_path, options):
    r = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-cuda",
                        f"-I{os.path.join(ROOT, 'include')}", *options,
                        os.path.join(ROOT, "tenax_b200", "csrc", "gemm_tc.cu"), "-o", str(tmp_path / "out.ii")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
