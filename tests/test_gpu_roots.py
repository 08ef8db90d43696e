"""The FP64 roots of the factorisations against CUDA's (roots_check.cu)."""
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_roots(tmp_path):
    exe = tmp_path / "roots"
    subprocess.run([NVCC, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3",
                    f"-I{ROOT / 'itensornumericalanalysis.jl_gb300' / 'csrc'}", str(ROOT / "tests" / "roots_check.cu"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
