"""The evaluation's schedule, on the host: every centre rule, table and
absorption choice gives the value of the plain contraction (eval_tree_check.cu)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not Path(NVCC).exists(), reason="needs nvcc")
def test_schedule_equals_contraction(tmp_path):
    exe = tmp_path / "check"
    subprocess.run([NVCC, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "-cudart", "shared",
                    f"-I{ROOT / 'include'}", f"-I{ROOT / 'itensornumericalanalysis.jl_gb300' / 'csrc'}",
                    str(ROOT / "tests" / "eval_tree_check.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
