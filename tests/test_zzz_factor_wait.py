"""A wait of the coarsest factorisation that runs out has a status of its own,
apart from a pivot's, and is over after its second; further waits of the same
factorisation then give up early."""
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_column_wait_gives_up(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "wait_harness"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "top_gpu_on_matlab_b200" / "csrc"), "-o", str(exe),
                    str(ROOT / "tests" / "wait_harness.cu")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout
    (s1, t1), (s2, t2) = [line.split() for line in out.splitlines()]
    assert int(s1) == 2 and 1000 <= float(t1) < 3000, out
    assert int(s2) == 2 and float(t2) < 30000, out
