"""The coarsest level's Cholesky factor and inverse, kernel by kernel, at sizes
around their 32-column blocks, 64-wide tiles and 128-column steps: A A^-1 = I
on well-conditioned matrices (condition below 4; the residual of an explicit
inverse through its Cholesky factor is of the order of n eps cond, 4 n eps is
asked for), exact symmetry, no pivot flagged."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
SIZES = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 160, 255, 257, 300, 449]


def test_factor_and_inverse(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "dense_harness"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "top_gpu_on_matlab_b200" / "csrc"), "-o", str(exe),
                    str(ROOT / "tests" / "dense_harness.cu")], check=True)
    out = subprocess.run([str(exe)] + [str(n) for n in SIZES], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = [line.split() for line in out.splitlines()]
    assert [int(r[0]) for r in rows] == SIZES
    for n, res, asym, status in rows:
        assert float(res) <= max(4, 4 * int(n)) * np.finfo(float).eps, (n, res)
        assert float(asym) == 0.0 and int(status) == 0, (n, asym, status)


@pytest.mark.parametrize("args,status", [(["sms=12"], 0), (["sms=5"], 0), (["neg=0"], 1), (["neg=200"], 1), (["neg=448"], 1)])
def test_panel_widths_and_pivots(tmp_path, args, status):
    """panels of 32 and 64 rows a CTA (n = 449: 321 rows below the first
    128 columns, 21 CTAs of 16 rows, 11 of 32) to the bound above, and a
    pivot that is not positive is flagged wherever it stands"""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "dense_harness"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "top_gpu_on_matlab_b200" / "csrc"), "-o", str(exe),
                    str(ROOT / "tests" / "dense_harness.cu")], check=True)
    out = subprocess.run([str(exe)] + args + ["449"], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert int(out[3]) == status
    if not status:
        assert float(out[1]) <= 4 * 449 * np.finfo(float).eps and float(out[2]) == 0.0
