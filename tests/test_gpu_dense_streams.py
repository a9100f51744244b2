"""The coarsest level's factorisation with its trailing updates and the inverse
of the factor on streams of their own, as the solver calls it: A A^-1 = I to the
bound of the one-stream test (4 n eps, and n eps more for the product that checks
it), W equal to the same kernels' on one stream, and to itself over repeats, bit for
bit; sizes of one to several steps with W beside the factor and after it."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
SIZES = [100, 129, 257, 449, 700, 1386, 2304]


def test_streams(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "streams_harness"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "top_gpu_on_matlab_b200" / "csrc"), "-o", str(exe),
                    str(ROOT / "tests" / "streams_harness.cu")], check=True)
    out = subprocess.run([str(exe)] + [str(n) for n in SIZES], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = [line.split() for line in out.splitlines()]
    assert [(int(r[0]), int(r[1])) for r in rows] == [(n, b) for n in SIZES for b in (1, 0)]
    for n, beside, res, fromOne, repeats, status in rows:
        assert float(res) <= 5 * int(n) * np.finfo(float).eps, (n, beside, res)
        assert int(fromOne) == 0 and int(repeats) == 0 and int(status) == 0, (n, beside, fromOne, repeats, status)
