"""The quick exponentials, logarithms and powers of the device have the
series' bits wherever their rounding test settles them, also compiled with
FMA contraction, as the mixed form's translation unit is."""
import subprocess
from pathlib import Path

import pytest

from a2c_gb300 import build as B

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def test_bits_under_contraction(gpu, tmp_path):
    exe = tmp_path / "contraction_check"
    r = subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-I",
                        str(ROOT / "a2c_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "contraction_check.cu"), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), "300000"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.returncode
    n, settled, different = map(int, r.stdout.split())
    assert n == 5 * 300_000 and settled > 0.9 * n
    assert different == 0
