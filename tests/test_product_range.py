"""The integer product of ddmath.cuh is the product for every pair of factors
that its range test admits, at the ends of that range too (the host
compiles the header as plain C++): a vector of magnitude 2^512 and more
squares to infinity, not to a small number."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_products_at_the_ends_of_the_range(tmp_path):
    exe = tmp_path / "product_range_check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "a2c_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "product_range_check.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0
    n, different = map(int, r.stdout.split())
    assert n > 1500 and different == 0
