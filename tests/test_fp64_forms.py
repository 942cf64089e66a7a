"""The fast FP64 forms of the device code against the plain ones, bit for
bit, on the host (the headers compile as plain C++): the quick exp, log and
pow of ddmath.cuh wherever Ziv's rounding test settles them, fexp_mid, mul_int,
the quotients and the pair functions of eam64_pair.cuh -- over their whole
ranges and at the switch radii, a central-difference step to either side."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SRC = ROOT / "tests" / "cpp" / "fp64_forms_check.cpp"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("forms") / "fp64_forms_check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "a2c_gb300" / "csrc"),
                        str(SRC), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


# least share of the calls that the rounding test must settle (the rest
# take the series): all but 2^-10 in the mean, less for logarithms near 1
@pytest.mark.parametrize("form,count,share", [("exp", 300_000, 0.999), ("log", 300_000, 0.8),
                                              ("pow", 200_000, 0.999), ("fexp", 1_000_000, 1.0),
                                              ("mul", 2_000_000, 1.0),
                                              ("quotient", 1_000_000, 1.0), ("pair", 200_000, 1.0)])
def test_fast_form_has_the_plain_bits(check, form, count, share):
    r = subprocess.run([str(check), form, str(count), "11"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    n, settled, different = map(int, r.stdout.split())
    assert n >= 0.9 * count
    assert settled >= share * n
    assert different == 0
