"""The rule that turns a chosen tile into the one that runs (tile.h, plain
C++) on the host: it may be applied again, and to the three numbers a caller
reads back, without changing what runs.  And the tile tuner over made-up
times: its choice is never slower than the library's own."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("sms", [1, 132, 152])
def test_the_rule_gives_the_same_tile_again(tmp_path, sms):
    exe = tmp_path / "tile_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "a2c_gb300" / "csrc"),
                        "-I", str(ROOT / "include"),
                        str(ROOT / "tests" / "cpp" / "tile_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe), str(sms)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.returncode
    n, wide, twin, copies = map(int, r.stdout.split())
    assert n == 39 * 2 * 80 and wide > 0 and twin > 0 and copies > 0
