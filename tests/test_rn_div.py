"""The quotients by a known divisor (csrc/rn_div.h) equal the plain division
bit for bit wherever they do not report themselves odd.  The header is
compiled for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_equal_the_plain_division(tmp_path):
    exe = str(tmp_path / "rn_div_check")
    cc = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                         os.path.join(ROOT, "zoomy-dmplex_b200", "csrc"),
                         os.path.join(ROOT, "tests", "rn_div_check.cpp"), "-o", exe], capture_output=True, text=True)
    if cc.returncode != 0:
        pytest.fail(cc.stderr)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    words = r.stdout.split()
    assert int(words[1]) == 4000000 and 0 < int(words[3]) < 400000
