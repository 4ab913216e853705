"""The quotients by a known divisor (csrc/rn_div.h) equal the plain division
bit for bit wherever they do not report themselves odd, and so does the Newton
blocks' elimination built on them (csrc/gepp_regs.h).  The headers are compiled
for the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name,count,most_odd", [("rn_div_check", 4000000, 400000), ("gepp_rn_check", 500000, 300000)])
def test_quotients_equal_the_plain_division(tmp_path, name, count, most_odd):
    exe = str(tmp_path / name)
    cc = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                         os.path.join(ROOT, "zoomy-dmplex_b200", "csrc"),
                         os.path.join(ROOT, "tests", name + ".cpp"), "-o", exe], capture_output=True, text=True)
    if cc.returncode != 0:
        pytest.fail(cc.stderr)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    words = r.stdout.split()
    assert int(words[1]) == count and 0 < int(words[3]) < most_odd
