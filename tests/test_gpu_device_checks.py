"""Device code checked by a small program of its own (compiled here with
nvcc): the state store for more components than any shipped plugin has, and
the quotients by a known divisor, whose device form starts from the hardware's
approximate reciprocal, against the device's own division."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name,counts", [("soa_aos_check", {"checked": 364 * 1129}),
                                         ("rn_div_device_check", {"checked": 1 << 26})])
def test_device_program(tmp_path, name, counts):
    if not shutil.which("nvcc"):
        pytest.fail("nvcc is needed")
    exe = str(tmp_path / name)
    cc = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-fmad=false",
                         "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "zoomy-dmplex_b200", "csrc"),
                         "-I", os.path.join(ROOT, "include"),
                         os.path.join(ROOT, "tests", name + ".cu"), "-o", exe], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    w = r.stdout.split()
    got = dict(zip(w[::2], map(int, w[1::2])))
    assert got["wrong"] == 0 and all(got[k] == v for k, v in counts.items()), r.stdout
