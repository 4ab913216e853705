"""The tiles a new handle starts with (csrc/prepared_mesh.h, compiled for the
host): within zsme_set_launch's limits for every component count, up to the
ones that leave the whole-stage kernel no room for 64 faces."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_default_tiles_are_accepted(tmp_path):
    exe = str(tmp_path / "check")
    cc = subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "zoomy-dmplex_b200", "csrc"), "-I",
                         os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "default_tiles_check.cpp"),
                         "-o", exe], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
    rows = [tuple(map(int, w)) for w in (line.split() for line in r.stdout.splitlines()) if w[0].isdigit()]
    got = {(nq, faces): v for nq, faces, *v in rows}
    # one wave of small tiles with two threads per cell; one wave of large ones; 256 faces beyond it
    for nq in (3, 4, 6, 8, 12):
        assert got[nq, 1600] == [96, 1, 2]
        assert got[nq, 77000] == [{3: 224, 4: 224, 6: 320, 8: 320, 12: 256}[nq], 1, 1]
        assert got[nq, 3000000] == [256, 1, 1]
    assert got[54, 1600][:2] == [64, 0] and got[54, 3000000][:2] == [158, 0]
