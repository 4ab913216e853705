"""The whole-stage kernel for component counts that no shipped plugin has (a
1-D level-2 plugin has 5, level 6 has 9): odd ones, whose sums one thread forms
component by component, and ones that the threads of a cell do not share
evenly.  It compiles (nvcc, no GPU needed) and, on a GPU, gives every component
the values it has in a four-component plugin, bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from zoomy_dmplex_b200 import mesh as M

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zoomy-dmplex_b200", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("nvcc"):
        pytest.fail("nvcc is needed")
    exe = str(tmp_path_factory.mktemp("stage") / "check")
    cc = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-fmad=false",
                         "--expt-relaxed-constexpr", "--split-compile", "0", "-I", CSRC, "-I",
                         os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "stage_components_check.cu"),
                         os.path.join(CSRC, "prepared_mesh.cpp"), "-o", exe], capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr[-4000:]
    return exe


def test_every_component_count_compiles(program):
    assert os.path.exists(program)


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", ["triangles", "quadrilaterals"])
def test_components_equal_the_four_component_plugin(program, tmp_path, mesh):
    m = M.jittered_square(12, seed=3) if mesh == "triangles" else M.mixed_square(12, seed=3)
    a = m.as_abi_arrays()
    path = str(tmp_path / "mesh.bin")
    with open(path, "wb") as f:
        f.write(np.array([a["dim"], a["n_cells"], a["n_faces"], a["max_faces"]], dtype=np.int32).tobytes())
        for k in ("cell_centroid", "cell_volume", "cell_faces", "face_cells", "face_centroid", "face_normal",
                  "face_bc"):
            f.write(a[k].tobytes())
    r = subprocess.run([program, path], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    # both gradients, three thread counts, 5 + 9 + 13 + 14 components
    assert r.stdout.split()[-4:] == ["checked", str(2 * 3 * 41), "wrong", "0"]
