"""Which values solver.set_launch passes for the keys that a call does not
name (a stand-in for the library keeps them; no GPU needed)."""
import pytest

from zoomy_dmplex_b200 import solver
from zoomy_dmplex_b200.solver import LAUNCH_DEFAULTS, LAUNCH_KEYS, get_launch, set_launch


class FakeLibrary:
    """A handle on the whole-stage kernel with two threads per cell."""

    def __init__(self):
        self.own = dict(LAUNCH_DEFAULTS, tile_faces=96, fuse_final=1, prep_lean=2, face_occ=4, finalize_occ=4)

    def zsme_set_launch(self, h, b):
        self.own = dict(zip(LAUNCH_KEYS, [int(x) for x in b]))
        return 0

    def zsme_get_launch(self, h, b):
        for i, k in enumerate(LAUNCH_KEYS):
            b[i] = self.own[k]
        return 0


@pytest.fixture
def library(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(solver.native, "load", lambda: lib)
    return lib


@pytest.mark.parametrize("cfg", [{"finalize": 64}, {"face": 64, "prep_occ": 4}, {}])
def test_a_call_that_names_no_kernel_keeps_the_handles_kernels(library, cfg):
    set_launch(None, cfg)
    own = get_launch(None)
    assert (own["tile_faces"], own["fuse_final"], own["prep_lean"]) == (96, 1, 2)
    for k in set(LAUNCH_KEYS) - {"tile_faces", "fuse_final", "prep_lean"}:
        assert own[k] == cfg.get(k, LAUNCH_DEFAULTS[k])


@pytest.mark.parametrize("cfg", [{"tile_faces": 0}, {"tile_faces": 128}, {"fuse_final": 1},
                                 {"tile_faces": 0, "fuse_final": 1, "prep_lean": 4}])
def test_a_call_that_names_a_kernel_takes_the_defaults_for_the_rest(library, cfg):
    set_launch(None, cfg)
    assert get_launch(None) == dict(LAUNCH_DEFAULTS, **cfg)


def test_threads_per_cell_alone(library):
    set_launch(None, {"prep_lean": 4})
    own = get_launch(None)
    assert (own["tile_faces"], own["fuse_final"], own["prep_lean"]) == (96, 1, 4)
