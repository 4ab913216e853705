"""Which kernel bench.py takes the kind "flux" for: what the profiled run
launched decides, not the launch configuration alone."""
import pytest

import bench


@pytest.mark.parametrize("tile_faces,fuse_final,prep,form", [
    (0, 1, 4, "face"), (0, 0, 4, "face"), (256, 0, 4, "tile"), (256, 1, 0, "stage"),
    (256, 1, 2, "tile"),     # "mood" at order 1, or a tile that does not fit
])
def test_flux_form(tile_faces, fuse_final, prep, form):
    launch = {"tile_faces": tile_faces, "fuse_final": fuse_final}
    assert bench.flux_form(launch, {"prep": (0.0, prep), "flux": (1.0, 4)}) == form
