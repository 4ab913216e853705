"""zsme_set_launch without memory for the new tiles' tables: the call returns an
error, and the handle goes on with the separate kernels (never on tables that
are not there), takes the configuration once there is memory and steps as a
fresh handle does."""
import numpy as np
import pytest
import torch

from zoomy_dmplex_b200 import cases, native
from zoomy_dmplex_b200.solver import Solver, get_launch, set_launch

from test_gpu_parity import params

pytestmark = pytest.mark.gpu

SMALL_TILES = {"tile_faces": 64, "fuse_final": 1, "prep_lean": 1}   # more rim cells: larger tables than a new handle's


def _fill_device_memory():
    """Blocks that leave less than 2 MB (the allocation granularity) free."""
    blocks, size = [], torch.cuda.mem_get_info()[0]
    while size >= 1 << 21:
        try:
            blocks.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size //= 2
    return blocks


def test_a_failed_set_launch_leaves_a_handle_that_steps():
    c = cases.plain_l0(400)    # tables of 46 MB, 57 with the small tiles
    torch.zeros(1, device="cuda")
    p = params(c.model, c.params)
    ref = Solver(c.model, c.mesh, c.settings, p)
    ref.set_state(c.q0)
    ref.step(3)
    want = ref.get_state()
    ref.close()
    g = Solver(c.model, c.mesh, c.settings, p)
    g.set_state(c.q0)
    own = get_launch(g.h)
    blocks = _fill_device_memory()
    try:
        with pytest.raises(native.ZsmeError):
            set_launch(g.h, SMALL_TILES)
    finally:
        del blocks
        torch.cuda.empty_cache()
    assert get_launch(g.h)["tile_faces"] == 0
    g.step(3)
    assert np.array_equal(g.get_state(), want)
    for cfg in (own, SMALL_TILES):
        set_launch(g.h, cfg)
        assert get_launch(g.h)["tile_faces"] == cfg["tile_faces"]
        g.set_state(c.q0)
        g.step(3)
        assert np.array_equal(g.get_state(), want)
    g.close()
