"""The end of a captured step where cells need the generic Newton path (level
4 with Manning friction couples the directions, so no cell is solved in
registers): the tail's blocks finish the deferred cells, the last one ends the
step, begins the next and clears its counters.  Equal to the separate kernels
bit for bit, over two calls of several steps, at both orders (order 1 finalizes
from the stage's output buffer) and in an ensemble."""
import dataclasses

import numpy as np
import pytest

from zoomy_dmplex_b200 import cases
from zoomy_dmplex_b200.solver import BatchSolver, Solver, set_launch

from test_gpu_parity import params

pytestmark = pytest.mark.gpu

MANNING = dict(g=9.81, nu=1e-3, n_manning=0.03, **{"lambda": 0.1})
STAGE, SEPARATE = {"tile_faces": 128, "fuse_final": 1}, {"tile_faces": 0}


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("side", [9, 40])
def test_deferred_cells_in_captured_steps(order, side):
    c = cases.roofline_l4(side)
    st = dataclasses.replace(c.settings, reconstruction_order=order)
    outs = []
    for cfg in (STAGE, SEPARATE):
        g = Solver(c.model, c.mesh, st, params(c.model, MANNING))
        set_launch(g.h, cfg)
        g.set_state(c.q0)
        counts = []
        for n in (3, 4, 1):
            g.step(n)
            counts.append(g.sync().n_newton_deferred)
        outs.append((g.get_state(), g.get_aux(), g.time(), counts))
        g.close()
    a, b = outs
    assert b[3][0] > 0 and a[3] == b[3]
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2] == b[2]


def test_deferred_cells_of_an_ensemble():
    members = [cases.roofline_l4(n, seed=n) for n in (8, 13, 10)]
    st = dataclasses.replace(members[0].settings, t_end=0.004)
    outs = []
    for cfg in (STAGE, SEPARATE):
        b = BatchSolver(members[0].model, [c.mesh for c in members], st,
                        [params(c.model, MANNING) for c in members])
        set_launch(b.h, cfg)
        for i, c in enumerate(members):
            b.set_state(i, c.q0)
        b.step(3)
        b.step(5)
        outs.append([(b.get_state(i), b.time(i)) for i in range(len(members))])
        b.close()
    for (qa, ta), (qb, tb) in zip(*outs):
        assert np.array_equal(qa, qb) and ta == tb
