"""Steps of a handle whose operator-split source is off (zsme_settings.source
= 0): every launch configuration gives the same state, time and aux bit for
bit, on captured steps and with imposed dts, and the oracle's state."""
import dataclasses

import numpy as np
import pytest

import oracle_py as O
from zoomy_dmplex_b200 import cases
from zoomy_dmplex_b200.settings import SolverSettings
from zoomy_dmplex_b200.solver import Solver, set_launch

from test_gpu_parity import TOL, errs, params

pytestmark = pytest.mark.gpu


class NoSource(SolverSettings):
    def to_struct(self):
        s = super().to_struct()
        s.source = 0
        return s


LAUNCHES = [{"tile_faces": 0, "fuse_final": 0}, {"tile_faces": 0, "fuse_final": 1},
            {"tile_faces": 0, "fuse_final": 1, "finalize_occ": 3}, {"tile_faces": 128, "fuse_final": 0},
            {"tile_faces": 128, "fuse_final": 1}, None]


@pytest.mark.parametrize("make", [lambda: cases.plain_l0(20), lambda: cases.level2(17), lambda: cases.mixed_level2(9)])
@pytest.mark.parametrize("order", [1, 2])
def test_steps_without_the_source(make, order):
    O.set_threads(0)
    c = make()
    st = NoSource(**dict(dataclasses.asdict(c.settings), reconstruction_order=order))
    p = params(c.model, c.params)
    o = O.Oracle(c.model, c.mesh.as_abi_arrays(), st.to_struct(), p)
    o.set_state(c.q0)
    dts = []
    for _ in range(6):
        dts.append(o.time()[1])
        o.step(1)
    outs = []
    for imposed in (False, True):
        for cfg in LAUNCHES:
            g = Solver(c.model, c.mesh, st, p)
            if cfg is not None:
                set_launch(g.h, cfg)
            g.set_state(c.q0)
            if imposed:
                g.step(6, dts=dts)
            else:
                g.step(2)
                g.step(4)
            outs.append((imposed, cfg, g.get_state(), g.get_aux(), g.time()))
            g.close()
    for imposed, cfg, q, a, t in outs:
        ref = outs[len(LAUNCHES) if imposed else 0]
        assert np.array_equal(q, ref[2]) and np.array_equal(a, ref[3]) and t == ref[4], (imposed, cfg)
        assert errs(q, o.get_state()).max() <= TOL, (imposed, cfg)
