"""The IMEX stages' Newton iteration on and off its register path, against the
oracle: dry and near-dry cells (identity block, no source) with slip friction
bit for bit; Manning friction, which couples the directions (6 x 6 in registers
at level 2, the full matrix at level 4), to the bar cbrt allows."""
import dataclasses

import numpy as np
import pytest

import oracle_py as O
from zoomy_dmplex_b200 import cases
from zoomy_dmplex_b200.solver import Solver

from test_gpu_parity import TOL, errs, params

pytestmark = pytest.mark.gpu


def _pair(c, p):
    st = dataclasses.replace(c.settings, time_integration="imex", cfl=0.3)
    g = Solver(c.model, c.mesh, st, params(c.model, p))
    o = O.Oracle(c.model, c.mesh.as_abi_arrays(), st.to_struct(), params(c.model, p))
    q = c.q0.copy()
    q[::7, 1] *= 1e-4       # depths on both sides of 1e-6 and 1e-4
    q[::7, 2:] *= 1e-4
    for s in (g, o):
        s.set_state(q)
    return g, o


@pytest.mark.parametrize("level", [0, 1, 2, 4])
@pytest.mark.parametrize("manning", [0.0, 0.03])
def test_imex_newton_paths(level, manning):
    O.set_threads(0)
    c = cases.wet_dry_patchwork(14, level=level)
    g, o = _pair(c, dict(g=9.81, nu=1e-3, n_manning=manning, **{"lambda": 0.1}))
    for k in range(4):
        _, dt = o.time()
        o.step(1)
        g.step(1, dts=[dt])
        a, b = g.get_state(), o.get_state()
        if manning:
            assert errs(a, b).max() <= TOL, k
            g.set_state(b, o.time()[0])
            o.set_state(b, o.time()[0])
        else:
            assert np.array_equal(a, b), k
