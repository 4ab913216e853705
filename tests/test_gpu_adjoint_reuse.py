"""Several adjoint calls on one handle, whose captured segments outlive the
call: each gives a fresh handle's loss, gradients, dts and final state bit for
bit, whatever changed between the calls."""
import numpy as np
import pytest

from zoomy_dmplex_b200 import cases
from zoomy_dmplex_b200.solver import Solver, set_launch

from test_gpu_parity import params

pytestmark = pytest.mark.gpu


def _observations(c, nsteps, n, seed):
    rng = np.random.default_rng(seed)
    steps = np.sort(rng.integers(0, nsteps + 1, n)).astype(np.int32)
    cells = rng.integers(0, c.mesh.n_cells, n).astype(np.int32)
    return steps, cells, np.ones(n, dtype=np.int32), rng.uniform(0.5, 1.5, n)


def _call(g, c, q, p, nsteps, every, obs, profiled=False):
    g.set_params(p)
    g.set_state(q)
    g.set_profiling(profiled)
    r = g.adjoint(nsteps, *obs, checkpoint_every=every)
    g.set_profiling(False)
    return r + (g.get_state(), np.array(g.time()))


def test_calls_on_one_handle_equal_fresh_handles():
    c = cases.adjoint_l1(20)
    p = params(c.model, c.params)
    q2 = c.q0.copy()
    q2[:, 1] *= 1.05
    p2 = params(c.model, dict(c.params, n_manning=0.05))
    tiles = {"tile_faces": 128, "prep_lean": 2}
    # (state, parameters, steps, interval, observations, launch before the call, profiled)
    calls = [(c.q0, p, 12, 4, 40, None, False), (c.q0, p, 12, 4, 40, None, False),    # the same again
             (q2, p, 12, 4, 40, None, False), (q2, p2, 12, 4, 40, None, False),       # state, parameters
             (q2, p2, 12, 4, 90, None, False), (q2, p2, 12, 4, 7, None, False),       # more, fewer observations
             (q2, p2, 20, 4, 7, None, False), (c.q0, p2, 8, 4, 7, None, False),       # more, fewer steps
             (c.q0, p2, 13, 4, 7, None, False), (c.q0, p2, 12, 4, 7, None, False),    # overlapped, not, and back
             (c.q0, p, 12, 3, 7, None, False), (c.q0, p, 12, 4, 7, None, False),      # another interval and back
             (c.q0, p, 12, 4, 7, tiles, False), (q2, p, 12, 4, 7, None, False),       # another launch configuration
             (q2, p, 12, 4, 7, None, True), (q2, p, 12, 4, 7, None, False)]           # a profiled call
    g = Solver(c.model, c.mesh, c.settings, p)
    for k, (q, pp, nsteps, every, n, launch, profiled) in enumerate(calls):
        if launch is not None:
            set_launch(g.h, launch)
        obs = _observations(c, nsteps, n, seed=k // 2)
        got = _call(g, c, q, pp, nsteps, every, obs, profiled)
        h = Solver(c.model, c.mesh, c.settings, p)
        want = _call(h, c, q, pp, nsteps, every, obs)
        h.close()
        for i, (a, b) in enumerate(zip(got, want)):
            assert np.array_equal(a, b), (k, i)
        if k == 4:      # plain steps in between
            g.step(3)
    g.close()
