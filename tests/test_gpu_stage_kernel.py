"""The whole-stage kernel against the separate face-state, face and gather
kernels, bit for bit: tile sizes from one with many rims to one that holds the
whole mesh, every thread count per cell, both gradients, limiter on and off,
both orders, SSP stage counts that alternate its buffers, and states that send
cells off its main path (dry and clamped cells, exact ties of the limiter's
ratios, vanishing values, infinities and NaN)."""
import dataclasses

import numpy as np
import pytest

from zoomy_dmplex_b200 import cases, models
from zoomy_dmplex_b200 import mesh as M
from zoomy_dmplex_b200.solver import BatchSolver, Solver, get_launch, set_launch

pytestmark = pytest.mark.gpu


def _open_sides(c):
    """Every other boundary face without a condition."""
    bc = c.mesh.face_bc.copy()
    bc[np.nonzero(c.mesh.face_cells[:, 1] < 0)[0][::2]] = M.FACE_NO_CONDITION
    return dataclasses.replace(c, mesh=dataclasses.replace(c.mesh, face_bc=bc))


def _strip(c):
    m = M.interval(np.linspace(0.0, 1.0, 302))
    q = np.zeros((m.n_cells, 3))
    q[:, 1] = 1.0 + 0.1 * np.sin(9 * m.cell_centroid[:, 0])
    q[:, 2] = 0.2 * q[:, 1]
    return dataclasses.replace(c, model="sme1d_l0_malpasset", mesh=m, q0=q, params={})


CASES = {"l0": lambda: cases.plain_l0(20), "l1": lambda: cases.adjoint_l1(17), "l2": lambda: cases.level2(23),
         "l4": lambda: cases.roofline_l4(19), "mixed": lambda: cases.mixed_level2(15),
         "open": lambda: _open_sides(cases.level2(14)), "1d": lambda: _strip(cases.plain_l0(4))}


def _solver(c, cfg, **kw):
    st = dataclasses.replace(c.settings, **kw)
    names, vals = models.parameter_table(c.model)
    for k, v in c.params.items():
        vals[names.index(k)] = v
    g = Solver(c.model, c.mesh, st, np.array(vals))
    set_launch(g.h, cfg)
    g.set_state(c.q0)
    return g


def _states(c):
    """The case's state, perturbed, and with cells that leave the main path."""
    rng = np.random.default_rng(4)
    n, nq = c.q0.shape
    q = c.q0 + 1e-3 * rng.standard_normal(c.q0.shape)
    yield "noise", q
    t = q.copy()
    t[:, 1:] = np.round(t[:, 1:] * 4) / 4        # equal differences: ties of the ratios
    yield "ties", t
    t = q.copy()
    t[rng.uniform(size=n) < 0.3, 1:] = 0.0
    t[rng.uniform(size=n) < 0.2, 2:] *= 1e3      # clamped momenta, dry neighbours
    yield "dry", t
    t = q.copy()
    t[:, 2:] *= 10.0 ** rng.uniform(-320, 0, (n, nq - 2))
    yield "vanishing", t
    t = q.copy()
    t[rng.integers(n, size=3), rng.integers(2, nq, 3)] = [np.inf, -np.inf, np.nan]
    yield "nonfinite", t


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("gradient", ["green_gauss", "least_squares"])
@pytest.mark.parametrize("order,limiter", [(2, "tvd"), (2, "none"), (1, "tvd")])
def test_rhs_equals_the_separate_kernels(name, gradient, order, limiter):
    c = CASES[name]()
    kw = dict(gradient=gradient, reconstruction_order=order, limiter=limiter)
    ref = _solver(c, {"tile_faces": 0, "prep_lean": 0}, **kw)
    states = dict(_states(c))
    want = {k: ref.rhs(q) for k, q in states.items()}
    for tile in (64, 96, 160, 256, 512):
        for threads in (1, 2, 4):
            g = _solver(c, {"tile_faces": tile, "fuse_final": 1, "prep_lean": threads}, **kw)
            for k, q in states.items():
                assert np.array_equal(g.rhs(q), want[k], equal_nan=True), (k, tile, threads)
            g.close()


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("gradient", ["green_gauss", "least_squares"])
@pytest.mark.parametrize("positivity", ["zhang_shu", "mood"])
def test_positivity_rhs_equals_the_separate_kernels(name, gradient, positivity):
    c = CASES[name]()
    kw = dict(gradient=gradient, positivity=positivity)
    ref = _solver(c, {"tile_faces": 0}, **kw)
    states = dict(_states(c))
    want = {k: ref.rhs(q) for k, q in states.items()}
    for tile in (64, 160, 256):
        g = _solver(c, {"tile_faces": tile, "fuse_final": 1}, **kw)
        for k, q in states.items():
            assert np.array_equal(g.rhs(q), want[k], equal_nan=True), (k, tile)
        g.close()


@pytest.mark.parametrize("order,positivity", [(2, "zhang_shu"), (2, "mood"), (1, "zhang_shu"), (1, "mood")])
def test_positivity_steps_equal_the_separate_kernels(order, positivity):
    c = cases.wet_dry_patchwork(24)
    kw = dict(reconstruction_order=order, positivity=positivity)
    ref = _solver(c, {"tile_faces": 0}, **kw)
    g = _solver(c, {"tile_faces": 96, "fuse_final": 1}, **kw)
    for s in (ref, g):
        s.step(12)
    assert np.array_equal(g.get_state(), ref.get_state()) and g.time() == ref.time()
    assert g.sync().n_mood_cells == ref.sync().n_mood_cells


@pytest.mark.parametrize("name", ["l0", "l4", "mixed", "1d"])
@pytest.mark.parametrize("order,stages", [(1, 2), (2, 2), (2, 3), (2, 5)])
def test_steps_equal_the_separate_kernels(name, order, stages):
    c = CASES[name]()
    kw = dict(reconstruction_order=order, ssp_stages=stages)
    ref = _solver(c, {"tile_faces": 0}, **kw)
    g = _solver(c, {"tile_faces": 128, "fuse_final": 1, "prep_lean": 2}, **kw)
    for s in (ref, g):
        s.step(7)
        s.source(1e-3)      # the next step starts from a state that is not clamped
        s.step(4)
    assert np.array_equal(g.get_state(), ref.get_state()) and g.time() == ref.time()
    assert np.array_equal(g.get_aux(), ref.get_aux())


def test_a_tile_too_large_for_shared_memory_takes_the_separate_kernels():
    c = CASES["l4"]()
    g = _solver(c, {"tile_faces": 700, "fuse_final": 1})
    ref = _solver(c, {"tile_faces": 0})
    for s in (ref, g):
        s.step(5)
    assert np.array_equal(g.get_state(), ref.get_state())


def test_ensemble_of_uneven_members_and_end_times():
    """Members that stop at their own last step (the inactive ones keep their
    state) in tiles that span members."""
    members = cases.ensemble(5, seed=11, side_range=(5, 20), processes=1)
    st = dataclasses.replace(members[0].settings, t_end=0.02)
    outs = []
    for cfg in ({"tile_faces": 0}, {"tile_faces": 256, "fuse_final": 1}):
        b = BatchSolver(members[0].model, [c.mesh for c in members], st, [c.params for c in members])
        set_launch(b.h, cfg)
        for i, c in enumerate(members):
            b.set_state(i, c.q0)
        b.step(12)
        outs.append([(b.get_state(i), b.time(i)) for i in range(len(members))])
        b.close()
    for (qa, ta), (qb, tb) in zip(*outs):
        assert np.array_equal(qa, qb) and ta == tb


@pytest.mark.parametrize("side,one_wave", [(12, True), (60, True), (330, False)])
def test_default_launch(side, one_wave):
    c = cases.level2(side)
    g = Solver(c.model, c.mesh, c.settings)
    d = get_launch(g.h)
    assert d["fuse_final"] == 1 and d["tile_faces"] >= 96
    assert (d["tile_faces"] == 96 and d["prep_lean"] == 2) if one_wave else (d["tile_faces"] == 256 and
                                                                           d["prep_lean"] == 1)
    set_launch(g.h, d)      # what get_launch returns is accepted and stays
    assert get_launch(g.h) == d
