"""The autotuner where the whole-stage kernel runs, on the host: a stand-in
solver reports no face-state launches with tiles and fuse_final, scores its
profiled steps with one cost and takes another, known time for captured ones.
The tuner leaves the knobs alone that do not act, never returns a configuration
whose captured steps are slower than those of the one the handle came with, and
does not use tunings cached under another version of the knobs."""
import json

import pytest

from zoomy_dmplex_b200 import autotune
from zoomy_dmplex_b200.solver import LAUNCH_DEFAULTS

START = dict(LAUNCH_DEFAULTS, tile_faces=96, fuse_final=1, prep_lean=2, face_occ=4, finalize_occ=4)


class FakeSolver:
    def __init__(self, profiled, captured, clock):
        self.h = self
        self.cfg = dict(START)
        self.profiled, self.captured, self.clock = profiled, captured, clock
        self.profiling, self.acc, self.steps = False, 0.0, 0

    def set_profiling(self, on):
        self.profiling, self.acc = on, 0.0

    def step(self, n):
        self.steps += n
        if self.profiling:
            self.acc += n * self.profiled(self.cfg)
        else:
            self.clock[0] += n * self.captured(self.cfg)

    def sync(self, check=True):
        pass

    def read_profile(self):
        stage = self.cfg["fuse_final"] and self.cfg["tile_faces"]
        return {"prep": (0.0, 0) if stage else (0.5 * self.acc, 2), "flux": (self.acc if stage else 0.5 * self.acc, 2)}


@pytest.fixture
def clock(monkeypatch):
    now = [0.0]
    monkeypatch.setattr(autotune, "set_launch", lambda h, cfg: setattr(h, "cfg", dict(cfg)))
    monkeypatch.setattr(autotune, "get_launch", lambda h: dict(h.cfg))
    monkeypatch.setattr(autotune.time, "perf_counter", lambda: now[0])
    return now


def cost(cfg):
    """Shortest with the whole-stage kernel on 160 faces, 4 threads per cell."""
    c = 1.0 + abs(cfg["tile_faces"] - 160) / 1000 + (0.1 if cfg["prep_lean"] != 4 else 0.0)
    return c + (0.0 if cfg["fuse_final"] else 1.0) + (0.05 if cfg["finalize_occ"] != 3 else 0.0)


def _tune(s, **kw):
    return autotune.tune(s, "sme2d_l2", 10000, **dict(dict(use_cache=False, write_cache=False), **kw))


def test_finds_the_stage_kernels_shape_and_leaves_the_rest(clock):
    s = FakeSolver(cost, cost, clock)
    cfg = _tune(s)
    assert (cfg["tile_faces"], cfg["fuse_final"], cfg["prep_lean"], cfg["finalize_occ"]) == (160, 1, 4, 3)
    assert all(cfg[k] == START[k] for k in autotune.NOT_STAGE)
    assert s.cfg == cfg
    # the inert knobs cost trials only where they act: without tiles
    tried = [k for k, _, _ in autotune.last_trace]
    assert "prep" not in tried and "gather" not in tried and "prep_lean/prep_occ" not in tried


@pytest.mark.parametrize("captured", [lambda c: 1.0 if c == START else 1.1, lambda c: 1.0])
def test_keeps_the_handles_own_configuration_unless_faster(clock, captured):
    s = FakeSolver(cost, captured, clock)
    assert _tune(s) == START and s.cfg == START


def test_separate_kernels_are_searched_where_they_win(clock):
    def separate(cfg):
        return (0.5 if cfg["tile_faces"] == 0 else 1.0) + (0.0 if cfg["prep_occ"] == 6 else 0.1)

    s = FakeSolver(separate, separate, clock)
    cfg = _tune(s)
    assert cfg["tile_faces"] == 0 and cfg["prep_occ"] == 6


def test_a_tuning_of_another_version_is_not_used(clock, tmp_path):
    cache = tmp_path / "tuned.json"
    old = autotune.cache_key("sme2d_l2", 10000).rsplit("|", 1)[0]
    cache.write_text(json.dumps({old: {"config": dict(LAUNCH_DEFAULTS), "trace": []}}))
    s = FakeSolver(cost, cost, clock)
    cfg = _tune(s, use_cache=True, write_cache=True, cache=str(cache))
    assert s.steps > 0 and cfg["tile_faces"] == 160
    steps = s.steps
    assert _tune(s, use_cache=True, cache=str(cache)) == cfg and s.steps == steps


def test_every_size_a_handle_may_start_with_is_tried():
    sizes = dict(autotune.KNOBS)["tile_faces"]
    assert set(range(96, 321, 32)) <= set(sizes)
