"""The autotuner's choice among timed candidates, over a stand-in for the solver and the clock (no GPU)."""
import types

import pytest

from glmmhdturb_b200 import autotune


class FakeSolver:
    """Its step takes what `cost` says for the tile it was made with."""
    made = []

    def __init__(self, n, *, tile=(0, 0, 0), **kw):
        self.n, self.tile, self.dx = n, tile, 1.0 / n[0]
        FakeSolver.made.append(tile)

    def alloc(self):
        return None

    def ic_turbulent(self, *a, **kw):
        pass

    def cfl(self, u):
        return 1.0, 1.0

    def step(self, *a, **kw):
        FakeSolver.now += FakeSolver.cost(self.tile)

    def kernel_info(self):
        return {"tile": tuple(self.tile) if self.tile[0] else (16, 16, self.n[2])}

    def close(self):
        pass


class FakeEvent:
    def __init__(self, enable_timing=False):
        self.t = 0.0

    def record(self):
        self.t = FakeSolver.now

    def elapsed_time(self, other):
        return other.t - self.t


@pytest.fixture
def tuner(monkeypatch):
    cuda = types.SimpleNamespace(Event=FakeEvent, synchronize=lambda: None)
    monkeypatch.setattr(autotune, "torch", types.SimpleNamespace(cuda=cuda))
    monkeypatch.setattr(autotune, "Solver", FakeSolver)
    FakeSolver.now, FakeSolver.made = 0.0, []
    return autotune.tune


def test_the_librarys_own_choice_is_a_candidate(tuner):
    """FP64: the automatic route is the fastest and no tile takes it."""
    FakeSolver.cost = staticmethod(lambda tile: 1.0 if tile[0] == 0 else 2.0)
    tile, ms, res = tuner(64, dtype="f64", save=False)
    assert tile == (0, 0, 0) and ms == 1.0 and len(res) > 1


def test_a_faster_tile_still_wins(tuner):
    FakeSolver.cost = staticmethod(lambda tile: 0.5 if tile[:2] == (16, 8) else 2.0)
    tile, ms, _ = tuner(64, dtype="f32", save=False)
    assert tile[:2] == (16, 8) and ms == 0.5


def test_a_grid_that_no_tile_divides_can_be_tuned(tuner):
    FakeSolver.cost = staticmethod(lambda tile: 1.0)
    tile, _, res = tuner((201, 135, 99), dtype="f32", save=False)
    assert tile == (0, 0, 0) and len(res) == 1


def test_tiles_of_the_caller_are_the_only_candidates(tuner):
    FakeSolver.cost = staticmethod(lambda tile: 1.0 if tile[0] == 0 else 2.0)
    tile, _, _ = tuner(64, dtype="f64", save=False, tiles=[(16, 16)], chunks=[0])
    assert tile[:2] == (16, 16)
