"""Host logic of the learned planner's choices: no two candidates plan the same
passes, and the autotuner measures every plan once (a stand-in for the device
records what it is asked to measure)."""
import numpy as np
import pytest

from aleph_b200 import learned, workloads
from aleph_b200.circuit import flatten


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_candidates_plan_different_passes(precision):
    f = flatten(workloads.brickwall(24, 12, seed=3).instructions)
    cs = learned.candidates(precision)
    assert len({learned.plan_key(24, f, c, precision) for c in cs}) == len(cs)
    assert set(learned.large_choices(precision)) <= set(cs)
    assert {4, 5} <= {c.tile_r for c in learned.large_choices(precision)}


def test_autotune_measures_each_plan_once(monkeypatch):
    P = learned.PlanChoice

    class Backend:
        precision = "f64"

        def set_tuning(self, key, value):
            return self

    class Planner:  # the same plan under three names first
        def score(self, n, flat, precision):
            names = [P(tile_r=4), P(tile_r=4, tile_occupancy=3), P(tile_r=4, tile_occupancy=4), learned.GREEDY,
                     P(tile_r=3, tile_occupancy=3), P(tile_r=3)]
            return [learned.Scored(c, float(k), 1) for k, c in enumerate(names)]

    asked = []

    def measure(backend, n, flat, choice, repeats=2):
        asked.append(choice)
        return 1.0 / len(asked), None, np.zeros(1)

    monkeypatch.setattr(learned, "measure", measure)
    res = learned.autotune(Backend(), 24, workloads.brickwall(24, 12, seed=3).instructions, Planner(), top_k=2)
    assert asked == [learned.GREEDY, P(tile_r=4), P(tile_r=3, tile_occupancy=3)]
    assert res.choice == asked[-1] and set(res.measured) == set(asked)
