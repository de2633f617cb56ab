"""The autotuner's decisions, without a GPU: timings and the plan are stand-ins."""
from types import SimpleNamespace

import pytest

from singleventriclesegmentation_b200 import autotune


def params(**kw):
    p = dict(boundary=1, length_type=0, length_z=1.0, length_y=1.0, length_x=1.0, max_outer_iterations=300)
    p.update(kw)
    return SimpleNamespace(**p)


class Plan:
    """Variant requests as a plan takes them: any request takes a level off the chip."""

    def __init__(self, dims, resident=True, **kw):
        self.dims, self.device, self.params = dims, None, params(**kw)
        self.can_stay, self.level, self.pairs = resident, {}, {}

    def set_level_tile(self, level, tile):
        self.level[level] = tile

    def set_pair_tile(self, level, pair, tile):
        self.pairs[level, pair] = tile

    def requests(self, level):
        return self.level.get(level, 0), tuple(self.pairs.get((level, i), 0) for i in range(len(self.dims)))

    def level_resident(self, level):
        tile, pairs = self.requests(level)
        return len(self.dims) if self.can_stay and not tile and not any(pairs) else 0


@pytest.fixture(autouse=True)
def _gpu_name(monkeypatch):
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda device: "some GPU")


def test_cache_key_holds_what_the_choice_depends_on():
    dims = [(80, 80, 80)]
    keys = {autotune._key(None, "f32", dims, params(**kw))
            for kw in ({}, dict(boundary=0), dict(max_outer_iterations=10), dict(length_type=1),
                       dict(length_type=1, length_x=2.0))}
    assert len(keys) == 5
    # lengths say nothing where the spacing is one
    assert autotune._key(None, "f32", dims, params()) == autotune._key(None, "f32", dims, params(length_x=7.0))


class Times:
    """Stand-ins for the two timing functions: a level's ms per iteration by its requests, shortly after the
    start (few iterations) and for good."""

    def __init__(self, monkeypatch, short, settled):
        self.short, self.settled, self.long_calls = short, settled, 0
        monkeypatch.setattr(autotune, "time_variant", self.variant)
        monkeypatch.setattr(autotune, "time_level", self.at)

    def variant(self, plan, level, tile, iters=6):
        plan.set_level_tile(level, tile)
        return self.at(plan, level, iters)

    def at(self, plan, level, iters=6):
        long = iters * self.short[(0, 0)] >= autotune.SETTLE_MS
        self.long_calls += long
        tile, pairs = plan.requests(level)
        return (self.settled if long else self.short).get((tile, max(pairs)))


def tune(plan, levels=1, **kw):
    return autotune.tune(plan, "f32", levels, candidates=[0, 3, 7], use_cache=False, **kw)


def test_close_timings_are_settled_by_a_long_one(monkeypatch):
    short = {(0, 0): 1.0, (3, 0): 0.95, (7, 0): 0.97}
    t = Times(monkeypatch, short, {(0, 0): 1.0, (3, 0): 1.1, (7, 0): 1.1})
    assert tune(Plan([(80, 80, 80)] * 2)) == [0] and t.long_calls == 2
    t = Times(monkeypatch, short, {(0, 0): 1.0, (3, 0): 0.96, (7, 0): 1.1})
    assert tune(Plan([(80, 80, 80)] * 2)) == [3]


def test_no_margin_where_nothing_stays_on_chip(monkeypatch):
    t = Times(monkeypatch, {(0, 0): 1.0, (3, 0): 0.95, (7, 0): 0.97}, {})
    assert tune(Plan([(80, 80, 80)] * 2, resident=False)) == [3] and t.long_calls == 0


def test_clear_timings_need_no_long_one(monkeypatch):
    t = Times(monkeypatch, {(0, 0): 1.0, (3, 0): 0.9, (7, 0): 1.2}, {})
    assert tune(Plan([(80, 80, 80)] * 2)) == [3] and t.long_calls == 0
    t = Times(monkeypatch, {(0, 0): 1.0, (3, 0): 1.05, (7, 0): 1.2}, {})
    assert tune(Plan([(80, 80, 80)] * 2)) == [0] and t.long_calls == 0


def test_a_class_takes_a_level_off_the_chip_only_for_good(monkeypatch):
    dims = [(40, 40, 40), (40, 40, 48)]
    short = {(0, 0): 1.0, (3, 0): 1.2, (7, 0): 1.3, (0, 3): 0.95, (0, 7): 0.97}
    for settled, left in (({(0, 0): 1.0, (0, 3): 0.99}, False), ({(0, 0): 1.0, (0, 3): 0.9}, True)):
        Times(monkeypatch, short, settled)
        plan = Plan(dims)
        assert tune(plan, per_class=True) == [0]
        assert bool(plan.class_tiles[0]) == left
        assert (plan.level_resident(0) == 0) == left
