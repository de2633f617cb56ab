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
