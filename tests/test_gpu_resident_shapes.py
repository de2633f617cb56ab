"""Every compiled shape of the on-chip iterations, asserted through level_resident_shape, bitwise against
a split-role per-iteration variant: the shape of five voxel pairs per thread with remainders on every
axis, and levels that mix on-chip pairs with pairs too large for the chip."""
import pytest

from test_gpu_resident import both, pytestmark  # noqa: F401  (gpu, timeout)


@pytest.mark.parametrize("storage", ["f32", "f16-flow32", "bf16-flow32", "f16", "bf16"])
@pytest.mark.parametrize("shape,iters", [
    ((66, 71, 79), 4),   # odd in x and y; z no multiple of five
    ((70, 67, 75), 5),   # an odd number of iterations (the other ping-pong copy)
    ((71, 79, 66), 2),   # even in x, one plane beside the last group of five
    ((63, 77, 81), 9),   # one voxel beside the last pair
])
def test_five_pairs_per_thread(cuda, storage, shape, iters):
    _, plan = both(storage, [shape], 1, 2, iters)
    assert plan.level_resident(0) == 1 and plan.level_resident_shape(0) == 3


@pytest.mark.parametrize("shape,which", [((24, 24, 24), 1), ((64, 65, 66), 2), ((9, 11, 12), 4)])
def test_other_shapes(cuda, shape, which):
    _, plan = both("f16-flow32", [shape], 1, 1, 5)
    assert plan.level_resident_shape(0) == which


@pytest.mark.parametrize("storage,shapes,which", [
    ("f32", [(48, 48, 48), (48, 48, 48), (104, 104, 100)], 2),
    ("f16-flow32", [(48, 48, 48), (104, 104, 100), (48, 48, 48)], 2),
    ("f32", [(72, 70, 68), (104, 104, 100), (66, 71, 72)], 3),
])
@pytest.mark.parametrize("iters", [5, 20])
def test_beside_a_volume_too_large(cuda, storage, shapes, which, iters):
    _, plan = both(storage, shapes, 1, 2, iters)
    assert plan.level_resident(0) == 2 and plan.level_resident_shape(0) == which
