"""The per-iteration kernels where the automatic choice would keep iterations on chip: with on-chip
iterations off (svs_tvl1_plan_set_resident) the automatic variant groups, the z chunks of tail columns
and the persistent loop are compared bitwise with the on-chip form and with one variant for all."""
import pytest
import torch

from singleventriclesegmentation_b200 import _lib, synthetic
from singleventriclesegmentation_b200.tvl13d import TVL13DOpticalFlow

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


def make_solver(storage, scales=3, warps=1, iters=10):
    return TVL13DOpticalFlow(scales, warps, iters, 1.0, 0.025, 2, (0.5, 0.5, 0.25, 1.0), True, (5.0, 0.5), True, 1.0,
                             "CUBIC_HERMITESPLINE", "MIRROR", "numDofs", (1, 1, 1), torch.device("cuda"), storage=storage)


def frames(shapes):
    pairs = [synthetic.frame_pair(s, seed=40 + i % 5) for i, s in enumerate(shapes)]
    return [[torch.from_numpy(p[k]).cuda() for p in pairs] for k in (0, 1)]


def solve(plan, I):
    outs = [torch.empty(d + (3,), device="cuda") for d in plan.dims]
    plan.solve(*I, outs)
    torch.cuda.synchronize()
    plan.check()
    return outs


def equal(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


def test_automatic_variant_groups(cuda):
    shapes = [(12, 64, 64)] * 20 + [(12, 80, 80)] * 16 + [(12, 72, 96)] * 4
    I = frames(shapes)
    main, own = _lib.auto_tiles(4, shapes, torch.cuda.get_device_properties(0).multi_processor_count)
    plan = make_solver("f16-flow32").plan_for(shapes)
    on_chip = solve(plan, I)
    nodes = plan.graph_kernels
    plan.set_resident(False)
    groups = solve(plan, I)
    assert [plan.level_resident(level) for level in range(3)] == [0, 0, 0]
    assert plan.pair_tiles(0) == [o or main for o in own] and len(set(plan.pair_tiles(0))) >= 2
    assert plan.graph_kernels > nodes  # a launch per iteration and group, not per warp and box list
    plan.set_tile(28)
    assert equal(solve(plan, I), groups) and equal(on_chip, groups)
    plan.set_tile(0)
    plan.set_resident(True)
    assert equal(solve(plan, I), groups) and plan.graph_kernels == nodes


def test_tail_columns_in_chunks(cuda):
    shape, n = (48, 48, 48), 34
    I = frames([shape] * n)
    plan = make_solver("f16-flow32", scales=1).plan_for([shape] * n)
    plan.set_resident(False)
    outs = solve(plan, I)
    info = _lib.tile_info(plan.level_tiles()[0])
    cols = n * -(-shape[1] // info["ty"]) * -(-shape[2] // info["tx"])
    assert plan.level_resident(0) == 0 and plan.level_ctas(0) > cols
    plan.set_level_chunks(0, 1)
    assert equal(solve(plan, I), outs) and plan.level_ctas(0) == cols
    plan.set_level_chunks(0, 0)
    plan.set_resident(True)
    assert equal(solve(plan, I), outs)


@pytest.mark.parametrize("storage", ["f32", "f16-flow32"])
def test_chunks_and_pair_variants(cuda, storage):
    shapes = [(24, 24, 24), (21, 37, 45), (20, 40, 40)]
    I = frames(shapes)
    plan = make_solver(storage, scales=2, warps=2, iters=20).plan_for(shapes)
    plan.set_resident(False)
    outs = solve(plan, I)
    assert plan.level_resident(0) == 0 and plan.level_resident(1) == 0
    for level, pair, tile in ((0, 1, 17), (0, 2, 12), (1, 0, 9)):
        plan.set_pair_tile(level, pair, tile)
    assert equal(solve(plan, I), outs)
    for level in range(2):
        plan.set_level_chunks(level, 3)
    assert equal(solve(plan, I), outs)


@pytest.mark.parametrize("storage,shapes", [("f32", [(32, 32, 32)] * 3), ("f16-flow32", [(40, 40, 40)] * 4)])
def test_persistent_loop(cuda, storage, shapes):
    I = frames(shapes)
    plan = make_solver(storage, warps=2, iters=30).plan_for(shapes)
    plan.set_resident(False)
    outs = solve(plan, I)
    assert not any(plan.level_persistent(3)) and plan.level_resident(0) == 0
    plan.set_persistent(True)
    assert equal(solve(plan, I), outs) and any(plan.level_persistent(3))


def test_reserved_plans_keep_the_choice(cuda):
    """retarget() keeps it, as it keeps the other options of a plan."""
    from singleventriclesegmentation_b200.tvl13d import SolverPlan
    solver = make_solver("f16-flow32")
    plan = SolverPlan.reserve(solver.params(), 2, 200 << 20, torch.device("cuda"))
    plan.set_resident(False)
    for shapes in ([(24, 24, 24), (20, 28, 32)], [(32, 32, 32)]):
        plan.retarget(shapes)
        I = frames(shapes)
        outs = solve(plan, I)
        assert plan.level_resident(0) == 0
        assert equal(outs, solver.compute_batch(*I))
    plan.close()
