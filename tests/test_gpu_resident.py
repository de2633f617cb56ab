"""The on-chip iterations (resident_kernel): all iterations of a warp in one launch, boxes of a
volume in registers and shared memory, faces exchanged between CTAs. Results must be bitwise those
of a split-role per-iteration variant, u and p, for every storage mode, at the edges of boxes and
volumes, alone, packed with other pairs and beside pairs too large for the chip."""
import pytest
import torch

from singleventriclesegmentation_b200 import synthetic
from singleventriclesegmentation_b200.tvl13d import TVL13DOpticalFlow

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(600)]

SPLIT = 9  # 32x8 voxel pairs, prefetch distance 3


def make_solver(storage, scales, warps, iters, boundary="MIRROR", length_type="numDofs", length=(1, 1, 1)):
    return TVL13DOpticalFlow(scales, warps, iters, 1.0, 0.025, 2, (0.5, 0.5, 0.25, 1.0), True, (5.0, 0.5), True, 1.0,
                             "CUBIC_HERMITESPLINE", boundary, length_type, length, torch.device("cuda"), storage=storage)


def both(storage, shapes, scales, warps, iters, **kw):
    pairs = [synthetic.frame_pair(s, seed=70 + i % 3) for i, s in enumerate(shapes)]
    I0, I1 = ([torch.from_numpy(p[k]).cuda() for p in pairs] for k in (0, 1))
    res, plans = [], []
    for tile in (0, SPLIT):
        solver = make_solver(storage, scales, warps, iters, **kw)
        solver.tile_id = tile
        u, p = solver.compute_batch(I0, I1, want_p=True)
        plan = solver.plan_for(shapes)
        torch.cuda.synchronize()
        plan.check()
        res.append(u + p)
        plans.append((solver, plan))
    for a, b in zip(*res):
        assert torch.equal(a, b)
    assert all(plans[1][1].level_resident(level) == 0 for level in range(scales))
    return plans[0]


@pytest.mark.parametrize("storage", ["f32", "f16-flow32", "bf16-flow32", "f16", "bf16"])
@pytest.mark.parametrize("shape,iters", [
    ((4, 4, 4), 2),      # the smallest volume the interior stencils serve, one box
    ((4, 9, 5), 7),      # odd sizes, an odd number of iterations (the other ping-pong copy)
    ((17, 33, 31), 6),   # remainders on every axis
    ((40, 24, 41), 9),   # one voxel beside the last pair
    ((64, 65, 66), 4),   # more pairs per thread (16-bit fields)
])
def test_one_volume(cuda, storage, shape, iters):
    _, plan = both(storage, [shape], 1, 2, iters)
    assert plan.level_resident(0) == 1


@pytest.mark.parametrize("storage", ["f32", "f16-flow32"])
def test_pyramid_and_packed_launches(cuda, storage):
    """Pairs of several sizes share launches, more pairs than one launch holds."""
    shapes = [(24, 20, 28), (33, 18, 21), (12, 40, 16)] * 9
    _, plan = both(storage, shapes, 2, 2, 11)
    assert plan.level_resident(1) == len(shapes)


def test_beside_a_volume_too_large(cuda):
    """A level with one pair that does not fit: the others on chip, that one per iteration."""
    _, plan = both("f16-flow32", [(32, 30, 28), (104, 104, 100), (24, 24, 24)], 2, 1, 5)
    assert plan.level_resident(0) in (0, 2) and plan.level_resident(1) >= 2


def test_other_stencils_stay_per_iteration(cuda):
    for kw in (dict(boundary="NEAREST"), dict(length_type="fixed", length=(9.0, 8.0, 7.0))):
        _, plan = both("f32", [(16, 17, 18)], 1, 1, 6, **kw)
        assert plan.level_resident(0) == 0
    _, plan = both("f32", [(3, 8, 8)], 1, 1, 6)   # the adjoint of 3 nodes is not the interior one
    assert plan.level_resident(0) == 0


def test_repeated_solves_and_stopped_pairs(cuda):
    """The exchange words are clean for the next launch; a stopped pair leaves a launch to the others."""
    shapes = [(24, 24, 24), (20, 28, 32)]
    pairs = [synthetic.frame_pair(s, seed=5 + i) for i, s in enumerate(shapes)]
    I0, I1 = ([torch.from_numpy(p[k]).cuda() for p in pairs] for k in (0, 1))
    tol = 0.0
    for stopping in (False, True):
        out = []
        for tile in (0, SPLIT):
            solver = make_solver("f16-flow32", 2, 4, 20)
            solver.tile_id = tile
            plan = solver.plan_for(shapes)
            plan.set_residuals(True, tol)
            us = [torch.empty(s + (3,), device="cuda") for s in shapes]
            for _ in range(3):
                plan.solve(I0, I1, us)
            plan.check()
            out.append((us, plan.residuals(), plan.level_resident(0)))
        assert out[0][2] == 2 and out[1][2] == 0
        assert (out[0][1] == out[1][1]).all()
        for a, b in zip(out[0][0], out[1][0]):
            assert torch.equal(a, b)
        assert (out[0][1] < 0).any() == stopping
        # between the first pair's second and third change at the coarse level: it stops early there
        tol = float(out[0][1][0, 1, 1] + out[0][1][0, 1, 2]) / 2


def test_two_streams(cuda):
    """Solves of two plans queued on two streams take turns and give the results of one after the other."""
    shape = (48, 40, 44)
    pairs = [synthetic.frame_pair(shape, seed=s) for s in (1, 2)]
    I = [[torch.from_numpy(p[k]).cuda() for k in (0, 1)] for p in pairs]
    solvers = [make_solver("f16-flow32", 3, 3, 50) for _ in range(2)]
    want = [s.compute(*i)[0].clone() for s, i in zip(solvers, I)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    got = [[], []]
    for _ in range(3):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                got[k].append(solvers[k].compute(*I[k])[0])
    torch.cuda.synchronize()
    for k in range(2):
        solvers[k].plan_for([shape]).check()
        for u in got[k]:
            assert torch.equal(u, want[k])


@pytest.mark.parametrize("storage", ["f32", "f16-flow32", "bf16"])
@pytest.mark.parametrize("shapes,iters", [
    ([(4, 4, 4)], 3),                                 # one box
    ([(9, 11, 12)], 7),                               # fewer boxes than a power of two
    ([(20, 20, 20)], 6),
    ([(5, 23, 19)], 5),                               # odd sizes
    ([(10, 11, 9 + i % 4) for i in range(23)], 5),    # more clusters than one launch or the GPU holds
])
def test_volumes_in_one_cluster(cuda, storage, shapes, iters):
    _, plan = both(storage, shapes, 1, 2, iters)
    assert plan.level_resident(0) == len(shapes)
