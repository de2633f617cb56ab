"""Host time of a batch's set-up (re-targeting, the choice per level, capture): choosing which pairs stay
on chip must stay a small part of it, also for many pairs of different sizes."""
import random
import time

import pytest
import torch

from singleventriclesegmentation_b200.tvl13d import SolverPlan, TVL13DOpticalFlow

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


def test_choice_is_a_small_part_of_a_set_up(cuda):
    """120 uneven pairs: set-up with on-chip iterations takes at most five times that without (three times
    were measured; a choice that divides for every box and pair took eleven)."""
    solver = TVL13DOpticalFlow(3, 1, 2, 1.0, 0.025, 2, (0.5, 0.5, 0.25, 1.0), True, (5.0, 0.5), True, 1.0,
                               "CUBIC_HERMITESPLINE", "MIRROR", "numDofs", (1, 1, 1), torch.device("cuda"),
                               storage="f16-flow32")
    plan = SolverPlan.reserve(solver.params(), 120, 24 << 30, torch.device("cuda"))
    rng = random.Random(0)
    best = {}
    for repeat in range(8):
        dims = [tuple(rng.randrange(24, 97) for _ in range(3)) for _ in range(120)]
        I = [torch.zeros(d, device="cuda") for d in dims]
        outs = [torch.empty(d + (3,), device="cuda") for d in dims]
        for on in (False, True):
            plan.set_resident(on)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            plan.retarget(dims)
            plan.solve(I, I, outs)
            best[on] = min(best.get(on, 1e9), time.perf_counter() - t0)
            torch.cuda.synchronize()
            plan.check()
            assert (plan.level_resident(1) > 0) == on
    plan.close()
    print("set-up", best)
    assert best[True] <= 5 * best[False], best
