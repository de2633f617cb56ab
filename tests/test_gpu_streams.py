"""Solves of several plans on several streams: on-chip launches whose boxes wait for one another take
turns, and nothing else does. A bounded sleep kernel in front of one stream's solve shows which
work of the other stream waits for it."""
import time

import pytest
import torch

from singleventriclesegmentation_b200 import synthetic
from singleventriclesegmentation_b200.tvl13d import TVL13DOpticalFlow

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

SLEEP = 1_000_000_000  # cycles: about half a second


class Solve:
    """One plan with its own stream, inputs and result."""

    def __init__(self, shape, scales, warps, iters, seed=1):
        self.shape = shape
        solver = TVL13DOpticalFlow(scales, warps, iters, 1.0, 0.025, 2, (0.5, 0.5, 0.25, 1.0), True, (5.0, 0.5), True,
                                   1.0, "CUBIC_HERMITESPLINE", "MIRROR", "numDofs", (1, 1, 1), torch.device("cuda"),
                                   storage="f16-flow32")
        self.solver, self.plan = solver, solver.plan_for([shape])
        f = synthetic.frame_pair(shape, seed=seed)
        self.I = [torch.from_numpy(f[k]).cuda() for k in (0, 1)]
        self.out = torch.empty(shape + (3,), device="cuda")
        self.stream, self.done = torch.cuda.Stream(), torch.cuda.Event()
        self.go()                      # set-up and capture
        torch.cuda.synchronize()
        self.want = self.out.clone()
        self.out.zero_()
        torch.cuda.synchronize()

    def go(self, sleep=0):
        with torch.cuda.stream(self.stream):
            if sleep:
                torch.cuda._sleep(sleep)
            self.plan.solve([self.I[0]], [self.I[1]], [self.out])
            self.done.record()

    def check(self):
        self.done.synchronize()
        self.plan.check()
        assert torch.equal(self.out, self.want)


def test_on_chip_launches_take_turns(cuda):
    a, b = Solve((32, 32, 32), 1, 2, 20), Solve((40, 24, 32), 1, 2, 20, seed=2)
    assert a.plan.level_resident_shape(0) in (1, 2, 3) and b.plan.level_resident_shape(0) in (1, 2, 3)
    a.go(SLEEP)
    b.go()
    time.sleep(0.1)
    assert not a.done.query() and not b.done.query()
    a.check()
    b.check()


def test_volumes_in_one_cluster_take_none(cuda):
    """Neither wait for the solve before them nor hold up the next one."""
    first, small = Solve((32, 32, 32), 1, 2, 20), Solve((9, 11, 12), 1, 2, 20)
    assert first.plan.level_resident_shape(0) in (1, 2, 3) and small.plan.level_resident_shape(0) == 4
    for a, b in ((first, small), (small, first)):
        a.go(SLEEP)
        b.go()
        b.done.synchronize()
        assert not a.done.query()
        a.check()
        b.check()


def test_levels_per_iteration_are_not_part_of_a_turn(cuda):
    """A large volume's finest level, one launch per iteration, runs beside another stream's solve."""
    large, small = Solve((104, 104, 100), 2, 5, 300), Solve((32, 32, 32), 1, 1, 10)
    assert large.plan.level_resident(0) == 0 and large.plan.level_resident_shape(1) in (1, 2, 3)
    assert small.plan.level_resident_shape(0) in (1, 2, 3)
    large.go()
    small.go()
    small.done.synchronize()
    assert not large.done.query()
    large.check()
    small.check()
