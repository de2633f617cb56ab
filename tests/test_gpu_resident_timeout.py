"""The bounded waits of the on-chip iterations, run out without faulting or hanging the GPU: a test hook
(svs_tvl1_plan_set_mute_test) has one box keep its faces to itself and shortens the waits to a few
milliseconds. The neighbours give up, the others follow, the host reads SVS_ERR_TIMEOUT once, and the
next solve of the plan is bitwise that of an undisturbed one: for the face words of every shape and
for the mbarriers within a cluster."""
import pytest
import torch

from singleventriclesegmentation_b200 import _lib, synthetic
from singleventriclesegmentation_b200.tvl13d import TVL13DOpticalFlow

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


@pytest.mark.parametrize("storage", ["f32", "f16-flow32"])
@pytest.mark.parametrize("shape,which,box", [
    ((24, 24, 24), 1, 0),      # a corner of the volume
    ((24, 24, 24), 1, 77),     # inside
    ((64, 65, 66), 2, 5),
    ((66, 71, 79), 3, 60),
    ((9, 11, 12), 4, 0),       # a cluster
    ((20, 20, 20), 4, 9),      # a cluster of 16 boxes
])
def test_mute_box_times_out_and_the_plan_recovers(cuda, storage, shape, which, box):
    solver = TVL13DOpticalFlow(1, 2, 24, 1.0, 0.025, 2, (0.5, 0.5, 0.25, 1.0), True, (5.0, 0.5), True, 1.0,
                               "CUBIC_HERMITESPLINE", "MIRROR", "numDofs", (1, 1, 1), torch.device("cuda"), storage=storage)
    f = synthetic.frame_pair(shape, seed=11)
    I = [[torch.from_numpy(f[k]).cuda()] for k in (0, 1)]
    plan = solver.plan_for([shape])
    out = lambda: [torch.empty(shape + (3,), device="cuda")]
    ref, bad, again = out(), out(), out()
    plan.solve(*I, ref)
    plan.check()
    assert plan.level_resident_shape(0) == which
    plan.set_mute_test(level=0, box=box, wait_us=4000)
    plan.solve(*I, bad)
    with pytest.raises(_lib.SVSError) as e:
        plan.check()
    assert e.value.status == _lib.SVS_ERR_TIMEOUT
    assert plan.level_resident_shape(0) == which   # the waits that ran out were the on-chip ones
    plan.check()                                   # reported once
    plan.set_mute_test()
    plan.solve(*I, again)
    plan.check()
    assert torch.equal(again[0], ref[0])
