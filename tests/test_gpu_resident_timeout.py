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


def make_solver(**kw):
    return TVL13DOpticalFlow(1, 2, 24, 1.0, 0.025, 2, (0.5, 0.5, 0.25, 1.0), True, (5.0, 0.5), True, 1.0,
                             "CUBIC_HERMITESPLINE", "MIRROR", "numDofs", (1, 1, 1), torch.device("cuda"), **kw)


def test_callers_that_never_check_are_told(cuda):
    """compute() of a solver: the next one raises, once; solver.check() does; and the plan's end does."""
    shape = (24, 24, 24)
    f = synthetic.frame_pair(shape, seed=11)
    I = [torch.from_numpy(f[k]).cuda() for k in (0, 1)]
    solver = make_solver(max_cached_plans=1)
    ref = solver.compute(*I)[0]
    plan = solver.plan_for([shape])
    solver.check()
    for report in (lambda: solver.compute(*I), solver.check, plan.poll):
        plan.set_mute_test(level=0, box=3, wait_us=4000)
        solver.compute(*I)
        torch.cuda.synchronize()
        plan.set_mute_test()
        with pytest.raises(_lib.SVSError) as e:
            report()
        assert e.value.status == _lib.SVS_ERR_TIMEOUT
        assert torch.equal(solver.compute(*I)[0], ref)
        solver.check()
    plan.set_mute_test(level=0, box=3, wait_us=4000)
    solver.compute(*I)
    with pytest.raises(_lib.SVSError) as e:
        solver.compute(I[0][:20].contiguous(), I[1][:20].contiguous())  # the one cached plan makes room
    assert e.value.status == _lib.SVS_ERR_TIMEOUT


def test_patient_files_are_not_passed_off_as_good(cuda, tmp_path):
    from singleventriclesegmentation_b200 import processor
    img = torch.from_numpy(synthetic.cine_sequence(T=3, shape=(20, 24, 24), seed=2)).cuda()
    solver = make_solver()
    processor.process_patients([("a", img, 0, 2)], solver, str(tmp_path))
    solver.plan_for([(20, 24, 24)] * 2).set_mute_test(level=0, box=1, wait_us=4000)
    with pytest.raises(_lib.SVSError):
        processor.process_patients([("b", img, 0, 2)], solver, str(tmp_path), modes=("forward",))


def test_server_hands_out_no_flows_of_a_failed_solve(cuda):
    from singleventriclesegmentation_b200.serving import FlowServer
    srv = FlowServer(budget_bytes=8 << 30, solver_args=dict(num_scales=1, max_warps=1, max_outer_iterations=24),
                     batch_voxels=4 * 24 ** 3, max_batch_pairs=4, num_plans=1)
    frames = torch.from_numpy(synthetic.cine_sequence(T=3, shape=(24, 24, 24), seed=1))
    srv.submit(frames).result(timeout=60)
    srv._slots[0].plan.set_mute_test(level=0, box=2, wait_us=4000)
    with pytest.raises(_lib.SVSError) as e:
        srv.submit(frames).result(timeout=60)
    assert e.value.status == _lib.SVS_ERR_TIMEOUT
    srv.close()


def test_making_and_ending_plans_pins_no_memory(cuda):
    """The status word costs a plan nothing: pinning memory for each took 4 to 20 ms where the rest of a
    plan's life takes about 3."""
    import time
    solver = make_solver()
    took = []
    for _ in range(20):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        solver.plan_for([(24, 24, 24)])
        solver._plans.popitem()[1].close()
        took.append(time.perf_counter() - t0)
    assert min(took) < 6e-3, took
