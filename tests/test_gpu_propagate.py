"""The mask chains in one native call against the same chains warped step by step: equal, for every
interpolation and boundary, no step and several, and the step-by-step form where the inputs ask for it."""
import pytest
import torch

from singleventriclesegmentation_b200.warping import Warp, propagate, propagate_batched

pytestmark = pytest.mark.gpu


def steps(warp, mask, flows):
    out = [mask]
    for f in flows:
        out.append(warp(out[-1], f.unsqueeze(0)))
    return torch.cat(out)


def thresholded(chain):
    return torch.where(chain > 0.5, 1.0, 0.0)


@pytest.mark.parametrize("interp", ["NEAREST", "LINEAR", "CUBIC_HERMITESPLINE"])
@pytest.mark.parametrize("boundary", ["NEAREST", "MIRROR", "REFLECT"])
@pytest.mark.parametrize("shape,T", [((7, 9, 33), 0), ((7, 16, 16), 1), ((5, 6, 43), 4)])
def test_native_chains_equal_steps(cuda, interp, boundary, shape, T):
    g = torch.Generator(device="cuda").manual_seed(T)
    warp = Warp(interp, boundary, "numDofs", (1, 1, 1))
    a, b = (torch.rand((1, 1) + shape, generator=g, device="cuda") for _ in range(2))
    f, k = (3 * torch.randn((T,) + shape + (3,), generator=g, device="cuda") for _ in range(2))
    fwd, bwd = propagate(warp, a, b, f, k)
    assert torch.equal(fwd, thresholded(steps(warp, a, f)))
    assert torch.equal(bwd, thresholded(steps(warp, b, k)).flip(0))
    # flows that are not contiguous, masks in double: the step-by-step form
    wide = torch.stack([f, f], -1)
    assert torch.equal(propagate(warp, a, b, wide[..., 0], wide[..., 1])[0], fwd)
    assert propagate(warp, a.double(), b.double(), f.double(), k.double())[0].dtype == torch.float32
    if T:
        flows = torch.stack([f, k], 1)
        chain = propagate_batched(warp, torch.cat([a, b]), flows)
        assert torch.equal(chain[:, 0], steps(warp, a, f)[:, None].reshape(chain[:, 0].shape))
        assert torch.equal(chain[:, 1], steps(warp, b, k)[:, None].reshape(chain[:, 1].shape))


def test_bad_shapes_still_raise(cuda):
    warp = Warp("LINEAR", "MIRROR", "numDofs", (1, 1, 1))
    a = torch.rand(1, 1, 4, 5, 6, device="cuda")
    with pytest.raises(RuntimeError):
        propagate(warp, a, a, torch.zeros(2, 4, 5, 7, 3, device="cuda"), torch.zeros(2, 4, 5, 7, 3, device="cuda"))
    with pytest.raises(AssertionError):
        propagate(warp, a, a, torch.zeros(2, 4, 5, 6, 3, device="cuda"), torch.zeros(1, 4, 5, 6, 3, device="cuda"))
