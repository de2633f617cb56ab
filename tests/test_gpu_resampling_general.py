"""The general kernels of the resampling operators, which serve what the grid kernels do not: launches
beyond a grid's limits (65,535 planes or volumes), and samples beyond the 32-bit coordinate range."""
import numpy as np
import pytest
import torch

from singleventriclesegmentation_b200 import opticalFlow as of

pytestmark = pytest.mark.gpu

TALL = 65540  # planes: beyond a grid's second dimension, so that the general warp kernel runs


def mesh(*n):
    return of.MeshInfo3D(*n, *(float(v - 1) for v in n))


FAR = [np.inf, -np.inf, np.nan, 3e9, -3e9, 1e12, -1e12, 2e6, -2e6, -2.5, 0.25]


def far_flow(ny, nx, axis, dtype):
    """Displacements of a plane: fractions of a voxel, on one axis the values of FAR."""
    g = torch.Generator(device="cuda").manual_seed(1)
    plane = torch.rand((ny, nx), generator=g, device="cuda", dtype=dtype) + 0.5
    phi = 0.3 * torch.rand((ny, nx, 3), generator=g, device="cuda", dtype=dtype)
    which = torch.arange(ny * nx, device="cuda").reshape(ny, nx) % len(FAR)
    phi[..., axis] = torch.tensor(FAR, device="cuda", dtype=dtype)[which]
    return plane, phi, which


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("interp", ["NEAREST", "LINEAR", "CUBIC_HERMITESPLINE"])
@pytest.mark.parametrize("boundary", ["NEAREST", "MIRROR", "REFLECT"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_far_samples_equal_the_general_kernel(cuda, dtype, interp, boundary, axis):
    """Displacements without end, without a value and beyond 2^31 voxels, one axis at a time: a volume of
    few planes against a tall one of the same planes. All planes are alike, so that both fold to the same
    values along z. What both kernels compute in the same operations up to a fused rounding agrees to a few ulp."""
    ny, nx = 5, 64
    plane, phi, _ = far_flow(ny, nx, axis, dtype)
    out = []
    for nz in (8, TALL):
        u = plane.expand(1, 1, nz, ny, nx).contiguous()
        f = phi.expand(1, nz, ny, nx, 3).contiguous()
        op = of.WarpingCNN3D(mesh(nz, ny, nx), getattr(of, "INTERPOLATE_" + interp), getattr(of, "BOUNDARY_" + boundary))
        out.append(op.forward(u, f)[0, 0, :6])
    tol = 64 * torch.finfo(dtype).eps
    torch.testing.assert_close(out[0], out[1], rtol=tol, atol=tol, equal_nan=True)


@pytest.mark.parametrize("interp", ["NEAREST", "LINEAR", "CUBIC_HERMITESPLINE"])
@pytest.mark.parametrize("boundary", ["NEAREST", "MIRROR", "REFLECT"])
def test_far_samples_leave_the_other_gradients(cuda, interp, boundary):
    """The backward pass with such samples among others: the others' flow gradients are those without them."""
    nz, ny, nx = 6, 9, 64
    plane, phi, which = far_flow(ny, nx, 1, torch.float64)
    u = plane.expand(nz, ny, nx).contiguous()
    near = phi.clone()
    near[..., 1] = torch.where(which < FAR.index(-2.5), torch.zeros_like(phi[..., 1]), phi[..., 1])
    op = of.Warping3D(mesh(nz, ny, nx), getattr(of, "INTERPOLATE_" + interp), getattr(of, "BOUNDARY_" + boundary))
    got, want = (op.backward(u, f.expand(nz, ny, nx, 3).contiguous(), torch.ones_like(u))[1] for f in (phi, near))
    ordinary = (which >= FAR.index(-2.5)).expand(nz, ny, nx)
    assert torch.equal(got[ordinary], want[ordinary])


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("interp", ["NEAREST", "LINEAR", "CUBIC_HERMITESPLINE"])
def test_tall_volumes(cuda, dtype, interp):
    """Planes 10 to 19 of a tall volume (general kernel) and of its first 30 planes (grid kernel)."""
    g = torch.Generator(device="cuda").manual_seed(3)
    ny, nx, C = 5, 13, 3
    u = torch.rand((TALL, ny, nx, C), generator=g, device="cuda", dtype=dtype)
    phi = 4 * torch.rand((TALL, ny, nx, 3), generator=g, device="cuda", dtype=dtype) - 2
    tol = 64 * torch.finfo(dtype).eps
    kind = (getattr(of, "INTERPOLATE_" + interp), of.BOUNDARY_MIRROR)
    for name, a in (("forward", u[..., 0].contiguous()), ("forwardVectorField", u)):
        tall, few = (getattr(of.Warping3D(mesh(n, ny, nx), *kind), name)(a[:n].contiguous(), phi[:n].contiguous())[10:20]
                     for n in (TALL, 30))
        torch.testing.assert_close(tall, few, rtol=tol, atol=tol)
    b = u[..., :2].permute(3, 0, 1, 2)[None]
    tall, few = (of.WarpingCNN3D(mesh(n, ny, nx), *kind).forward(b[:, :, :n].contiguous(), phi[None, :n].contiguous())[:, :, 10:20]
                 for n in (TALL, 30))
    torch.testing.assert_close(tall, few, rtol=tol, atol=tol)


@pytest.mark.parametrize("interp", ["LINEAR", "CUBIC_HERMITESPLINE"])
def test_many_volumes(cuda, interp):
    g = torch.Generator(device="cuda").manual_seed(4)
    n = 65540
    u = torch.rand((n, 1, 3, 2, 4), generator=g, device="cuda")
    phi = 3 * torch.rand((n, 3, 2, 4, 3), generator=g, device="cuda") - 1.5
    op = of.WarpingCNN3D(mesh(3, 2, 4), getattr(of, "INTERPOLATE_" + interp), of.BOUNDARY_REFLECT)
    tol = 64 * torch.finfo(torch.float32).eps
    torch.testing.assert_close(op.forward(u, phi)[-40:], op.forward(u[-40:].contiguous(), phi[-40:].contiguous()), rtol=tol, atol=tol)


@pytest.mark.parametrize("interp", ["NEAREST", "LINEAR", "CUBIC_HERMITESPLINE"])
def test_tall_targets(cuda, oracle, interp):
    """A prolongation onto more planes than a grid has, with components padded and cropped."""
    src, dst, C = (4, 3, 5), (TALL, 2, 3), 3
    u = np.random.default_rng(5).standard_normal(src + (C,)).astype(np.float32)
    op = of.Prolongation3D(mesh(*src), mesh(*dst), getattr(of, "INTERPOLATE_" + interp), of.BOUNDARY_MIRROR)
    t = torch.from_numpy(u).cuda()
    got = op.forwardVectorField(t)
    want = oracle.prolongate(u, tuple(float(s - 1) for s in src), dst, tuple(float(s - 1) for s in dst), interp, "MIRROR")
    if interp == "NEAREST":  # a target half way between two nodes may go to either
        assert (np.abs(got.cpu().numpy() - want) > 2e-5).mean() < 1e-4
    else:
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2e-5, atol=2e-5)
    for n in (1, C, C + 2):
        assert torch.equal(op.forwardVectorFieldPadded(t, n), torch.nn.functional.pad(got, (0, n - C)))
