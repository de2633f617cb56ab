"""The general kernels of the resampling operators, which serve what the grid kernels do not: samples
beyond the 32-bit coordinate range."""
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
