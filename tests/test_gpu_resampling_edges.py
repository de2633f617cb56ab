"""Edges of the grid kernels of the resampling operators: the warps where a block ends, against the
oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def T(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda")


@pytest.fixture(scope="module")
def of():
    from singleventriclesegmentation_b200 import opticalFlow
    return opticalFlow


@pytest.mark.parametrize("interp", ["LINEAR", "CUBIC_HERMITESPLINE"])
@pytest.mark.parametrize("shape", [(1, 16, 16), (2, 1, 257), (3, 5, 51), (4, 4, 4)])
def test_warp_edges(cuda, oracle, of, interp, shape):
    """Planes of 256, 257, 255 and 16 voxels; displacements that reach over every face, and whole
    and almost whole ones (w + 1 rounding up to 2)."""
    rng = np.random.default_rng(sum(shape))
    m = rng.standard_normal((2, 2) + shape).astype(np.float32)
    phi = (rng.standard_normal((2,) + shape + (3,)) * 3).astype(np.float32)
    phi[0, ..., 0] = np.round(phi[0, ..., 0])
    phi[1, ..., 1] = -1e-8
    mesh = of.MeshInfo3D(*shape, *(max(s - 1, 1) for s in shape))
    h = tuple(v if np.isfinite(v) else 1.0 for v in mesh.h())
    mesh._h = h
    op = of.WarpingCNN3D(mesh, getattr(of, "INTERPOLATE_" + interp), of.BOUNDARY_MIRROR)
    got = op.forward(T(m), T(phi)).cpu().numpy()
    want = oracle.warp_cnn(m, phi, h, interp, "MIRROR")
    np.testing.assert_allclose(got, want, rtol=2e-5, atol=2e-5)
