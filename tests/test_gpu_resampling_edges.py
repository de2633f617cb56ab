"""Edges of the grid kernels of the resampling operators: the warps and the prolongation where a block,
a run of z planes or a component row ends, against the oracle; padded and cropped time axes."""
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


@pytest.mark.parametrize("interp", ["NEAREST", "LINEAR", "CUBIC_HERMITESPLINE"])
@pytest.mark.parametrize("src,dst,C", [((3, 9, 8), (17, 6, 11), 1), ((16, 5, 7), (16, 8, 9), 3), ((5, 6, 7), (33, 4, 3), 25),
                                       ((20, 7, 6), (7, 5, 4), 9)])
def test_prolongation_edges(cuda, oracle, of, interp, src, dst, C):
    """z runs of exactly 16 and one more, planes shared by several targets and skipped between them,
    component rows that end inside a block."""
    rng = np.random.default_rng(C)
    u = rng.standard_normal(src + (C,)).astype(np.float32)
    old, new = of.MeshInfo3D(*src, *(s - 1 for s in src)), of.MeshInfo3D(*dst, *(s - 1 for s in dst))
    op = of.Prolongation3D(old, new, getattr(of, "INTERPOLATE_" + interp), of.BOUNDARY_MIRROR)
    got = op.forwardVectorField(T(u))
    one = of.Prolongation3D(old, new, getattr(of, "INTERPOLATE_" + interp), of.BOUNDARY_MIRROR)
    for c in range(C):
        assert torch.equal(one.forward(T(u[..., c])), got[..., c])
    want = oracle.prolongate(u, tuple(float(s - 1) for s in src), dst, tuple(float(s - 1) for s in dst), interp, "MIRROR")
    np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2e-5, atol=2e-5)
    for n in (1, C, C + 6):
        assert torch.equal(op.forwardVectorFieldPadded(T(u), n), torch.nn.functional.pad(got, (0, n - C)))


def test_frame_counts_that_are_none_are_refused(cuda):
    """A fraction of a frame, which torch's pad refuses; any integer type is one."""
    from singleventriclesegmentation_b200.preprocessing import resample_patient
    img = torch.rand(5, 6, 7, 4, device="cuda")
    want = resample_patient(img, shape=(6, 6, 6), pad_time=6)[0]
    assert tuple(want.shape) == (6, 6, 6, 6)
    assert torch.equal(resample_patient(img, shape=(6, 6, 6), pad_time=np.int64(6))[0], want)
    for t in (6.0, 6.5, "6"):
        with pytest.raises(TypeError):
            resample_patient(img, shape=(6, 6, 6), pad_time=t)
