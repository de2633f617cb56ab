"""The median filters against a sort of every window (torch), exactly: sizes at the edges of the z
runs and blocks, ties, and values that take the fallback (NaN, infinities)."""
import pytest
import torch

from singleventriclesegmentation_b200.flow_utils import apply_median_filter

pytestmark = pytest.mark.gpu


def fold(i, n):
    i = torch.where(i < 0, -i - 1, i)
    return torch.where(i > n - 1, 2 * n - 1 - i, i).clamp(0, n - 1)


def windows(x, ks):
    """[Z, Y, X, C] -> [Z, Y, X, C, ks^3], scipy 'reflect' at the faces, taps in (z, y, x) order."""
    r = ks // 2
    for axis in range(3):
        n = x.shape[axis]
        x = x.index_select(axis, fold(torch.arange(-r, n + r, device=x.device), n))
    return x.unfold(0, ks, 1).unfold(1, ks, 1).unfold(2, ks, 1).flatten(-3)


@pytest.mark.parametrize("ks", [3, 5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(1, 1, 1, 3), (8, 3, 43, 3), (9, 5, 42, 3), (17, 2, 128, 1), (10, 4, 129, 1), (7, 6, 5, 9)])
def test_median_is_the_middle_of_the_sorted_window(cuda, ks, dtype, shape):
    g = torch.Generator(device="cuda").manual_seed(sum(shape) + ks)
    x = torch.randn(shape, generator=g, device="cuda", dtype=dtype)
    for v in (x, (2 * x).round(), torch.where(x.abs() > 1.5, x * float("inf"), x)):  # ties, infinities
        want = windows(v, ks).sort(-1).values[..., ks ** 3 // 2]
        assert torch.equal(apply_median_filter(v, ks), want)


def test_median3_leaves_nans_out(cuda):
    """A window's NaNs are left out as if greater than every value; with fewer than 14 values left
    the first tap stays."""
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn((9, 11, 13, 3), generator=g, device="cuda")
    x[torch.rand(x.shape, generator=g, device="cuda") < 0.3] = float("nan")
    w = windows(x, 3)
    want = torch.where((~w.isnan()).sum(-1) >= 14, w.nan_to_num(nan=float("inf")).sort(-1).values[..., 13], w[..., 0])
    got = apply_median_filter(x, 3)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))
