"""Integral images of planes that clusters of two to seven CTAs share (more rows than eight CTAs hold, more planes than there is room for
clusters of eight), their first and last row in other CTAs, against a float64 sum; alone and in front of the slabs' forward.

Tolerance: a value is the sum of at most h + w + 16 rounded partial sums, none larger than the sum of magnitudes that it covers, so it is off by
at most (h + w + 16) 2^-24 of the largest such sum; outputs as in the parity tests."""
import pytest
import torch

from test_gpu_quad_pair_backward import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(41, 160, 872), (40, 161, 871), (37, 402, 681), (53, 612, 1077), (85, 272, 528), (85, 265, 527), (102, 467, 279),
                                   (46, 1153, 64), (47, 513, 131), (140, 331, 385), (70, 1030, 29), (34, 1100, 128)])
def test_integral_images(shape):
    import box_convolution as bc
    x = torch.randn(shape, device="cuda", generator=torch.Generator("cuda").manual_seed(sum(shape)))
    got = bc.integral_image(x)
    P, h, w = shape
    scale = x.double().abs().sum((1, 2)).max().item()
    bound = (h + w + 16) * 2.0 ** -24 * scale
    assert got.shape[-2:] == (h + 1, w + 1)
    got = got.view(P, h + 1, w + 1)
    assert not got[:, 0].any() and not got[:, :, 0].any()
    for p in range(0, P, 16):
        want = x[p:p + 16].double().cumsum(1).cumsum(2)
        assert (got[p:p + 16, 1:, 1:] - want).abs().max().item() <= bound


@pytest.mark.parametrize("shape", [(2, 20, 1, 272, 530), (1, 41, 2, 161, 871)])
def test_forward_by_slabs(shape):
    m, x, _ = _case(shape, True, True)
    with torch.no_grad():
        out = m(x)
        want = torch.cat([m.double()(x[i:i + 1].double()) for i in range(shape[0])])
    assert (out - want).abs().max() <= 1e-4 * want.abs().max()
