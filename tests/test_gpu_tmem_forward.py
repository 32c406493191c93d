"""Forward of whole planes through tensor memory: planes, filters and column tiles at which its streaming kernels begin, end
and change (one plane a CTA, two, three and many; units that fill the four quarters and units that do not), against the
float64 kernels, and where an address that no vector access fits sends the same call to another kernel.

Tolerance: 1e-4 of the largest output, as in the parity tests; the 16-bit types round the output once more, by at most half
a unit in the last place of 8 (bfloat16) or 11 (float16) bits, 2^-8 or 2^-11 of its own magnitude.
"""
import numpy as np
import pytest
import torch

from conftest import kernels_run, max_rel

pytestmark = pytest.mark.gpu

ROUNDING = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _module(bc, shape, exact, normalize):
    N, C, F, h, w = shape
    rng = np.random.default_rng(h * 1000 + w + F)
    m = bc.BoxConv2d(C, F, h, w, normalize=normalize)
    m.exact = exact
    for lo, hi, rep, size in ((m.x_min, m.x_max, m.reparametrization_h, h), (m.y_min, m.y_max, m.reparametrization_w, w)):
        centre, half = rng.uniform(-size / 2, size / 2, (C, F)), rng.uniform(1.2, size / 3 + 1.2, (C, F))
        lo.data.copy_(torch.from_numpy((centre - half) / rep))
        hi.data.copy_(torch.from_numpy((centre + half) / rep))
    return m.cuda()


# (8 x 128: one tile; 64 x 128 and 32 x 160: two CTAs an SM, 74 planes and up to two rounds and a bit of them; 72 x 68, 64 x 256 and
# 128 x 128: one CTA; 72 x 200 and 128 x 256: one plane a CTA; 3, 6 and 9 units)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(2, 37, 4, 8, 128), (1, 297, 4, 64, 128), (3, 211, 3, 40, 68), (2, 40, 8, 16, 100), (5, 64, 2, 32, 160), (2, 80, 3, 24, 256),
                                   (1, 75, 6, 72, 68), (3, 101, 2, 64, 256), (2, 60, 4, 128, 128), (1, 74, 2, 72, 200), (1, 90, 4, 128, 256),
                                   (1, 74, 32, 16, 72)])
def test_forward_against_float64(shape, dtype):
    import box_convolution as bc
    N, C, F, h, w = shape
    x = torch.randn(N, C, h, w, device="cuda", generator=torch.Generator("cuda").manual_seed(w)).to(dtype)
    for exact, normalize in ((True, True), (False, True), (True, False)):
        m = _module(bc, shape, exact, normalize)
        with torch.no_grad():
            got = m.to(dtype)(x)
            want = m.double()(x.double())
        assert max_rel(got.double().cpu().numpy(), want.cpu().numpy()) < 1e-4 + ROUNDING[dtype]


@pytest.mark.parametrize("shape", [(3, 50, 4, 64, 128), (1, 80, 4, 128, 256), (2, 60, 4, 96, 128)])
def test_same_values_at_another_address(shape):
    import box_convolution as bc
    N, C, F, h, w = shape
    m = _module(bc, shape, True, True)
    x = torch.randn(N, C, h, w, device="cuda", generator=torch.Generator("cuda").manual_seed(w))
    off = torch.empty(x.numel() + 1, device="cuda")[1:].view_as(x).copy_(x)
    with torch.no_grad():
        assert max_rel(m(off).cpu().numpy(), m(x).cpu().numpy()) < 1e-5      # (other kernels, another order of additions at most)


def test_boxes_beyond_the_plane():
    """All rows of a box above, below, left or right of the plane: sums over what is not there, zero."""
    import box_convolution as bc
    from box_convolution.function import BoxConvolutionFunction
    C, F, h, w = 80, 4, 64, 128
    m = _module(bc, (1, C, F, h, w), True, False)
    far = torch.tensor([[-200.0, -150.0, -3.0, 3.0], [150.0, 200.0, -3.0, 3.0], [-3.0, 3.0, -400.0, -300.0], [-3.0, 3.0, 300.0, 400.0]])
    pixels = [far[:, j].repeat(C, 1).cuda() for j in range(4)]
    m.eval()
    with torch.no_grad():
        for p, v, rep in zip((m.x_min, m.x_max, m.y_min, m.y_max), pixels, [m.reparametrization_h] * 2 + [m.reparametrization_w] * 2):
            p.copy_(v / rep)
        x = torch.rand(1, C, h, w, device="cuda")
        out = BoxConvolutionFunction.apply(x, m.x_min, m.x_max, m.y_min, m.y_max, m.reparametrization_h, m.reparametrization_w, False, True)
    # what is left is the rounding of 16 terms, sums of up to h w values in [0, 1) each, that cancel
    assert out.abs().max() < 16 * 2.0 ** -24 * h * w


@pytest.mark.parametrize("side", range(4))
def test_boxes_that_are_no_numbers(side):
    """A parameter that is NaN, or infinite where fractions count, makes all outputs of its filter NaN, those above the plane too;
    the other filters keep theirs."""
    import box_convolution as bc
    C, F, h, w = 80, 4, 64, 128
    x = torch.rand(1, C, h, w, device="cuda")
    pixels = [torch.full((C, F), v, device="cuda") for v in (-90.0, -70.0, -3.0, 3.0)]      # (above the plane for every row)
    pixels[0][:, ::2], pixels[1][:, ::2] = -2.5, 2.25
    clean = bc.BoxConvolutionFunction.apply(x, *pixels, 1.0, 1.0, False, True).view(C, F, h, w)
    for value in (float("nan"), float("inf") * (-1 if side % 2 == 0 else 1)):
        p = [v.clone() for v in pixels]
        p[side][:, 1], p[side][:, 2] = value, value
        assert "forward_tmem_stream_kernel" in kernels_run(lambda: bc.BoxConvolutionFunction.apply(x, *p, 1.0, 1.0, False, True))
        out = bc.BoxConvolutionFunction.apply(x, *p, 1.0, 1.0, False, True).view(C, F, h, w)
        assert out[:, 1:3].isnan().all()
        assert torch.equal(out[:, ::3], clean[:, ::3])


# both sides of the rule's lines: planes, tiles for either kernel, filters that leave quarters of tensor memory idle, alignment, heights
@pytest.mark.parametrize("shape,kernel", [
    ((2, 37, 4, 64, 128), "forward_tmem_stream_kernel"), ((1, 73, 4, 64, 128), "forward_quad_kernel"),
    ((1, 74, 4, 128, 128), "forward_tmem_stream_kernel"), ((1, 74, 4, 128, 256), "forward_tmem_kernel"),
    ((1, 223, 4, 128, 128), "forward_tmem_stream_kernel"), ((1, 149, 4, 128, 128), "forward_quad_kernel"),
    ((1, 80, 5, 64, 128), "forward_quad_kernel"), ((1, 80, 4, 60, 128), "forward_quad_kernel"), ((1, 80, 4, 64, 126), "forward_quad_kernel"),
    ((1, 80, 4, 136, 128), "forward_quad_kernel"), ((1, 80, 4, 96, 132), "forward_plane_kernel"), ((1, 80, 4, 64, 64), "forward_plane_kernel")])
def test_kernel_that_serves_a_plane(shape, kernel):
    import box_convolution as bc
    N, C, F, h, w = shape
    m, x = _module(bc, shape, True, True), torch.randn(N, C, h, w, device="cuda")
    with torch.no_grad():
        assert kernel in kernels_run(lambda: m(x))
