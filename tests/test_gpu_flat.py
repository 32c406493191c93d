"""Whole planes by strips dealt out to lanes: sizes at which its tiles, row groups, CTAs and clusters begin and end (one strip a
row and several a tile, rows over several tiles, eight row groups and more, samples that share a CTA and a last CTA of fewer, two tiles a
warp, filters and tiles over several CTAs, planes that leave no
room for scan corners), rows that no vector access fits, 16-bit tensors, the input's integral image instead of the input, and what infinities
reach; against the float64
kernels.

Tolerances as in the parity tests: outputs and grad-input 1e-4 and parameter gradients 1e-3 of the largest magnitude; 16-bit results are
rounded once more, by at most 2^-8 (bfloat16) or 2^-11 (float16) of their magnitude.
"""
import pytest
import torch

from conftest import kernels_run, max_rel
from test_gpu_quad_pair_backward import NAMES, ROUNDING, _case, _grads

pytestmark = pytest.mark.gpu

# samples, channels, filters, rows, columns
SHAPES = [(1, 1, 1, 1, 1), (3, 2, 2, 7, 3), (2, 1, 3, 9, 29), (700, 1, 2, 8, 4), (650, 2, 1, 20, 25), (331, 2, 2, 21, 31), (301, 1, 4, 33, 37), (75, 4, 2, 72, 48), (2, 3, 3, 65, 61),
          (1, 4, 2, 64, 300), (2, 2, 5, 24, 516), (1, 3, 8, 40, 260), (150, 1, 2, 88, 124), (3, 1, 4, 100, 130), (1, 150, 1, 110, 117), (2, 2, 3, 200, 60), (1, 2, 2, 280, 26), (1, 2, 6, 1020, 30), (150, 1, 2, 256, 64),
          (1, 2, 3, 31, 1020), (2, 3, 4, 120, 200), (1, 2, 4, 126, 252), (150, 1, 3, 96, 140), (149, 1, 2, 110, 130)]
# ... of which fixed tiles serve
FIXED = {(700, 1, 2, 8, 4): "backward_square_kernel", (150, 1, 2, 88, 124): "backward_quad_kernel", (1, 150, 1, 110, 117): "backward_quad_kernel"}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", SHAPES)
def test_gradients_against_float64(shape, dtype):
    m, x, g = _case(shape, shape[3] % 3 != 0, True, dtype)
    assert FIXED.get(shape, "backward_plane_kernel") in kernels_run(lambda: _grads(m, x, g))
    gin, gp = _grads(m, x, g)
    want_in, want_p = _grads(m.double(), x.double(), g.double())
    assert max_rel(gin.double().cpu().numpy(), want_in.cpu().numpy()) < 1e-4 + ROUNDING[dtype]
    assert max_rel(gp.cpu().numpy(), want_p.cpu().numpy()) < 1e-3 + ROUNDING[dtype]


FORWARD = [(1, 2, 3, 72, 133), (3, 2, 4, 96, 132), (2, 75, 1, 130, 50), (40, 4, 6, 280, 26), (1, 2, 4, 1020, 30), (1, 2, 2, 1024, 32), (1, 1, 3, 31, 1020), (2, 3, 3, 93, 157), (150, 1, 2, 110, 117),
           (2, 4, 4, 126, 252), (1, 16, 2, 192, 136), (5, 2, 1, 40, 300)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", FORWARD)
def test_outputs_against_float64(shape, dtype):
    m, x, _ = _case(shape, shape[3] % 3 != 0, True, dtype)
    with torch.no_grad():
        m.eval()
        assert "forward_flat_kernel" in kernels_run(lambda: m(x))
        out = m(x)
        want = m.double()(x.double())
    assert max_rel(out.double().cpu().numpy(), want.cpu().numpy()) < 1e-4 + ROUNDING[dtype]


# (no room for scan corners in the tall ones)
@pytest.mark.parametrize("shape", [(20, 1, 3, 72, 133), (20, 1, 4, 1020, 30), (20, 1, 3, 1024, 32), (20, 1, 3, 31, 1020), (19, 1, 3, 93, 157), (20, 2, 3, 126, 252)])
def test_outputs_from_the_integral_image_alone(shape):
    import box_convolution as bc
    m, x, _ = _case(shape, True, True)
    pixels = [p.detach() for p in m.get_actual_parameters()]
    integ = bc.integral_image(x.double()).float()
    assert kernels_run(lambda: bc.box_convolution_forward(integ, *pixels, True, True)) == ["forward_flat_kernel"]
    out = bc.box_convolution_forward(integ, *pixels, True, True)
    with torch.no_grad():
        want = m.eval().double()(x.double())
    assert max_rel(out.cpu().numpy(), want.cpu().numpy()) < 1e-4


@pytest.mark.parametrize("shape", [(180, 1, 4, 96, 132), (180, 1, 4, 97, 133), (33, 1, 4, 96, 144), (20, 1, 8, 80, 188)])
def test_gradients_from_the_integral_image_alone(shape):
    """13 to 16 tiles: two a warp, and filters over clusters of as many CTAs as run at once."""
    import box_convolution as bc
    m, x, g = _case(shape, True, True)
    pixels = [p.detach() for p in m.get_actual_parameters()]
    integ = bc.integral_image(x.double()).float()

    def grads():
        return bc.box_convolution_backward(integ, *pixels, g, g, m.reparametrization_h, m.reparametrization_w, True, True, True, True, True, True, True)
    assert "backward_plane_kernel" in kernels_run(grads)
    got = grads()
    want_in, want_p = _grads(m.double(), x.double(), g.double())
    rounding = 8 * 2.0 ** -24 * float(integ.abs().max())      # (as below)
    assert max_rel(got[0].cpu().numpy(), want_in.cpu().numpy()) < 1e-4
    assert max_rel(torch.stack([t.double() for t in got[1:]]).cpu().numpy(), want_p.cpu().numpy()) < 1e-3 + rounding


@pytest.mark.parametrize("shape", FORWARD)
def test_fused_and_from_the_integral_image(shape):
    import box_convolution as bc
    N, C, F, h, w = shape
    m, x, g = _case(shape, True, True)
    m.eval()
    scale, shift = torch.rand(C * F, device="cuda") + 0.5, torch.rand(C * F, device="cuda") - 0.5
    with torch.no_grad():
        out = bc.fused_box_block(m, x, input_relu=True, scale=scale, shift=shift, residual=g, output_relu=True, out=g.clone())
        alias = g.clone()
        bc.fused_box_block(m, x, input_relu=True, scale=scale, shift=shift, residual=alias, output_relu=True, out=alias)
        integ = bc.integral_image(x.double()).float()
        from_integ = bc.box_convolution_forward(integ, *m.get_actual_parameters(), True, True)
        plain, m64 = m(x), m.double()
        want = (m64(x.double().relu()) * scale.double().view(1, -1, 1, 1) + shift.double().view(1, -1, 1, 1) + g.double()).relu()
    assert torch.equal(out, alias)
    assert max_rel(out.double().cpu().numpy(), want.cpu().numpy()) < 1e-4
    assert max_rel(from_integ.cpu().numpy(), plain.cpu().numpy()) < 1e-4
    if F == 1:      # in place: output over input
        own = x.clone()
        bc.fused_box_block(m.float(), own, out=own)
        assert torch.equal(own, plain)


@pytest.mark.parametrize("shape", [s for s in SHAPES if s[0] * s[1] * s[3] * s[4] < 200000])
def test_four_functions_and_subsets(shape):
    import box_convolution as bc
    m, x, g = _case(shape, True, True)
    gin, gp = _grads(m, x, g)
    pixels = [p.detach() for p in m.get_actual_parameters()]
    integ = bc.integral_image(x.double()).float()
    grads = bc.box_convolution_backward(integ, *pixels, g, g, m.reparametrization_h, m.reparametrization_w, True, True, True, True, True, True, True)
    # (the input's pixels are differences of its rounded integral image)
    rounding = 8 * 2.0 ** -24 * float(integ.abs().max())
    assert max_rel(grads[0].cpu().numpy(), gin.cpu().numpy()) < 1e-4
    assert max_rel(torch.stack([t.double() for t in grads[1:]]).cpu().numpy(), gp.cpu().numpy()) < 1e-3 + rounding
    for n in NAMES:
        getattr(m, n).requires_grad_(False)
    x = x.detach().requires_grad_()
    m(x).backward(g)
    assert max_rel(x.grad.cpu().numpy(), gin.cpu().numpy()) < 1e-6


# (the last one or two: tiles of 8 x 128, one a warp up to 148 planes and two above)
@pytest.mark.parametrize("shape,kernels", [((40, 8, 6, 50, 40), {"backward_plane_kernel"}), ((300, 1, 5, 90, 60), {"backward_plane_kernel"}), ((160, 1, 3, 152, 96), {"backward_plane_kernel"}),
                                           ((200, 1, 3, 72, 160), {"backward_plane_kernel"}), ((300, 1, 4, 128, 72), {"backward_plane_kernel"}),
                                           ((150, 1, 2, 56, 160), {"backward_quad_kernel", "backward_quad_pair_kernel"}), ((300, 1, 2, 128, 72), {"backward_quad_kernel", "backward_quad_pair_kernel"}),
                                           ((80, 2, 4, 64, 200), {"backward_quad_kernel", "backward_quad_pair_kernel"}), ((75, 2, 6, 112, 92), {"backward_quad_kernel", "backward_quad_pair_kernel"})])
def test_a_part_of_a_batch_gives_the_bits_of_the_whole(shape, kernels):
    """Few samples have their filters spread over a cluster of CTAs, or one tile a warp instead of two."""
    m, x, g = _case(shape, True, True)
    whole, _ = _grads(m, x, g)
    ran = [k for n in (3, shape[0]) for k in kernels_run(lambda: _grads(m, x[:n], g[:n])) if k.startswith("backward")]
    assert set(ran) == kernels
    for a, b in ((0, 1), (5, 8), (3, 40), (shape[0] - 30, shape[0])):
        part, _ = _grads(m, x[a:b], g[a:b])
        assert torch.equal(part, whole[a:b])


@pytest.mark.parametrize("shape,same", [((64, 2, 3, 93, 157), True), ((16, 16, 4, 160, 64), False)])
def test_outputs_of_a_part_of_a_batch(shape, same):
    """Equal within a kernel; where few samples have another, equal to rounding."""
    m, x, _ = _case(shape, True, True)
    m.eval()
    with torch.no_grad():
        whole, part = m(x), m(x[3:5])
        kernels = set(kernels_run(lambda: (m(x), m(x[3:5]))))
    assert kernels == ({"forward_flat_kernel"} if same else {"forward_plane_kernel", "forward_flat_kernel"})
    if same:
        assert torch.equal(part, whole[3:5])
    else:
        assert max_rel(part.cpu().numpy(), whole[3:5].cpu().numpy()) < 1e-5


@pytest.mark.parametrize("shape", [(2, 2, 2, 65, 61), (300, 1, 2, 21, 31), (1, 1, 2, 13, 300)])
def test_infinities_reach_no_further_than_their_boxes(shape):
    """An infinity in the last row of grad_output, and boxes that look away from it: grad-input of rows that do not gather from it, and
    the parameter gradients of filters none of whose pixels do, stay as they are without it."""
    m, x, g = _case(shape, True, True)
    N, C, F, h, w = shape
    with torch.no_grad():      # filter 0 of every channel gathers from rows above the pixel's own, the mirrored box below... and filter 1 from below
        m.x_min.copy_(torch.tensor([2.5, -4.5]).expand(C, F) / m.reparametrization_h)
        m.x_max.copy_(torch.tensor([4.25, -2.25]).expand(C, F) / m.reparametrization_h)
    clean, clean_p = _grads(m, x, g)
    g = g.clone().view(N, C, F, h, w)
    g[0, 0, 0, h - 1, w // 2] = float("inf")
    gin, gp = _grads(m, x, g.view(N, C * F, h, w))
    # the mirrored box of filter 0 reaches from row p - 5 to p - 2: only rows that do not exist would see the last row
    assert torch.equal(gin, clean)
    assert torch.equal(gp, clean_p)
