"""Backward of aligned planes of 14 to 32 tiles of 8 x 128 with two tiles a warp: the smallest and largest of them, numbers of planes
at which those of up to 16 tiles begin, widths that leave the second column tile nearly empty or fill it, every subset of gradients,
16-bit tensors, and the planes beside them that other kernels serve: odd numbers of tiles, more than 16 of one column, and an
address that no vector access fits; against the float64 kernels.

Tolerances as in the parity tests: grad-input 1e-4 and parameter gradients 1e-3 of the largest magnitude (the four together: one
of them can come out near zero by accident); 16-bit results are rounded once more, by at most 2^-8 (bfloat16) or 2^-11
(float16) of their magnitude.
"""
import numpy as np
import pytest
import torch

from conftest import kernels_run, max_rel

pytestmark = pytest.mark.gpu

ROUNDING = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}
NAMES = ("x_min", "x_max", "y_min", "y_max")


def _case(shape, exact, normalize, dtype=torch.float32):
    import box_convolution as bc
    N, C, F, h, w = shape
    rng = np.random.default_rng(h * 1000 + w + F)
    m = bc.BoxConv2d(C, F, h, w, normalize=normalize)
    m.exact = exact
    for lo, hi, rep, size in ((m.x_min, m.x_max, m.reparametrization_h, h), (m.y_min, m.y_max, m.reparametrization_w, w)):
        centre, half = rng.uniform(-size / 2, size / 2, (C, F)), rng.uniform(1.2, size / 3 + 1.2, (C, F))
        lo.data.copy_(torch.from_numpy((centre - half) / rep))
        hi.data.copy_(torch.from_numpy((centre + half) / rep))
    gen = torch.Generator("cuda").manual_seed(w)
    x = torch.randn(N, C, h, w, device="cuda", generator=gen).to(dtype)
    g = torch.randn(N, C * F, h, w, device="cuda", generator=gen).to(dtype)
    return m.cuda().to(dtype), x, g


def _grads(m, x, g):
    m.zero_grad(set_to_none=True)
    x = x.detach().requires_grad_()
    m(x).backward(g)
    return x.grad, torch.stack([getattr(m, n).grad.double() for n in NAMES])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("exact,normalize", [(True, True), (False, True), (True, False)])
@pytest.mark.parametrize("shape", [(1, 2, 2, 72, 132), (2, 3, 1, 72, 256), (3, 2, 3, 80, 200), (1, 2, 4, 128, 256), (2, 1, 2, 128, 228), (1, 150, 2, 72, 160), (1, 148, 2, 112, 68), (1, 149, 2, 112, 68),
                                   (2, 75, 3, 128, 128), (1, 150, 2, 56, 160), (5, 30, 1, 64, 256),
                                   # one column of 13, 15, 17 and of 18 to 32 tiles
                                   (1, 150, 2, 104, 128), (2, 75, 1, 120, 96), (2, 3, 2, 136, 128),
                                   (1, 2, 2, 144, 68), (2, 3, 4, 160, 128), (1, 160, 1, 192, 96), (2, 2, 3, 240, 100), (1, 2, 4, 256, 128)])
def test_gradients_against_float64(shape, exact, normalize, dtype):
    if dtype == torch.float16 and not normalize:
        pytest.skip("sums that are divided by nothing exceed 65504")
    m, x, g = _case(shape, exact, normalize, dtype)
    gin, gp = _grads(m, x, g)
    want_in, want_p = _grads(m.double(), x.double(), g.double())
    assert max_rel(gin.double().cpu().numpy(), want_in.cpu().numpy()) < 1e-4 + ROUNDING[dtype]
    assert max_rel(gp.cpu().numpy(), want_p.cpu().numpy()) < 1e-3 + ROUNDING[dtype]


@pytest.mark.parametrize("wanted", ["input", "parameters"])
def test_subsets_equal_the_whole(wanted):
    m, x, g = _case((2, 3, 2, 80, 200), True, True)
    gin, gp = _grads(m, x, g)
    for n in NAMES:
        getattr(m, n).requires_grad_(wanted == "parameters")
    m.zero_grad(set_to_none=True)
    x = x.detach().requires_grad_(wanted == "input")
    m(x).backward(g)
    if wanted == "input":
        assert max_rel(x.grad.cpu().numpy(), gin.cpu().numpy()) < 1e-6
    else:
        assert max_rel(torch.stack([getattr(m, n).grad.double() for n in NAMES]).cpu().numpy(), gp.cpu().numpy()) < 1e-6


def test_same_values_at_another_address():
    m, x, g = _case((2, 3, 2, 80, 200), True, True)
    gin, gp = _grads(m, x, g)
    off = torch.empty(g.numel() + 1, device="cuda")[1:].view_as(g).copy_(g)
    gin_off, gp_off = _grads(m, x, off)
    assert max_rel(gin_off.cpu().numpy(), gin.cpu().numpy()) < 1e-5      # (other kernels, another order of additions)
    assert max_rel(gp_off.cpu().numpy(), gp.cpu().numpy()) < 1e-4


# both sides of the rule's lines: one and two columns of 16 and 18 tiles, even and odd numbers, planes for two CTAs an SM, types
@pytest.mark.parametrize("shape,dtype,kernel", [
    ((1, 149, 2, 128, 128), torch.float32, "backward_quad_pair_kernel"), ((1, 149, 2, 112, 68), torch.bfloat16, "backward_quad_pair_kernel"),
    ((1, 148, 2, 128, 128), torch.float32, "backward_quad_kernel"), ((1, 149, 2, 120, 128), torch.float32, "backward_quad_kernel"),
    ((1, 149, 2, 104, 128), torch.float16, "backward_quad_kernel"), ((1, 149, 2, 96, 128), torch.float32, "backward_quad_kernel"),
    ((1, 3, 2, 144, 128), torch.float32, "backward_plane_kernel"), ((1, 3, 2, 136, 128), torch.float32, "backward_plane_kernel"),
    ((1, 3, 2, 256, 68), torch.bfloat16, "backward_plane_kernel"), ((1, 3, 2, 72, 132), torch.float32, "backward_quad_pair_kernel"),
    ((1, 3, 2, 128, 256), torch.float16, "backward_quad_pair_kernel"), ((1, 3, 2, 96, 160), torch.bfloat16, "backward_plane_kernel"),
    ((1, 3, 2, 73, 256), torch.float32, "backward_plane_kernel"), ((1, 3, 2, 72, 254), torch.float32, "backward_plane_kernel")])
def test_kernel_that_serves_a_plane(shape, dtype, kernel):
    m, x, g = _case(shape, True, True, dtype)
    assert kernel in kernels_run(lambda: _grads(m, x, g))
