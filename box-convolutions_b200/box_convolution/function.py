"""``reparametrize`` and the differentiable box convolution, with the reference's call signatures
(``box_convolution/box_convolution_function.py:5-65``).

The autograd node itself is C++ (``csrc/torch_binding.cpp``).  Unlike the reference it does not chain
integral_image -> forward and does not save the integral image or the output for the backward pass:
the fused entry points work from the input itself (integral images live on chip for planes that fit
there) and the term the reference takes from the saved output is recomputed, so only the input and a
packed copy of the parameters are kept alive between forward and backward.

float64 tensors (gradient checks) take the general kernels, chained as the reference chains them.
float16 / bfloat16 tensors: planes that the shared-memory kernels hold are read and written in their
16-bit type by those kernels (float arithmetic on chip, float parameter gradients rounded at the end);
larger planes go through float copies, and results and gradients are rounded back.
"""
import torch

from . import _torch_binding as _native


def reparametrize(x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
                  inplace=False, inverse=False):
    """Scales box parameters between pixel units and the stored, roughly [-1, 1] units.
    ``inverse=True``: stored -> pixels (multiply by the factors); otherwise pixels -> stored.
    Returns four new tensors unless ``inplace``."""
    factor_h = reparametrization_h if inverse else 1 / reparametrization_h
    factor_w = reparametrization_w if inverse else 1 / reparametrization_w
    with torch.no_grad():
        if not inplace:
            return x_min * factor_h, x_max * factor_h, y_min * factor_w, y_max * factor_w
        x_min *= factor_h
        x_max *= factor_h
        y_min *= factor_w
        y_max *= factor_w


class BoxConvolutionFunction:
    """apply(input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
    normalize, exact) -> output (N, C*F, h, w).  The parameters are the stored ones.

    One optional tenth argument: ``snapshot``, a packed float32 ``(4, C, F)`` copy of the four
    parameter tensors as they are at this call (``ext.clip_parameters_packed`` makes it while
    clipping).  Without it the parameters are copied when something is to be differentiated."""

    @staticmethod
    def apply(input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, normalize, exact,
              snapshot=None):
        return _native.apply(input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
                             normalize, exact, snapshot)
