"""``reparametrize`` and the differentiable box convolution, with the reference's call signatures
(``box_convolution/box_convolution_function.py:5-65``).

The autograd node that ordinary calls get is C++ (``csrc/torch_binding.cpp``); calls inside a trace, a function
transform or forward-mode differentiation take the Python class below.  Unlike the reference it does not chain
integral_image -> forward and does not save the integral image or the output for the backward pass:
the fused entry points work from the input itself (integral images live on chip for planes that fit
there) and the term the reference takes from the saved output is recomputed, so only the input and a
packed copy of the parameters are kept alive between forward and backward.

float64 tensors (gradient checks) take the general kernels, chained as the reference chains them.
float16 / bfloat16 tensors of up to 2048 columns and 32 filters are read and written in their 16-bit type
(float arithmetic and integral images, parameter gradients rounded once at the end); wider planes and
more filters go through float copies, and results and gradients are rounded back.
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


class BoxConvolutionFunction(torch.autograd.Function):
    """apply(input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
    normalize, exact) -> output (N, C*F, h, w).  The parameters are the stored ones.

    One optional tenth argument: ``snapshot``, a packed float32 ``(4, C, F)`` copy of the four
    parameter tensors as they are at this call (``ext.clip_parameters_packed`` makes it while
    clipping).  Without it the parameters are copied when something is to be differentiated.

    ``apply`` puts a node of the same name in C++ behind its output where that answers the call alike;
    ``forward`` and ``backward`` serve ``torch.jit.trace``, which records the function as one
    operation, and subclasses.  Like the reference's function it has no forward-mode derivative
    and no rule for function transforms: PyTorch says so when it is asked for one."""

    @staticmethod
    def forward(ctx, input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, normalize, exact,
                snapshot=None):
        output, x, params = _native.forward_saved(
            input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, normalize, exact, snapshot)
        ctx.save_for_backward(x, params)
        ctx.options = (reparametrization_h, reparametrization_w, normalize, exact)
        return output

    @staticmethod
    def backward(ctx, grad_output):
        x, params = ctx.saved_tensors
        mask = sum(1 << i for i, needed in enumerate(ctx.needs_input_grad[:5]) if needed)
        grads = _native.backward_saved(x, params, grad_output, *ctx.options, mask)
        return tuple(grads) + (None,) * (len(ctx.needs_input_grad) - 5)

    @classmethod
    def apply(cls, input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, normalize, exact,
              snapshot=None):
        if cls is BoxConvolutionFunction:
            output = _native.apply(input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
                                   normalize, exact, snapshot)
            if output is not NotImplemented:
                return output
        return super().apply(input, x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
                             normalize, exact, snapshot)
