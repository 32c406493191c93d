"""The four functions of the reference's compiled module ``box_convolution_cpp_cuda``
(``src/bind.cpp:29-34``), with the same names, argument order and return values, served by the
sm_100a library.  Code written against ``box_convolution_cpp_cuda`` can import this module in
its place.  Tensors must be CUDA float32 or float64 (all arguments of one call in the same type);
there is no CPU implementation.

float16 and bfloat16 tensors are accepted as well, as storage types only: they are widened to float32
on the device, the float32 kernels run, and results are rounded back to the caller's type (the
reference runs its arithmetic in half precision, integral images included; nothing here does).

The work of these functions (checks, allocation, launches) is in ``csrc/torch_binding.cpp``.
"""
import torch

from . import _torch_binding as _native


def integral_image(input):
    """(..., h, w) -> (..., h+1, w+1) zero-padded 2-D prefix sum.
    Mirrors src/integral_image_interface.cpp:8-27."""
    return _native.integral_image(input)


def box_convolution_forward(input_integrated, x_min, x_max, y_min, y_max, normalize, exact):
    """Mirrors src/box_convolution_interface.cpp:13-139.  Parameters are in actual pixels."""
    return _native.box_forward(input_integrated, x_min, x_max, y_min, y_max, normalize, exact)


def box_convolution_backward(
        input_integrated, x_min, x_max, y_min, y_max, grad_output, output,
        reparametrization_h, reparametrization_w, normalize, exact,
        input_needs_grad, x_min_needs_grad, x_max_needs_grad, y_min_needs_grad, y_max_needs_grad):
    """Mirrors src/box_convolution_interface.cpp:141-395: returns
    [grad_input, grad_x_min, grad_x_max, grad_y_min, grad_y_max]; entries not asked for are
    0-element tensors (interface.cpp:182,394).  `output` is accepted and ignored."""
    mask = (bool(input_needs_grad) | bool(x_min_needs_grad) << 1 | bool(x_max_needs_grad) << 2
            | bool(y_min_needs_grad) << 3 | bool(y_max_needs_grad) << 4)
    return _native.box_backward(input_integrated, x_min, x_max, y_min, y_max, grad_output,
                                reparametrization_h, reparametrization_w, normalize, exact, mask)


def clip_parameters(x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
                    max_input_h, max_input_w, exact):
    """In place.  Mirrors src/box_convolution_interface.cpp:397-415."""
    _native.clip(x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, max_input_h, max_input_w,
                 exact, False)


def clip_parameters_packed(x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w,
                           max_input_h, max_input_w, exact):
    """``clip_parameters`` for contiguous float32 CUDA tensors that also returns a packed
    ``(4,) + x_min.shape`` copy of the clipped values, written by the same launch: the parameter
    snapshot that ``BoxConvolutionFunction.apply`` accepts."""
    if isinstance(x_min, torch.Tensor) and x_min.dtype != torch.float32:
        raise RuntimeError("box_convolution: x_min is %s but the call's other tensors are torch.float32" % x_min.dtype)
    return _native.clip(x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, max_input_h, max_input_w,
                        exact, True)
