"""Inference-only helpers for networks built from box blocks.

``fused_box_block`` runs, in one kernel pass over the data, what the reference's
``BottleneckBoxConv`` does around its ``BoxConv2d`` in eval mode as separate PyTorch operators
(``examples/Cityscapes/models/ENet.py:282-304``, ``examples/Cityscapes/models/ERFNet.py:117-137``):
the ReLU in front of it, the BatchNorm2d after it (folded to a per-channel scale and shift), the
skip connection and the final ReLU.  No gradients flow through it.

``GraphedForward`` replays a captured CUDA graph of any such forward on fixed buffers, which takes
the Python and launch overhead out of single-frame latency (the scenario of the reference's
``examples/Cityscapes/convnet-runtime-benchmark.py``).
"""
import torch

from . import _torch_binding as _native


def fold_batchnorm(bn):
    """(scale, shift) of an eval-mode ``nn.BatchNorm2d``: y = scale * x + shift per channel."""
    with torch.no_grad():
        inv = torch.rsqrt(bn.running_var + bn.eps)
        scale = inv * bn.weight if bn.weight is not None else inv
        shift = -bn.running_mean * scale
        if bn.bias is not None:
            shift = shift + bn.bias
    return scale.float().contiguous(), shift.float().contiguous()


def fused_box_block(module, input, *, input_relu=False, scale=None, shift=None, residual=None,
                    output_relu=False, out=None):
    """out = act(scale * module(act_in(input)) + shift + residual), per output channel.

    module    a ``BoxConv2d`` (its stored parameters are used as they are: call ``module.eval()``
              first so that they have been clipped once, as the reference does);
    scale, shift  tensors of ``in_planes * num_filters`` values or None;
    residual  tensor of the output's shape or None;
    out       where to write (may be ``residual`` for an in-place skip connection, and with one filter also
              ``input``); allocated if None.
    """
    return _native.fused_block(
        input, module.x_min, module.x_max, module.y_min, module.y_max,
        module.reparametrization_h, module.reparametrization_w, module.normalize, module.exact,
        input_relu, scale, shift, residual, output_relu, out, module.in_planes)


class GraphedForward:
    """CUDA graph of ``fn(*inputs)`` on fixed buffers.

    ``g = GraphedForward(fn, example)`` runs ``fn`` a few times on copies of the example inputs,
    captures one more run, and from then on ``g(x)`` copies ``x`` into the captured input buffer,
    replays the graph and returns the captured output tensor (overwritten by the next call).
    ``g.inputs`` / ``g.output`` give the buffers for callers that fill them in place and call
    ``g.replay()`` themselves.  ``fn`` must not allocate differently from run to run and must not
    synchronise; it runs under ``torch.no_grad()``.
    """

    def __init__(self, fn, *example_inputs, warmup=3):
        self.inputs = [t.detach().clone() for t in example_inputs]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side), torch.no_grad():
            for _ in range(max(1, warmup)):
                fn(*self.inputs)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(self.graph):
            self.output = fn(*self.inputs)

    def replay(self):
        self.graph.replay()
        return self.output

    def __call__(self, *inputs):
        for dst, src in zip(self.inputs, inputs):
            dst.copy_(src, non_blocking=True)
        return self.replay()
