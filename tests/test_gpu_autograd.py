"""What PyTorch asks of an autograd function besides a gradient: traces, saved-tensor hooks, forward-mode
differentiation, function transforms, gradients that are not there."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bc():
    import box_convolution
    assert torch.cuda.is_available()
    return box_convolution


def _module(bc, dtype=torch.float32, shape=(2, 3, 4, 40, 72)):
    N, C, F, h, w = shape
    torch.manual_seed(3)
    m = bc.BoxConv2d(C, F, h, w).cuda().to(dtype)
    return m, torch.randn(N, C, h, w, device="cuda").to(dtype)


def test_the_function_is_an_autograd_function(bc):
    assert issubclass(bc.BoxConvolutionFunction, torch.autograd.Function)
    m, x = _module(bc)
    assert m(x).grad_fn.name() == "BoxConvolutionFunctionBackward"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
def test_forward_and_backward_of_the_class(bc, dtype):
    """The Python halves against the node that ordinary calls get, bit for bit."""
    class Sub(bc.BoxConvolutionFunction):
        pass

    m, x = _module(bc, dtype)
    m.eval()
    runs = []
    for f in (bc.BoxConvolutionFunction, Sub):
        args = [t.detach().clone().requires_grad_() for t in (x, m.x_min, m.x_max, m.y_min, m.y_max)]
        out = f.apply(*args, m.reparametrization_h, m.reparametrization_w, True, True)
        runs.append([out] + list(torch.autograd.grad(out, args, torch.ones_like(out))))
        args[1].requires_grad_(False)
        out = f.apply(*args, m.reparametrization_h, m.reparametrization_w, True, True)
        runs[-1] += torch.autograd.grad(out, [args[0], args[4]], torch.ones_like(out))
    assert all(a.dtype == b.dtype and torch.equal(a, b) for a, b in zip(*runs))


def test_trace_computes_on_new_inputs(bc):
    m, x = _module(bc)
    m.eval()
    traced = torch.jit.trace(m, x, check_trace=False)
    for other in (x, torch.randn_like(x)):
        assert torch.equal(traced(other), m(other))


def test_forward_mode_is_refused(bc):
    import torch.autograd.forward_ad as fwad
    for training in (True, False):
        m, x = _module(bc)
        m.train(training)
        with fwad.dual_level():
            with pytest.raises((NotImplementedError, RuntimeError), match="forward|jvp"):
                m(fwad.make_dual(x, torch.ones_like(x)))


def test_function_transforms_are_refused(bc):
    m, x = _module(bc)
    m.eval()
    with pytest.raises(RuntimeError):
        torch.func.vmap(m)(torch.stack([x, x]))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: m(t).sum())(x)
    with pytest.raises(RuntimeError):      # nothing of the transform reaches the call
        torch.func.vmap(lambda k: m(x).sum() * k)(torch.ones(2, device="cuda"))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16])
def test_saved_tensor_hooks_see_input_and_parameters(bc, dtype):
    """What they hand back is what the backward pass works on, wherever it has been meanwhile."""
    m, x = _module(bc, dtype)
    x.requires_grad_()
    m(x).sum().backward()
    want = [x.grad] + [p.grad for p in m.parameters()]
    x.grad = None
    m.zero_grad(set_to_none=True)
    sizes = []

    def pack(t):
        sizes.append(tuple(t.shape))
        return t.detach().cpu().clone()

    def unpack(t):      # with other memory behind it
        return torch.cat([t.cuda().reshape(-1), torch.full((64,), 7, device="cuda", dtype=t.dtype)])[:t.numel()].view(t.shape)

    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        y = m(x)
    y.sum().backward()
    assert (4, 3, 4) in sizes and len(sizes) == 2
    assert all(torch.equal(a, b) for a, b in zip([x.grad] + [p.grad for p in m.parameters()], want))
    with torch.autograd.graph.save_on_cpu():
        y = m(x)
    x.grad = None
    y.sum().backward()
    assert torch.equal(x.grad, want[0])


def test_a_snapshot_changed_before_backward_is_noticed(bc):
    m, x = _module(bc)
    snapshot = torch.stack([p.detach() for p in m._parameters4()])
    y = bc.BoxConvolutionFunction.apply(x, *m._parameters4(), m.reparametrization_h, m.reparametrization_w, True, True, snapshot)
    snapshot.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


def test_a_missing_gradient_counts_as_zeros(bc):
    class Nothing(torch.autograd.Function):
        @staticmethod
        def forward(ctx, t):
            return t.clone()

        @staticmethod
        def backward(ctx, g):
            return None

    m, x = _module(bc)
    x.requires_grad_()
    grads = torch.autograd.grad(Nothing.apply(m(x)).sum(), [x] + list(m.parameters()))
    assert all((g == 0).all() for g in grads)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gradients_bring_no_scratch_with_them(bc, dtype):
    """The four parameter gradients share one buffer (which is reduced in one piece over ranks), and nothing else does."""
    m, x = _module(bc, dtype)
    m(x).sum().backward()
    assert {p.grad.untyped_storage().nbytes() for p in m.parameters()} == {4 * m.x_min.numel() * m.x_min.element_size()}
    packed, copied = bc.packed_box_gradient(m)
    assert not copied and torch.equal(packed, torch.stack([p.grad for p in m._parameters4()]))


def test_packed_clip_of_single_numbers(bc):
    """Parameters without dimensions are four numbers."""
    from box_convolution import ext
    p = [torch.tensor(v, device="cuda") for v in (-0.9, 0.9, 0.1, 0.1)]
    q = [t.clone().view(1, 1) for t in p]
    packed = ext.clip_parameters_packed(*p, 8.0, 16.0, 8.0, 16.0, True)
    want = ext.clip_parameters_packed(*q, 8.0, 16.0, 8.0, 16.0, True)
    assert packed.shape == (4,) and torch.equal(packed, want.view(4)) and torch.equal(packed, torch.stack(p))


# 32 x 32 tiles, whole planes in 8 x 128 tiles, slabs
@pytest.mark.parametrize("shape", [(2, 3, 4, 32, 32), (2, 3, 4, 40, 72), (1, 2, 2, 201, 260)])
def test_captured_step_finishes_in_a_launch_of_its_own(bc, shape):
    """Outside a graph small steps finish their parameter gradients in the backward kernel; a replay has the kernel that
    only does this, and the same bits."""
    from box_convolution import _cabi
    m, x = _module(bc, shape=shape)
    go = torch.randn(shape[0], shape[1] * shape[2], *shape[3:], device="cuda")

    def step():
        m.zero_grad(set_to_none=True)
        m(x).backward(go)
        return [p.grad for p in m.parameters()]

    want = [g.clone() for g in step()]
    before = _cabi.lib.bc_launch_count()
    step()
    eager = _cabi.lib.bc_launch_count() - before
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    before = _cabi.lib.bc_launch_count()
    with torch.cuda.graph(graph):
        got = step()
    assert _cabi.lib.bc_launch_count() - before == eager + 1
    for _ in range(2):
        for g in got:
            g.fill_(7)
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
