// The host path between PyTorch and the C ABI (include/boxconv_b200.h): argument checks, output and
// scratch allocation, the autograd node, one call from Python per operation.
//
// A training step of a small block is a handful of kernels of a few microseconds each, so what the host
// does between them is most of its time: the same path in Python (a Python autograd Function whose
// backward has to take the GIL on the engine's thread, ctypes calls, device context managers) took 230 us
// a step where the kernels of a (1, 8, 4, 32, 32) block take 15.  Here the checks, the allocations and the
// autograd node are C++, and the functions are plain CPython fast calls, because converting a dozen
// arguments through a generic binding layer costs as much as launching a kernel.
#include <ATen/TracerMode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <array>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>

#include "../../include/boxconv_b200.h"

namespace {

using at::Tensor;
using Four = std::array<Tensor, 4>;      // x_min, x_max, y_min, y_max
const char *const kParamNames[4] = {"x_min", "x_max", "y_min", "y_max"};

[[noreturn]] void fail(const std::string &text) { throw std::runtime_error(text); }

std::string dtype_name(at::ScalarType t)
{
    switch (t) {
        case at::kFloat: return "torch.float32";
        case at::kDouble: return "torch.float64";
        case at::kHalf: return "torch.float16";
        case at::kBFloat16: return "torch.bfloat16";
        default: return c10::toString(t);
    }
}

bool is_narrow(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }
int io_kind(at::ScalarType t) { return t == at::kHalf ? BC_IO_F16 : (t == at::kBFloat16 ? BC_IO_BF16 : BC_IO_F32); }

void check_status(int status, const char *what)
{
    if (status == BC_OK) return;
    std::string text = std::string(what) + " failed: " + bc_status_string(status);
    if (status == BC_ERR_CUDA && bc_last_cuda_error()[0]) text += std::string(" (") + bc_last_cuda_error() + ")";
    fail(text);
}

// CUDA tensor of float32 or float64, or of exactly `dtype` when that is given.
void require_cuda_float(const Tensor &t, const char *name, at::ScalarType dtype = at::ScalarType::Undefined,
                        bool narrow_too = false)
{
    if (!t.is_cuda())
        fail(std::string("box_convolution: ") + name + " is not a CUDA tensor; this build has no CPU implementation");
    const at::ScalarType have = t.scalar_type();
    if (have != at::kFloat && have != at::kDouble && !(narrow_too && is_narrow(have)))
        fail(std::string("box_convolution: ") + name + " must be float32 or float64, got " + dtype_name(have));
    if (dtype != at::ScalarType::Undefined && have != dtype)
        fail(std::string("box_convolution: ") + name + " is " + dtype_name(have) + " but the call's other tensors are " +
             dtype_name(dtype));
}

Tensor new_tensor(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor &like)
{
    return Tensor(at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt));
}

// Slice `i` of a dense tensor's first dimension as a tensor over the same storage, without the dispatcher and
// view bookkeeping of select() (a microsecond each, four times a backward pass).
Tensor slice_of(const Tensor &packed, int64_t i)
{
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(packed.storage()), packed.key_set(), packed.dtype());
    c10::TensorImpl *impl = t.unsafeGetTensorImpl();
    const auto sizes = packed.sizes().slice(1);
    impl->set_storage_offset(packed.storage_offset() + i * c10::multiply_integers(sizes));
    impl->set_sizes_contiguous(sizes);
    return t;
}

// (the caching allocator hands out blocks aligned to 512 bytes)
Tensor new_workspace(size_t bytes, const Tensor &like)
{
    return new_tensor({(int64_t)(bytes ? bytes : 1)}, at::kByte, like);
}

bc_stream_t current_stream(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

int to_int(int64_t v)
{
    if (v < 0 || v > 0x7fffffffLL) fail("box_convolution: a size does not fit the library");
    return (int)v;
}

struct Sizes {
    int N, C, F, h, w;
};

struct Options {
    double rep_h, rep_w;
    bool normalize, exact;
    Tensor snapshot;         // packed (4, C, F) float32 copy of the parameters, or undefined
    Tensor counters;         // what counters_of() finds the counters in that go with it, or undefined
};

// Checks of the module's forward; the parameters must have the input's dtype.
Sizes check_forward(const Tensor &input, const Four &p)
{
    require_cuda_float(input, "input", at::ScalarType::Undefined, true);
    if (input.dim() != 4) fail("BoxConv2d: input must have 4 dimensions");
    for (int i = 0; i < 4; ++i) {
        if (is_narrow(input.scalar_type()) && p[i].scalar_type() != input.scalar_type() && p[i].numel())
            fail("box_convolution: tensors of one call must share a dtype, got " + dtype_name(input.scalar_type()) + " and " +
                 dtype_name(p[i].scalar_type()));
        require_cuda_float(p[i], kParamNames[i], input.scalar_type(), true);
        if (p[i].device() != input.device()) fail("BoxConv2d: input and parameters are on different devices");
    }
    for (const Tensor &t : p)
        if (t.dim() != 2) fail("BoxConv2d: all parameters must have 2 dimensions");
    for (const Tensor &t : p)
        if (t.size(0) != input.size(1))
            fail("BoxConv2d: all parameters must have as many rows as there are input channels");
    for (const Tensor &t : p)
        if (t.size(1) != p[0].size(1)) fail("BoxConv2d: all parameters must have equal number of columns");
    return {to_int(input.size(0)), to_int(input.size(1)), to_int(p[0].size(1)), to_int(input.size(2)), to_int(input.size(3))};
}

// A packed float32 copy of the parameters, (4, C, F), with C counters behind it in its storage that are zero whenever
// no kernel of its backward pass is running.
Tensor new_snapshot(at::IntArrayRef sizes, const Tensor &like)
{
    const int64_t n = c10::multiply_integers(sizes), rows = sizes.empty() ? 0 : sizes[0];
    Tensor packed = new_tensor({4 * n + rows}, at::kFloat, like);
    std::vector<int64_t> shape{4};
    shape.insert(shape.end(), sizes.begin(), sizes.end());
    packed.unsafeGetTensorImpl()->set_sizes_contiguous(shape);
    return packed;
}
// The counters behind a tensor that new_snapshot() has made (and nobody else), null for an undefined one.
unsigned *counters_of(const Tensor &packed)
{
    return packed.defined() ? reinterpret_cast<unsigned *>(packed.data_ptr<float>() + packed.numel()) : nullptr;
}

// Packed float32 copy of the parameters as they are now, in one launch.
Tensor pack_parameters(const Four &p, const Sizes &s, bc_stream_t stream)
{
    Four q;
    for (int i = 0; i < 4; ++i) q[i] = p[i].contiguous();
    Tensor packed = new_snapshot({s.C, s.F}, p[0]);
    check_status(bc_pack_parameters(q[0].const_data_ptr(), q[1].const_data_ptr(), q[2].const_data_ptr(), q[3].const_data_ptr(),
                                    io_kind(p[0].scalar_type()), s.C * s.F, packed.data_ptr<float>(), counters_of(packed), s.C, stream),
                 "BoxConv2d forward");
    return packed;
}

// The kernels' view of the four parameter arrays: slices of a packed copy, or four tensors.
struct ParamPtrs {
    const float *p[4];
};
ParamPtrs of_packed(const Tensor &packed)
{
    const float *b = packed.const_data_ptr<float>();
    const int64_t n = packed.numel() / 4;
    return {{b, b + n, b + 2 * n, b + 3 * n}};
}

Tensor run_forward(const Tensor &x, const ParamPtrs &q, const Sizes &s, const Options &o, bc_stream_t stream)
{
    Tensor out = new_tensor({s.N, (int64_t)s.C * s.F, s.h, s.w}, x.scalar_type(), x);
    const bool narrow = is_narrow(x.scalar_type());
    Tensor ws;
    const size_t bytes = narrow ? bc_boxconv2d_narrow_workspace(s.N, s.C, s.F, s.h, s.w, 0)
                                : bc_boxconv2d_forward_workspace(s.N, s.C, s.F, s.h, s.w);
    if (bytes) ws = new_workspace(bytes, x);
    if (narrow) {
        check_status(bc_boxconv2d_forward_narrow_all(x.const_data_ptr(), io_kind(x.scalar_type()), q.p[0], q.p[1], q.p[2], q.p[3],
                                                     (float)o.rep_h, (float)o.rep_w, out.data_ptr(), s.N, s.C, s.F, s.h, s.w,
                                                     o.normalize, o.exact, bytes ? ws.data_ptr() : nullptr, bytes, stream),
                     "BoxConv2d forward");
        return out;
    }
    check_status(bc_boxconv2d_forward(x.const_data_ptr<float>(), q.p[0], q.p[1], q.p[2], q.p[3], (float)o.rep_h, (float)o.rep_w,
                                      out.data_ptr<float>(), s.N, s.C, s.F, s.h, s.w, o.normalize, o.exact,
                                      bytes ? ws.data_ptr() : nullptr, bytes, stream),
                 "BoxConv2d forward");
    return out;
}

// ---- the four functions of the extension interface -------------------------------------------
// float16 / bfloat16 tensors are storage types here: widened, computed in float32, rounded back.

Tensor integral_image(const Tensor &input)
{
    if (is_narrow(input.scalar_type())) return integral_image(input.to(at::kFloat)).to(input.scalar_type());
    require_cuda_float(input, "input");
    if (input.dim() < 2) fail("integral image input must have >=2 dimensions");
    const c10::cuda::CUDAGuard guard(input.device());
    const Tensor x = input.contiguous();
    auto sizes = x.sizes().vec();
    const int64_t h = sizes[sizes.size() - 2], w = sizes[sizes.size() - 1];
    sizes[sizes.size() - 2] = h + 1;
    sizes[sizes.size() - 1] = w + 1;
    Tensor out = new_tensor(sizes, x.scalar_type(), x);
    const int64_t planes = out.numel() / ((h + 1) * (w + 1));
    const bc_stream_t stream = current_stream(x);
    if (x.scalar_type() == at::kDouble)
        check_status(bc_integral_image_f64(x.const_data_ptr<double>(), out.data_ptr<double>(), planes, to_int(h), to_int(w), stream),
                     "integral_image");
    else
        check_status(bc_integral_image(x.const_data_ptr<float>(), out.data_ptr<float>(), planes, to_int(h), to_int(w), stream),
                     "integral_image");
    return out;
}

void check_four(Four &p, int64_t in_planes, const char *prefix, at::ScalarType dtype)
{
    for (int i = 0; i < 4; ++i) require_cuda_float(p[i], kParamNames[i], dtype);
    for (const Tensor &t : p)
        if (t.dim() != 2) fail(std::string(prefix) + "all parameters must have 2 dimensions");
    for (const Tensor &t : p)
        if (t.size(0) != in_planes)
            fail(std::string(prefix) + "all parameters must have as many rows as there are input channels");
    for (const Tensor &t : p)
        if (t.size(1) != p[0].size(1)) fail(std::string(prefix) + "all parameters must have equal number of columns");
    for (Tensor &t : p) t = t.contiguous();
}

// One dtype for all tensors of a narrow call; returns float32 copies.
Tensor widened(const Tensor &t, at::ScalarType narrow)
{
    if (!t.numel()) return t;
    if (t.scalar_type() != narrow)
        fail("box_convolution: tensors of one call must share a dtype, got " + dtype_name(narrow) + " and " +
             dtype_name(t.scalar_type()));
    return t.to(at::kFloat);
}

Tensor box_forward(const Tensor &integrated, Four p, bool normalize, bool exact)
{
    const at::ScalarType dtype = integrated.scalar_type();
    if (is_narrow(dtype)) {
        const Tensor wide = widened(integrated, dtype);
        for (Tensor &t : p) t = widened(t, dtype);
        return box_forward(wide, p, normalize, exact).to(dtype);
    }
    require_cuda_float(integrated, "input_integrated");
    if (integrated.device() != p[0].device()) fail("BoxConv2d: input and parameters are on different devices");
    const c10::cuda::CUDAGuard guard(integrated.device());
    const Tensor I = integrated.contiguous();
    if (I.dim() != 4) fail("BoxConv2d: input must have 4 dimensions");
    check_four(p, I.size(1), "BoxConv2d: ", dtype);
    const Sizes s{to_int(I.size(0)), to_int(I.size(1)), to_int(p[0].size(1)), to_int(I.size(2) - 1), to_int(I.size(3) - 1)};
    Tensor out = new_tensor({s.N, (int64_t)s.C * s.F, s.h, s.w}, dtype, I);
    const bc_stream_t stream = current_stream(I);
    if (dtype == at::kDouble)
        check_status(bc_box_convolution_forward_f64(I.const_data_ptr<double>(), p[0].const_data_ptr<double>(), p[1].const_data_ptr<double>(),
                                                    p[2].const_data_ptr<double>(), p[3].const_data_ptr<double>(), out.data_ptr<double>(),
                                                    s.N, s.C, s.F, s.h, s.w, normalize, exact, stream),
                     "box_convolution_forward");
    else
        check_status(bc_box_convolution_forward(I.const_data_ptr<float>(), p[0].const_data_ptr<float>(), p[1].const_data_ptr<float>(),
                                                p[2].const_data_ptr<float>(), p[3].const_data_ptr<float>(), out.data_ptr<float>(),
                                                s.N, s.C, s.F, s.h, s.w, normalize, exact, stream),
                     "box_convolution_forward");
    return out;
}

using Gradients = std::array<Tensor, 5>;     // of the input and the four parameters; undefined = not asked for

template <typename T>
int backward_call(const Tensor &I, const Four &p, const Tensor &g, double rep_h, double rep_w, const Sizes &s, bool normalize,
                  bool exact, int mask, void *gin, void *gparams, void *ws, size_t bytes, bc_stream_t stream)
{
    auto fn = [&] {
        if constexpr (std::is_same_v<T, double>) return &bc_box_convolution_backward_f64;
        else return &bc_box_convolution_backward;
    }();
    return fn(I.const_data_ptr<T>(), p[0].const_data_ptr<T>(), p[1].const_data_ptr<T>(), p[2].const_data_ptr<T>(),
              p[3].const_data_ptr<T>(), g.const_data_ptr<T>(), nullptr, (T)rep_h, (T)rep_w, s.N, s.C, s.F, s.h, s.w, normalize,
              exact, mask, static_cast<T *>(gin), static_cast<T *>(gparams), ws, bytes, stream);
}

Gradients box_backward(const Tensor &integrated, Four p, const Tensor &grad_output, double rep_h, double rep_w, bool normalize,
                       bool exact, int mask)
{
    const at::ScalarType dtype = integrated.scalar_type();
    if (is_narrow(dtype)) {
        const Tensor wide = widened(integrated, dtype);
        for (Tensor &t : p) t = widened(t, dtype);
        Gradients out = box_backward(wide, p, widened(grad_output, dtype), rep_h, rep_w, normalize, exact, mask);
        for (Tensor &t : out)
            if (t.defined()) t = t.to(dtype);
        return out;
    }
    require_cuda_float(integrated, "input_integrated");
    require_cuda_float(grad_output, "grad_output", dtype);
    const c10::cuda::CUDAGuard guard(integrated.device());
    const Tensor g = grad_output.contiguous(), I = integrated.contiguous();
    if (g.dim() != 4) fail("grad_output for box_convolution must have 4 dimensions");
    if (I.dim() != 4) fail("BoxConv2d: input must have 4 dimensions");
    check_four(p, I.size(1), "", dtype);
    const Sizes s{to_int(I.size(0)), to_int(I.size(1)), to_int(p[0].size(1)), to_int(I.size(2) - 1), to_int(I.size(3) - 1)};
    // the reference checks the height twice and never the width (interface.cpp:157-158); both here
    if (g.size(0) != s.N || g.size(1) != (int64_t)s.C * s.F || g.size(2) != s.h || g.size(3) != s.w)
        fail("box_convolution: sizes of grad_output and input_integrated don't match");
    Gradients out;
    if (!mask) return out;
    Tensor gparams;
    if (mask & BC_NEED_INPUT) out[0] = new_tensor({s.N, s.C, s.h, s.w}, dtype, I);
    if (mask & ~BC_NEED_INPUT) gparams = new_tensor({4, s.C, s.F}, dtype, I);
    const bool f64 = dtype == at::kDouble;
    const size_t bytes = f64 ? bc_box_convolution_backward_workspace_f64(s.N, s.C, s.F, s.h, s.w, mask)
                             : bc_box_convolution_backward_workspace(s.N, s.C, s.F, s.h, s.w, mask);
    Tensor ws = new_workspace(bytes, I);
    void *gin = out[0].defined() ? out[0].data_ptr() : nullptr, *gp = gparams.defined() ? gparams.data_ptr() : nullptr;
    const bc_stream_t stream = current_stream(I);
    check_status(f64 ? backward_call<double>(I, p, g, rep_h, rep_w, s, normalize, exact, mask, gin, gp, ws.data_ptr(), bytes, stream)
                     : backward_call<float>(I, p, g, rep_h, rep_w, s, normalize, exact, mask, gin, gp, ws.data_ptr(), bytes, stream),
                 "box_convolution_backward");
    for (int i = 0; i < 4; ++i)
        if (mask & (BC_NEED_X_MIN << i)) out[1 + i] = slice_of(gparams, i);
    return out;
}

bool all_contiguous(const Four &p)
{
    return p[0].is_contiguous() && p[1].is_contiguous() && p[2].is_contiguous() && p[3].is_contiguous();
}

// In place; `packed` (float32 and narrower): also returns a packed float32 copy of the clipped values (new_snapshot()).
Tensor clip(const Four &p, double rep_h, double rep_w, double max_h, double max_w, bool exact, bool packed)
{
    const at::ScalarType dtype = p[0].scalar_type();
    for (int i = 0; i < 4; ++i) {
        if (is_narrow(dtype) && p[i].scalar_type() != dtype && p[i].numel())
            fail("box_convolution: tensors of one call must share a dtype, got " + dtype_name(dtype) + " and " +
                 dtype_name(p[i].scalar_type()));
        require_cuda_float(p[i], kParamNames[i], dtype, true);
    }
    if (packed && dtype == at::kDouble) fail("box_convolution: a packed copy is made of float32 or narrower parameters only");
    if (is_narrow(dtype) && !packed && !all_contiguous(p)) {
        Four dense;
        for (int i = 0; i < 4; ++i) dense[i] = p[i].contiguous();
        clip(dense, rep_h, rep_w, max_h, max_w, exact, false);
        at::NoGradGuard no_grad;
        for (int i = 0; i < 4; ++i) p[i].copy_(dense[i]);
        return {};
    }
    for (int i = 0; i < 4; ++i)
        if (!p[i].is_contiguous()) fail(std::string(kParamNames[i]) + " must be contiguous");
    for (const Tensor &t : p)
        if (packed ? t.sizes() != p[0].sizes() : t.numel() != p[0].numel()) fail("box_convolution: parameter tensors differ in size");
    const c10::cuda::CUDAGuard guard(p[0].device());
    const bc_stream_t stream = current_stream(p[0]);
    const int count = to_int(p[0].numel());
    void *q[4];
    for (int i = 0; i < 4; ++i) q[i] = p[i].data_ptr();
    int status;
    Tensor out;
    if (dtype == at::kDouble) {
        status = bc_clip_parameters_f64((double *)q[0], (double *)q[1], (double *)q[2], (double *)q[3], count, rep_h, rep_w, max_h,
                                        max_w, exact, stream);
    } else {
        if (packed) out = new_snapshot(p[0].sizes(), p[0]);
        status = bc_clip_parameters_any(q[0], q[1], q[2], q[3], io_kind(dtype), count, rep_h, rep_w, max_h, max_w, exact,
                                        packed ? out.data_ptr<float>() : nullptr, counters_of(out),
                                        packed && count && p[0].dim() ? to_int(p[0].size(0)) : 0, stream);
    }
    check_status(status, "clip_parameters");
    return out;
}

// What was written behind autograd's back counts as a change in place.
void mark_changed(const Tensor &t)
{
    if (!t.is_inference()) t.unsafeGetTensorImpl()->bump_version();
}

// ---- the module's forward and its autograd node ------------------------------------------------
//
// Unlike the reference (box_convolution/box_convolution_function.py:30-65) the node does not keep the
// integral image or the output: the fused entry points work from the input itself, so only the input and
// one packed copy of the parameters live until backward.  The copy matters because the module changes its
// parameters in place (clipping) between a forward and the backward that belongs to it.
// float64 (gradient checks) chains the four functions, as the reference does.  16-bit tensors
// outside what the 16-bit entry points serve (very wide planes, many filters) go through float32 copies.

// The forward of one call.  `keep` receives what backward needs, or is null when nothing will be
// differentiated (then the parameters are read where they are, where the kernels can).
struct Kept {
    Tensor x;                    // the input; its integral image for float64
    Tensor params;               // packed (4, C, F): stored units, float32; pixels for float64
    Tensor counters;             // as in Options
};

Tensor forward_any(const Tensor &input, const Four &p, const Options &o, Kept *keep)
{
    const Sizes s = check_forward(input, p);
    const c10::cuda::CUDAGuard guard(input.device());
    const at::ScalarType dtype = input.scalar_type();
    Tensor x = input.contiguous();
    if (dtype == at::kDouble) {
        Tensor pixels = at::stack({p[0].detach() * o.rep_h, p[1].detach() * o.rep_h, p[2].detach() * o.rep_w, p[3].detach() * o.rep_w});
        const Tensor integrated = integral_image(x);
        if (keep) *keep = {integrated, pixels, Tensor()};
        return box_forward(integrated, {pixels.select(0, 0), pixels.select(0, 1), pixels.select(0, 2), pixels.select(0, 3)},
                           o.normalize, o.exact);
    }
    const bool narrow = is_narrow(dtype);
    if (narrow && s.h && s.w && s.F && !bc_boxconv2d_narrow_all_supported(s.F, s.h, s.w)) x = x.to(at::kFloat);
    const bc_stream_t stream = current_stream(x);
    Tensor packed = o.snapshot, counters = o.counters;
    if (packed.defined() && !(packed.scalar_type() == at::kFloat && packed.device() == x.device() && packed.is_contiguous() &&
                              packed.sizes() == at::IntArrayRef({4, s.C, s.F})))
        packed = Tensor();
    ParamPtrs q;
    Four dense;                  // (keeps contiguous copies alive across the launch)
    if (!packed.defined() && (keep || narrow)) packed = counters = pack_parameters(p, s, stream);
    if (packed.defined()) {
        q = of_packed(packed);
    } else {
        for (int i = 0; i < 4; ++i) {
            dense[i] = p[i].contiguous();
            q.p[i] = dense[i].const_data_ptr<float>();
        }
    }
    Tensor out = run_forward(x, q, s, o, stream);
    if (keep) *keep = {x, packed, counters};
    return out.scalar_type() == dtype ? out : out.to(dtype);
}

Gradients backward_any(const Tensor &x, const Tensor &params, Tensor grad_output, const Options &a, at::ScalarType caller, int mask)
{
    Gradients out;
    if (!mask) return out;
    if (caller == at::kDouble)
        return box_backward(x, {params.select(0, 0), params.select(0, 1), params.select(0, 2), params.select(0, 3)}, grad_output,
                            a.rep_h, a.rep_w, a.normalize, a.exact, mask);
    const c10::cuda::CUDAGuard guard(x.device());
    const Sizes s{(int)x.size(0), (int)x.size(1), (int)params.size(2), (int)x.size(2), (int)x.size(3)};
    const at::ScalarType dtype = x.scalar_type();
    if (is_narrow(caller)) {
        if (grad_output.scalar_type() != dtype) grad_output = grad_output.to(dtype);
    } else {
        require_cuda_float(grad_output, "grad_output", at::kFloat);
    }
    const Tensor g = grad_output.contiguous();
    if (mask & BC_NEED_INPUT) out[0] = new_tensor(x.sizes(), dtype, x);
    const size_t bytes = is_narrow(dtype) ? bc_boxconv2d_narrow_workspace(s.N, s.C, s.F, s.h, s.w, mask)
                                          : bc_boxconv2d_backward_workspace(s.N, s.C, s.F, s.h, s.w, mask);
    // (an allocation of its own for the scratch: the gradients' storage lives, and is saved and sent, as long as they are)
    Tensor gparams, scratch = new_workspace(bytes, x);
    if (mask & ~BC_NEED_INPUT) gparams = new_tensor({4, s.C, s.F}, dtype, x);
    const ParamPtrs q = of_packed(params);
    void *gin = out[0].defined() ? out[0].data_ptr() : nullptr, *gp = gparams.defined() ? gparams.data_ptr() : nullptr;
    const bc_stream_t stream = current_stream(x);
    check_status(bc_boxconv2d_backward_any(x.const_data_ptr(), io_kind(dtype), q.p[0], q.p[1], q.p[2], q.p[3], g.const_data_ptr(),
                                           (float)a.rep_h, (float)a.rep_w, s.N, s.C, s.F, s.h, s.w, a.normalize, a.exact, mask, gin, gp,
                                           scratch.data_ptr(), bytes, counters_of(a.counters), stream),
                 "BoxConv2d backward");
    if (dtype != caller) {
        if (out[0].defined()) out[0] = out[0].to(caller);
        if (gparams.defined()) gparams = gparams.to(caller);
    }
    for (int i = 0; i < 4; ++i)
        if (mask & (BC_NEED_X_MIN << i)) out[1 + i] = slice_of(gparams, i);
    return out;
}

// A plain autograd node: what torch::autograd::Function adds (a dictionary for the saved values, wrapping of the
// outputs) takes longer than launching the kernels.
struct BoxConvolutionBackward : torch::autograd::Node {
    // (hooks on saved tensors see both; the counters stay where they are and so belong to `options`)
    torch::autograd::SavedVariable x, params;
    Options options;
    at::ScalarType caller;       // dtype of the input as the caller passed it
    std::mutex mutex;

    torch::autograd::variable_list apply(torch::autograd::variable_list &&grads) override
    {
        int mask = 0;
        for (int i = 0; i < 5; ++i)
            if (task_should_compute_output(i)) mask |= 1 << i;
        torch::autograd::variable_list list(5);
        if (!mask) return list;
        const at::NoGradGuard no_grad;
        // (a function behind this one that returned nothing: zeros, as torch.autograd.Function has it)
        const Tensor grad = grads[0].defined() ? grads[0] : input_metadata(0).zeros_like();
        Tensor in, packed;
        {
            std::lock_guard<std::mutex> lock(mutex);
            in = x.unpack();      // (checks that the input has not been changed in place and that the graph is still alive)
            packed = params.unpack();
        }
        Gradients g = backward_any(in, packed, grad, options, caller, mask);
        for (int i = 0; i < 5; ++i) list[i] = std::move(g[i]);      // sole owner: a first accumulation takes the tensor itself
        return list;
    }

    void release_variables() override
    {
        std::lock_guard<std::mutex> lock(mutex);
        x.reset_data();
        params.reset_data();
        options.counters.reset();
    }

    std::string name() const override { return "BoxConvolutionFunctionBackward"; }
};

// Calls that the node cannot serve and that go through the Python class, a torch.autograd.Function: a trace records it
// as an operation (this call would leave its result in the trace as a constant), and it refuses tangents of
// forward-mode differentiation and function transforms (which would pass by unseen).
bool needs_python_function(const Tensor &input, const Four &p)
{
    using c10::impl::tls_is_dispatch_key_included;
    if (tls_is_dispatch_key_included(at::DispatchKey::Tracer) ||
        tls_is_dispatch_key_included(at::DispatchKey::FuncTorchDynamicLayerFrontMode))
        return true;
    auto has_tangent = [](const Tensor &t) { return t._fw_grad(/*level=*/0).defined(); };
    return has_tangent(input) || has_tangent(p[0]) || has_tangent(p[1]) || has_tangent(p[2]) || has_tangent(p[3]);
}

Tensor apply(const Tensor &input, const Four &p, const Options &o)
{
    const bool wanted = input.requires_grad() || p[0].requires_grad() || p[1].requires_grad() || p[2].requires_grad() ||
                        p[3].requires_grad();
    if (!wanted || !at::GradMode::is_enabled()) return forward_any(input, p, o, nullptr);
    Kept keep;
    Tensor out;
    {
        const at::NoGradGuard no_grad;
        out = forward_any(input, p, o, &keep);
    }
    auto node = std::shared_ptr<BoxConvolutionBackward>(new BoxConvolutionBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(input, p[0], p[1], p[2], p[3]));
    node->x = torch::autograd::SavedVariable(keep.x, false);
    node->params = torch::autograd::SavedVariable(keep.params, false);
    node->options = o;
    node->options.snapshot = Tensor();      // (node->params holds it)
    node->options.counters = keep.counters;
    node->caller = input.scalar_type();
    torch::autograd::set_history(out, node);
    return out;
}

// ---- inference tail of one box block (inference.py documents the arguments)
Tensor fused_block(const Tensor &input_arg, const Four &p, const Options &o, bool input_relu, const Tensor &scale_arg,
                   const Tensor &shift_arg, const Tensor &residual, bool output_relu, Tensor out, int64_t in_planes)
{
    require_cuda_float(input_arg, "input", at::kFloat);
    if (input_arg.dim() != 4 || input_arg.size(1) != in_planes)
        fail("fused_box_block: input must be (N, " + std::to_string(in_planes) + ", h, w)");
    const Sizes s = check_forward(input_arg, p);
    const c10::cuda::CUDAGuard guard(input_arg.device());
    const Tensor x = input_arg.contiguous();
    const int64_t planes = (int64_t)s.C * s.F;
    auto per_channel = [&](const Tensor &t, const char *name) {
        if (!t.defined()) return t;
        require_cuda_float(t, name, at::kFloat);
        if (t.numel() != planes || t.device() != x.device())
            fail(std::string("fused_box_block: ") + name + " must hold " + std::to_string(planes) + " values on the input's device");
        return t.contiguous();
    };
    const Tensor scale = per_channel(scale_arg, "scale"), shift = per_channel(shift_arg, "shift");
    auto full = [&](const Tensor &t, const char *name) {
        if (!t.defined()) return;
        require_cuda_float(t, name, at::kFloat);
        if (t.sizes() != at::IntArrayRef({s.N, planes, s.h, s.w}) || !t.is_contiguous() || t.device() != x.device())
            fail(std::string("fused_box_block: ") + name + " must be a contiguous (N, " + std::to_string(planes) +
                 ", h, w) tensor on the input's device");
    };
    full(residual, "residual");
    full(out, "out");
    if (!out.defined()) out = new_tensor({s.N, planes, s.h, s.w}, at::kFloat, x);
    Four dense;
    ParamPtrs q;
    for (int i = 0; i < 4; ++i) {
        dense[i] = p[i].contiguous();
        q.p[i] = dense[i].const_data_ptr<float>();
    }
    Tensor ws;
    const size_t bytes = bc_boxconv2d_forward_workspace(s.N, s.C, s.F, s.h, s.w);
    if (bytes) ws = new_workspace(bytes, x);
    auto ptr = [](const Tensor &t) { return t.defined() ? t.const_data_ptr<float>() : nullptr; };
    check_status(bc_boxconv2d_forward_fused(x.const_data_ptr<float>(), q.p[0], q.p[1], q.p[2], q.p[3], (float)o.rep_h,
                                            (float)o.rep_w, out.data_ptr<float>(), s.N, s.C, s.F, s.h, s.w, o.normalize, o.exact,
                                            input_relu, ptr(scale), ptr(shift), ptr(residual), output_relu,
                                            bytes ? ws.data_ptr() : nullptr, bytes, current_stream(x)),
                 "bc_boxconv2d_forward_fused");
    return out;
}

// ---- CPython entry points ---------------------------------------------------------------------
// Positional arguments only; the Python modules of the package give them names and documentation.

struct Args {
    PyObject *const *v;
    Py_ssize_t n, at = 0;
    Args(PyObject *const *v_, Py_ssize_t n_, Py_ssize_t wanted) : v(v_), n(n_)
    {
        TORCH_CHECK_TYPE(n == wanted, "wrong number of arguments");
    }
    Tensor tensor(const char *name)
    {
        PyObject *o = v[at++];
        TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a tensor");
        return THPVariable_Unpack(o);
    }
    Tensor optional_tensor(const char *name)
    {
        if (v[at] == Py_None) {
            ++at;
            return Tensor();
        }
        return tensor(name);
    }
    Four params()
    {
        Four p;
        for (int i = 0; i < 4; ++i) p[i] = tensor(kParamNames[i]);
        return p;
    }
    double number()
    {
        const double d = PyFloat_AsDouble(v[at++]);
        if (d == -1.0 && PyErr_Occurred()) throw py::error_already_set();
        return d;
    }
    int64_t integer()
    {
        const long long i = PyLong_AsLongLong(v[at++]);
        if (i == -1 && PyErr_Occurred()) throw py::error_already_set();
        return i;
    }
    bool flag()
    {
        const int b = PyObject_IsTrue(v[at++]);
        if (b < 0) throw py::error_already_set();
        return b != 0;
    }
};

PyObject *wrap(const Tensor &t)
{
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}

// module_forward(input, x_min, x_max, y_min, y_max, rep_h, rep_w, normalize, exact, clip, max_h, max_w)
//   -> NotImplemented, with nothing done, where the Python class has to be called
PyObject *py_module_forward(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 12);
    const Tensor input = a.tensor("input");
    const Four p = a.params();
    Options o{a.number(), a.number(), a.flag(), a.flag(), Tensor()};
    const bool clipping = a.flag();
    const double max_h = a.number(), max_w = a.number();
    if (needs_python_function(input, p)) Py_RETURN_NOTIMPLEMENTED;
    Tensor out;
    {
        py::gil_scoped_release release;
        // the launch that clips also leaves the copy of the parameters that backward will use
        if (clipping) {
            const at::ScalarType dtype = p[0].scalar_type();
            if (is_narrow(dtype) && !all_contiguous(p)) {
                // (clipped in copies and written back, without counting as a change to the parameters in place)
                clip({p[0].variable_data(), p[1].variable_data(), p[2].variable_data(), p[3].variable_data()}, o.rep_h, o.rep_w,
                     max_h, max_w, o.exact, false);
            } else {
                o.snapshot = o.counters = clip(p, o.rep_h, o.rep_w, max_h, max_w, o.exact, dtype != at::kDouble);
            }
        }
        out = apply(input, p, o);
    }
    return wrap(out);
    END_HANDLE_TH_ERRORS
}

// apply(input, x_min, x_max, y_min, y_max, rep_h, rep_w, normalize, exact, snapshot or None) -> output or NotImplemented
PyObject *py_apply(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 10);
    const Tensor input = a.tensor("input");
    const Four p = a.params();
    Options o{a.number(), a.number(), a.flag(), a.flag(), Tensor()};
    o.snapshot = a.optional_tensor("snapshot");
    if (needs_python_function(input, p)) Py_RETURN_NOTIMPLEMENTED;
    Tensor out;
    {
        py::gil_scoped_release release;
        out = apply(input, p, o);
    }
    return wrap(out);
    END_HANDLE_TH_ERRORS
}

// The two halves of the Python class.
// forward_saved(arguments of apply) -> (output, and the two tensors that backward_saved needs)
PyObject *py_forward_saved(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 10);
    const Tensor input = a.tensor("input");
    const Four p = a.params();
    Options o{a.number(), a.number(), a.flag(), a.flag(), Tensor()};
    o.snapshot = a.optional_tensor("snapshot");
    Tensor out;
    Kept keep;
    {
        py::gil_scoped_release release;
        at::NoGradGuard no_grad;
        at::tracer::impl::NoTracerDispatchMode no_tracer;      // (a trace records the function as a whole)
        out = forward_any(input, p, o, &keep);
    }
    if (c10::impl::tls_is_dispatch_key_included(at::DispatchKey::Tracer)) {      // an output whose allocation the trace has seen
        const Tensor seen = at::empty(out.sizes(), out.options());
        at::tracer::impl::NoTracerDispatchMode no_tracer;
        seen.copy_(out);
        out = seen;
    }
    THPObjectPtr list(PyTuple_New(3));
    if (!list) throw python_error();
    PyTuple_SET_ITEM(list.get(), 0, wrap(out));
    PyTuple_SET_ITEM(list.get(), 1, wrap(keep.x));
    PyTuple_SET_ITEM(list.get(), 2, wrap(keep.params));
    return list.release();
    END_HANDLE_TH_ERRORS
}

// backward_saved(the two tensors, grad_output, rep_h, rep_w, normalize, exact, need_mask) -> five gradients or None
PyObject *py_backward_saved(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 8);
    const Tensor x = a.tensor("input"), params = a.tensor("parameters"), g = a.tensor("grad_output");
    const Options o{a.number(), a.number(), a.flag(), a.flag(), Tensor()};
    const int mask = (int)a.integer();
    Gradients out;
    {
        py::gil_scoped_release release;
        at::NoGradGuard no_grad;
        out = backward_any(x, params, g, o, g.scalar_type(), mask);      // (the engine hands over the output's type)
    }
    THPObjectPtr list(PyList_New(5));
    if (!list) throw python_error();
    for (int i = 0; i < 5; ++i) PyList_SET_ITEM(list.get(), i, wrap(out[i]));
    return list.release();
    END_HANDLE_TH_ERRORS
}

PyObject *py_integral_image(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 1);
    const Tensor input = a.tensor("input");
    Tensor out;
    {
        py::gil_scoped_release release;
        at::NoGradGuard no_grad;
        out = integral_image(input);
    }
    return wrap(out);
    END_HANDLE_TH_ERRORS
}

// box_forward(input_integrated, x_min, x_max, y_min, y_max, normalize, exact)
PyObject *py_box_forward(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 7);
    const Tensor integrated = a.tensor("input_integrated");
    const Four p = a.params();
    const bool normalize = a.flag(), exact = a.flag();
    Tensor out;
    {
        py::gil_scoped_release release;
        at::NoGradGuard no_grad;
        out = box_forward(integrated, p, normalize, exact);
    }
    return wrap(out);
    END_HANDLE_TH_ERRORS
}

// box_backward(input_integrated, x_min, x_max, y_min, y_max, grad_output, rep_h, rep_w, normalize, exact, need_mask)
//   -> [grad_input, grad_x_min, grad_x_max, grad_y_min, grad_y_max], an empty CPU tensor where not asked for
PyObject *py_box_backward(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 11);
    const Tensor integrated = a.tensor("input_integrated");
    const Four p = a.params();
    const Tensor g = a.tensor("grad_output");
    const double rep_h = a.number(), rep_w = a.number();
    const bool normalize = a.flag(), exact = a.flag();
    const int mask = (int)a.integer();
    Gradients out;
    {
        py::gil_scoped_release release;
        at::NoGradGuard no_grad;
        out = box_backward(integrated, p, g, rep_h, rep_w, normalize, exact, mask);
        for (Tensor &t : out)
            if (!t.defined()) t = at::empty({0}, at::kFloat);
    }
    THPObjectPtr list(PyList_New(5));
    if (!list) throw python_error();
    for (int i = 0; i < 5; ++i) PyList_SET_ITEM(list.get(), i, wrap(out[i]));
    return list.release();
    END_HANDLE_TH_ERRORS
}

// clip(x_min, x_max, y_min, y_max, rep_h, rep_w, max_h, max_w, exact, packed) -> packed copy or None
PyObject *py_clip(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 10);
    const Four p = a.params();
    const double rep_h = a.number(), rep_w = a.number(), max_h = a.number(), max_w = a.number();
    const bool exact = a.flag(), packed = a.flag();
    Tensor out;
    {
        py::gil_scoped_release release;
        out = clip(p, rep_h, rep_w, max_h, max_w, exact, packed);
        // 16-bit parameters were once copied back by PyTorch, which checks that no saved value has changed; it still can
        if (!packed && is_narrow(p[0].scalar_type()) && all_contiguous(p))
            for (const Tensor &t : p) mark_changed(t);
    }
    return wrap(out);
    END_HANDLE_TH_ERRORS
}

// fused_block(input, x_min, x_max, y_min, y_max, rep_h, rep_w, normalize, exact, input_relu, scale, shift, residual,
//             output_relu, out, in_planes)
PyObject *py_fused_block(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    Args a(v, n, 16);
    const Tensor input = a.tensor("input");
    const Four p = a.params();
    const Options o{a.number(), a.number(), a.flag(), a.flag(), Tensor()};
    const bool input_relu = a.flag();
    const Tensor scale = a.optional_tensor("scale"), shift = a.optional_tensor("shift"), residual = a.optional_tensor("residual");
    const bool output_relu = a.flag();
    const Tensor out = a.optional_tensor("out");
    const int64_t in_planes = a.integer();
    Tensor result;
    {
        py::gil_scoped_release release;
        at::NoGradGuard no_grad;
        result = fused_block(input, p, o, input_relu, scale, shift, residual, output_relu, out, in_planes);
    }
    return wrap(result);
    END_HANDLE_TH_ERRORS
}

#define BC_FAST(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {BC_FAST(module_forward), BC_FAST(apply), BC_FAST(forward_saved), BC_FAST(backward_saved), BC_FAST(integral_image), BC_FAST(box_forward),
                         BC_FAST(box_backward), BC_FAST(clip), BC_FAST(fused_block), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding(void) { return PyModule_Create(&module_def); }
