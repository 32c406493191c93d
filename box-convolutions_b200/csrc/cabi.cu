// The extern "C" surface declared in include/boxconv_b200.h: argument checks, workspace
// carving and dispatch to the kernels.  No allocation, no synchronisation.
#include <stdio.h>
#include <atomic>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>
#include <string.h>

#include "bc_common.cuh"

namespace bc {

static thread_local char g_last_error[256] = "";

int check_launch(const char *what)
{
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return BC_OK;
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
    return BC_ERR_CUDA;
}

int cuda_failed(cudaError_t e, const char *what)
{
    cudaGetLastError();     // clear the sticky copy, if the error left one
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
    return BC_ERR_CUDA;
}

int raise_smem_limit(const void *kernel, int bytes)
{
    struct Done { const void *kernel; int device; };
    static thread_local std::vector<Done> done;
    int device = -1;
    if (cudaError_t e = cudaGetDevice(&device)) return cuda_failed(e, "cudaGetDevice");
    for (const Done &d : done)
        if (d.kernel == kernel && d.device == device) return BC_OK;
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes))
        return cuda_failed(e, "shared memory opt-in");
    try {
        done.push_back({kernel, device});
    } catch (const std::bad_alloc &) {      // (nothing is thrown through a C entry point; the call is made again next time)
    }
    return BC_OK;
}

bool is_capturing(cudaStream_t s)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &status) != cudaSuccess) {
        (void)cudaGetLastError();      // (the legacy stream while another one is captured)
        return false;
    }
    return status != cudaStreamCaptureStatusNone;
}

// ---- launch counter and per-kernel event timing
static std::atomic<uint64_t> g_launches{0};
static std::mutex g_prof_mutex;
static std::atomic<bool> g_prof_on{false};
static int g_prof_used = 0;
struct ProfRecord { int kid; cudaEvent_t a, b; };
static std::vector<ProfRecord> g_prof;

LaunchScope::LaunchScope(int kernel_id, cudaStream_t s) : stream(s), after(nullptr)
{
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (!g_prof_on.load(std::memory_order_acquire)) return;
    cudaEvent_t before;
    {
        // the record table may be grown by bc_profile_start() on another thread: take the two
        // events out under the lock and never touch the table again from this scope
        std::lock_guard<std::mutex> lock(g_prof_mutex);
        if (!g_prof_on.load(std::memory_order_relaxed) || g_prof_used >= (int)g_prof.size()) return;
        ProfRecord &r = g_prof[g_prof_used++];
        r.kid = kernel_id;
        before = r.a;
        after = r.b;
    }
    cudaEventRecord(before, stream);
}

LaunchScope::~LaunchScope()
{
    if (after) cudaEventRecord(after, stream);
}

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

static inline bool sizes_ok(int N, int C, int F, int h, int w)
{
    return N >= 0 && C >= 0 && F >= 0 && h >= 0 && w >= 0 && h < (1 << 24) && w < (1 << 24);
}

static inline bool any_empty(int N, int C, int F, int h, int w)
{
    return N == 0 || C == 0 || F == 0 || h == 0 || w == 0;
}

static inline size_t integral_bytes(int64_t planes, int h, int w)
{
    return align_up((size_t)planes * (size_t)(h + 1) * (size_t)(w + 1) * sizeof(float), 256);
}



static size_t plane_partials_bytes(int N, int C, int F) { return align_up((size_t)C * F * N * kNumSums * sizeof(float), 256); }

// Slabs, for float tensors whose `planes` integral images of a pass are not too few and too large for the kernel that
// makes them?  (16-bit tensors have no other way.)
static bool slabs_suit(int64_t planes, int F, int h, int w) { return slab_path_fits(F, h, w) && !integral_scan_starves(planes, h, w); }

// Backward from the input's integral image on the whole-plane kernels?  (They may hold the plane and slabs be
// faster all the same.)
static bool plane_backward_integ(int64_t planes, int F, int h, int w)
{
    return plane_path_fits_backward(F, h, w) && !(plane_path_prefers_slabs_backward(planes, F, h, w) && slabs_suit(planes * F, F, h, w));
}

// Backward of planes that do not fit in shared memory, by slabs (workspace already checked).
static int backward_slabs(const void *input, const float *x_integ, int io_kind, const void *grad_output, const BoxParams &bp, float rep_h, float rep_w,
                          int N, int C, int F, int h, int w, bool normalize, bool exact, int need_mask, void *grad_input,
                          void *grad_params, int grad_params_kind, void *workspace, cudaStream_t stream)
{
    float *go_integ = static_cast<float *>(workspace);
    float *partials = reinterpret_cast<float *>(static_cast<char *>(workspace) +
                                                align_up(slab_integral_floats((int64_t)N * C * F, h, w) * sizeof(float), 256));
    int st = launch_integral_quad_ordered(grad_output, io_kind, go_integ, (int64_t)N * C * F, h, w, stream);
    if (st != BC_OK) return st;
    return launch_backward_slab(input, x_integ, io_kind, go_integ, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact, need_mask, grad_input,
                                grad_params, grad_params_kind, partials, stream);
}

// ---- the four extension functions, for float and double ------------------------------------
template <typename T>
static size_t integral_bytes_t(int64_t planes, int h, int w)
{
    return align_up((size_t)planes * (size_t)(h + 1) * (size_t)(w + 1) * sizeof(T), 256);
}

template <typename T>
static int integral_image_entry(const T *in, T *out, int64_t planes, int h, int w, cudaStream_t stream)
{
    if (planes < 0 || h < 0 || w < 0 || h >= (1 << 24) || w >= (1 << 24)) return BC_ERR_BAD_SHAPE;
    if (planes == 0) return BC_OK;
    if (!out || (!in && h > 0 && w > 0)) return BC_ERR_NULL_POINTER;
    return launch_integral_image<T>(in, out, planes, h, w, stream);
}

template <typename T>
static int forward_entry(const T *input_integrated, const T *x_min, const T *x_max, const T *y_min,
                         const T *y_max, T *output, int N, int C, int F, int h, int w, int normalize,
                         int exact, cudaStream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    if (any_empty(N, C, F, h, w)) return BC_OK;
    if (!input_integrated || !x_min || !x_max || !y_min || !y_max || !output) return BC_ERR_NULL_POINTER;
    const BoxParamsT<T> bp{x_min, x_max, y_min, y_max, T(1), T(1)};
    if constexpr (std::is_same<T, float>::value) {
        // a plane whose integral image fits in shared memory is gathered from there, if that is faster
        if (plane_path_fits_forward(F, h, w) && !plane_path_prefers_global_forward_integ((int64_t)N * C, F, h, w))
            return launch_forward_plane_integ(input_integrated, bp, output, N, C, F, h, w, normalize != 0, exact != 0, stream);
    }
    return launch_forward_global<T>(input_integrated, bp, output, N, C, F, h, w, normalize != 0, exact != 0, stream);
}

template <typename T>
static size_t backward_workspace_entry(int N, int C, int F, int h, int w, int need_mask)
{
    if (!sizes_ok(N, C, F, h, w) || any_empty(N, C, F, h, w) || !(need_mask & BC_NEED_ALL)) return 0;
    if (std::is_same<T, float>::value) {
        if (plane_backward_integ((int64_t)N * C, F, h, w)) return plane_partials_bytes(N, C, F);
        if (slabs_suit((int64_t)N * C * F, F, h, w))
            return align_up(slab_integral_floats((int64_t)N * C * F, h, w) * sizeof(float), 256) +
                   align_up(slab_partials_bytes(N, C, F, h, w), 256);
    }
    return integral_bytes_t<T>((int64_t)N * C * F, h, w) +
           align_up(backward_partials_bytes(N, C, F, h, w, sizeof(T)), 256);
}

template <typename T>
static int backward_entry(const T *input_integrated, const T *x_min, const T *x_max, const T *y_min,
                          const T *y_max, const T *grad_output, T reparametrization_h,
                          T reparametrization_w, int N, int C, int F, int h, int w, int normalize,
                          int exact, int need_mask, T *grad_input, T *grad_params, void *workspace,
                          size_t workspace_bytes, cudaStream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    need_mask &= BC_NEED_ALL;
    if (!need_mask) return BC_OK;
    const bool need_params = (need_mask & ~BC_NEED_INPUT) != 0;
    if (any_empty(N, C, F, h, w)) {
        // nothing to gather; parameter gradients of an empty batch are zero
        if (need_params && C > 0 && F > 0) {
            if (!grad_params) return BC_ERR_NULL_POINTER;
            for (int j = 0; j < 4; ++j)
                if (need_mask & (BC_NEED_X_MIN << j))
                    if (cudaError_t e = cudaMemsetAsync(grad_params + (size_t)j * C * F, 0, sizeof(T) * C * F, stream))
                        return cuda_failed(e, "memset");
        }
        return BC_OK;
    }
    if (!input_integrated || !x_min || !x_max || !y_min || !y_max || !grad_output) return BC_ERR_NULL_POINTER;
    if ((need_mask & BC_NEED_INPUT) && !grad_input) return BC_ERR_NULL_POINTER;
    if (need_params && !grad_params) return BC_ERR_NULL_POINTER;
    const size_t ib = integral_bytes_t<T>((int64_t)N * C * F, h, w);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) ||
        workspace_bytes < backward_workspace_entry<T>(N, C, F, h, w, need_mask))
        return BC_ERR_WORKSPACE;
    const BoxParamsT<T> bp{x_min, x_max, y_min, y_max, T(1), T(1)};
    if constexpr (std::is_same<T, float>::value) {
        if (plane_backward_integ((int64_t)N * C, F, h, w))
            return launch_backward_plane_integ(input_integrated, grad_output, bp, reparametrization_h, reparametrization_w, N, C, F, h,
                                               w, normalize != 0, exact != 0, need_mask, grad_input, grad_params,
                                               static_cast<float *>(workspace), stream);
        if (slabs_suit((int64_t)N * C * F, F, h, w))
            return backward_slabs(nullptr, input_integrated, BC_IO_F32, grad_output, bp, reparametrization_h, reparametrization_w, N, C,
                                  F, h, w, normalize != 0, exact != 0, need_mask, grad_input, grad_params, BC_IO_F32, workspace, stream);
    }
    T *go_integ = static_cast<T *>(workspace);
    T *partials = reinterpret_cast<T *>(static_cast<char *>(workspace) + ib);

    int st = launch_integral_image<T>(grad_output, go_integ, (int64_t)N * C * F, h, w, stream);
    if (st != BC_OK) return st;
    return launch_backward_global<T>(nullptr, input_integrated, go_integ, bp, reparametrization_h,
                                     reparametrization_w, N, C, F, h, w, normalize != 0, exact != 0,
                                     need_mask, grad_input, grad_params, partials, stream);
}

template <typename T>
static int clip_entry(T *x_min, T *x_max, T *y_min, T *y_max, int count, double reparametrization_h,
                      double reparametrization_w, double max_input_h, double max_input_w, int exact,
                      cudaStream_t stream, T *packed = nullptr)
{
    if (count < 0) return BC_ERR_BAD_SHAPE;
    if (count == 0) return BC_OK;
    if (!x_min || !x_max || !y_min || !y_max) return BC_ERR_NULL_POINTER;
    if (reparametrization_h == 0.0 || reparametrization_w == 0.0) return BC_ERR_BAD_SHAPE;
    return launch_clip<T, T>(x_min, x_max, y_min, y_max, count, reparametrization_h, reparametrization_w,
                          max_input_h, max_input_w, exact != 0, stream, packed);
}

}  // namespace bc

using namespace bc;

extern "C" {

int bc_version(void) { return 100; }

const char *bc_status_string(int status)
{
    switch (status) {
        case BC_OK: return "ok";
        case BC_ERR_NULL_POINTER: return "a required pointer is NULL";
        case BC_ERR_BAD_SHAPE: return "invalid or too large size";
        case BC_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
        case BC_ERR_CUDA: return "CUDA error at kernel launch";
        case BC_ERR_UNSUPPORTED: return "unsupported combination of arguments";
        default: return "unknown status";
    }
}

const char *bc_last_cuda_error(void) { return g_last_error; }

int bc_integral_image(const float *in, float *out, int64_t planes, int h, int w, bc_stream_t stream)
{
    return integral_image_entry<float>(in, out, planes, h, w, stream);
}

int bc_integral_image_f64(const double *in, double *out, int64_t planes, int h, int w, bc_stream_t stream)
{
    return integral_image_entry<double>(in, out, planes, h, w, stream);
}

int bc_box_convolution_forward(const float *input_integrated, const float *x_min,
                               const float *x_max, const float *y_min, const float *y_max,
                               float *output, int N, int C, int F, int h, int w, int normalize,
                               int exact, bc_stream_t stream)
{
    return forward_entry<float>(input_integrated, x_min, x_max, y_min, y_max, output, N, C, F, h, w,
                                normalize, exact, stream);
}

int bc_box_convolution_forward_f64(const double *input_integrated, const double *x_min,
                                   const double *x_max, const double *y_min, const double *y_max,
                                   double *output, int N, int C, int F, int h, int w, int normalize,
                                   int exact, bc_stream_t stream)
{
    return forward_entry<double>(input_integrated, x_min, x_max, y_min, y_max, output, N, C, F, h, w,
                                 normalize, exact, stream);
}

size_t bc_box_convolution_backward_workspace(int N, int C, int F, int h, int w, int need_mask)
{
    return backward_workspace_entry<float>(N, C, F, h, w, need_mask);
}

size_t bc_box_convolution_backward_workspace_f64(int N, int C, int F, int h, int w, int need_mask)
{
    return backward_workspace_entry<double>(N, C, F, h, w, need_mask);
}

int bc_box_convolution_backward(const float *input_integrated, const float *x_min,
                                const float *x_max, const float *y_min, const float *y_max,
                                const float *grad_output, const float *output,
                                float reparametrization_h, float reparametrization_w, int N,
                                int C, int F, int h, int w, int normalize, int exact,
                                int need_mask, float *grad_input, float *grad_params,
                                void *workspace, size_t workspace_bytes, bc_stream_t stream)
{
    (void)output;
    return backward_entry<float>(input_integrated, x_min, x_max, y_min, y_max, grad_output,
                                 reparametrization_h, reparametrization_w, N, C, F, h, w, normalize,
                                 exact, need_mask, grad_input, grad_params, workspace, workspace_bytes,
                                 stream);
}

int bc_box_convolution_backward_f64(const double *input_integrated, const double *x_min,
                                    const double *x_max, const double *y_min, const double *y_max,
                                    const double *grad_output, const double *output,
                                    double reparametrization_h, double reparametrization_w, int N,
                                    int C, int F, int h, int w, int normalize, int exact,
                                    int need_mask, double *grad_input, double *grad_params,
                                    void *workspace, size_t workspace_bytes, bc_stream_t stream)
{
    (void)output;
    return backward_entry<double>(input_integrated, x_min, x_max, y_min, y_max, grad_output,
                                  reparametrization_h, reparametrization_w, N, C, F, h, w, normalize,
                                  exact, need_mask, grad_input, grad_params, workspace, workspace_bytes,
                                  stream);
}

int bc_clip_parameters(float *x_min, float *x_max, float *y_min, float *y_max, int count,
                       double reparametrization_h, double reparametrization_w,
                       double max_input_h, double max_input_w, int exact, bc_stream_t stream)
{
    return clip_entry<float>(x_min, x_max, y_min, y_max, count, reparametrization_h, reparametrization_w,
                             max_input_h, max_input_w, exact, stream);
}

int bc_clip_parameters_packed(float *x_min, float *x_max, float *y_min, float *y_max, int count,
                              double reparametrization_h, double reparametrization_w,
                              double max_input_h, double max_input_w, int exact, float *packed_out,
                              bc_stream_t stream)
{
    if (count > 0 && !packed_out) return BC_ERR_NULL_POINTER;
    return clip_entry<float>(x_min, x_max, y_min, y_max, count, reparametrization_h, reparametrization_w,
                             max_input_h, max_input_w, exact, stream, packed_out);
}

int bc_clip_parameters_f64(double *x_min, double *x_max, double *y_min, double *y_max, int count,
                           double reparametrization_h, double reparametrization_w,
                           double max_input_h, double max_input_w, int exact, bc_stream_t stream)
{
    return clip_entry<double>(x_min, x_max, y_min, y_max, count, reparametrization_h, reparametrization_w,
                              max_input_h, max_input_w, exact, stream);
}

int bc_clip_parameters_any(void *x_min, void *x_max, void *y_min, void *y_max, int io_kind, int count,
                           double reparametrization_h, double reparametrization_w, double max_input_h,
                           double max_input_w, int exact, float *packed_out, unsigned *zeroed, int zeroed_count,
                           bc_stream_t stream)
{
    if (count < 0 || zeroed_count < 0 || zeroed_count > count) return BC_ERR_BAD_SHAPE;
    if (count == 0) return BC_OK;
    if (!x_min || !x_max || !y_min || !y_max) return BC_ERR_NULL_POINTER;
    if (reparametrization_h == 0.0 || reparametrization_w == 0.0) return BC_ERR_BAD_SHAPE;
    return launch_clip_any(x_min, x_max, y_min, y_max, io_kind, count, reparametrization_h, reparametrization_w,
                           max_input_h, max_input_w, exact != 0, stream, packed_out, zeroed, zeroed_count);
}

int bc_pack_parameters(const void *x_min, const void *x_max, const void *y_min, const void *y_max, int io_kind, int count,
                       float *packed_out, unsigned *zeroed, int zeroed_count, bc_stream_t stream)
{
    if (count < 0 || zeroed_count < 0 || zeroed_count > count) return BC_ERR_BAD_SHAPE;
    if (count == 0) return BC_OK;
    if (!x_min || !x_max || !y_min || !y_max || !packed_out) return BC_ERR_NULL_POINTER;
    return launch_pack(x_min, x_max, y_min, y_max, io_kind, count, packed_out, zeroed, zeroed_count, stream);
}

size_t bc_boxconv2d_forward_workspace(int N, int C, int F, int h, int w)
{
    if (!sizes_ok(N, C, F, h, w) || any_empty(N, C, F, h, w)) return 0;
    if (plane_path_fits_forward(F, h, w)) return 0;
    if (slabs_suit((int64_t)N * C, F, h, w)) return align_up(slab_integral_floats((int64_t)N * C, h, w) * sizeof(float), 256);
    if (band_path_fits_forward(h, w)) return align_up(band_integral_floats((int64_t)N * C, h, w) * sizeof(float), 256);
    return integral_bytes((int64_t)N * C, h, w);
}

// Forward of planes that do not fit in shared memory: integral images to the workspace, in the row layout
// of the kernel that gathers from them: slabs up to 2048 columns (32 filters), column bands for wider planes of
// few rows, the general kernel for the rest.
static int forward_from_workspace(const float *input, const BoxParams &bp, const Fusion *fu, float *output, int N,
                                  int C, int F, int h, int w, bool normalize, bool exact, float *integ,
                                  cudaStream_t stream)
{
    const bool relu_in = fu && fu->input_relu;
    if (slabs_suit((int64_t)N * C, F, h, w)) {
        int st = launch_integral_quad(input, BC_IO_F32, integ, (int64_t)N * C, h, w, relu_in, stream);
        if (st != BC_OK) return st;
        return launch_forward_slab(integ, bp, fu, output, BC_IO_F32, N, C, F, h, w, normalize, exact, stream);
    }
    if (band_path_fits_forward(h, w)) {
        int st = launch_integral_image_f32(input, integ, (int64_t)N * C, h, w, relu_in, stream, band_lpad(), band_rpad(w));
        if (st != BC_OK) return st;
        return launch_forward_band(integ, bp, fu, output, N, C, F, h, w, normalize, exact, stream);
    }
    int st = launch_integral_image_f32(input, integ, (int64_t)N * C, h, w, relu_in, stream);
    if (st != BC_OK) return st;
    if (fu) return launch_forward_global_fused(integ, bp, *fu, output, N, C, F, h, w, normalize, exact, stream);
    return launch_forward_global<float>(integ, bp, output, N, C, F, h, w, normalize, exact, stream);
}

int bc_boxconv2d_forward(const float *input, const float *x_min, const float *x_max,
                         const float *y_min, const float *y_max, float reparametrization_h,
                         float reparametrization_w, float *output, int N, int C, int F, int h,
                         int w, int normalize, int exact, void *workspace,
                         size_t workspace_bytes, bc_stream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    if (any_empty(N, C, F, h, w)) return BC_OK;
    if (!input || !x_min || !x_max || !y_min || !y_max || !output) return BC_ERR_NULL_POINTER;
    const BoxParams bp{x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w};
    if (plane_path_fits_forward(F, h, w))
        return launch_forward_plane(input, bp, output, N, C, F, h, w, normalize != 0, exact != 0, stream);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) ||
        workspace_bytes < bc_boxconv2d_forward_workspace(N, C, F, h, w))
        return BC_ERR_WORKSPACE;
    return forward_from_workspace(input, bp, nullptr, output, N, C, F, h, w, normalize != 0, exact != 0,
                                  static_cast<float *>(workspace), stream);
}

int bc_boxconv2d_forward_fused(const float *input, const float *x_min, const float *x_max,
                               const float *y_min, const float *y_max, float reparametrization_h,
                               float reparametrization_w, float *output, int N, int C, int F, int h,
                               int w, int normalize, int exact, int input_relu, const float *out_scale,
                               const float *out_shift, const float *residual, int output_relu,
                               void *workspace, size_t workspace_bytes, bc_stream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    if (any_empty(N, C, F, h, w)) return BC_OK;
    if (!input || !x_min || !x_max || !y_min || !y_max || !output) return BC_ERR_NULL_POINTER;
    const BoxParams bp{x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w};
    const Fusion fu{input_relu != 0, out_scale, out_shift, residual, output_relu != 0};
    if (plane_path_fits_forward(F, h, w))
        return launch_forward_plane_fused(input, bp, fu, output, N, C, F, h, w, normalize != 0, exact != 0, stream);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) ||
        workspace_bytes < bc_boxconv2d_forward_workspace(N, C, F, h, w))
        return BC_ERR_WORKSPACE;
    float *integ = static_cast<float *>(workspace);
    return forward_from_workspace(input, bp, &fu, output, N, C, F, h, w, normalize != 0, exact != 0, integ, stream);
}

static size_t backward_slabs_bytes(int N, int C, int F, int h, int w)
{
    return align_up(slab_integral_floats((int64_t)N * C * F, h, w) * sizeof(float), 256) +
           align_up(slab_partials_bytes(N, C, F, h, w), 256);
}

// Scratch of the float backward pass in at most `limit` bytes, where it has the choice: slabs pad the rows of their
// integral images more than the older kernels for large planes do (one column: 12 floats against 2), which serve
// what then exceeds the limit.
static bool backward_on_slabs(int N, int C, int F, int h, int w, size_t limit)
{
    return slabs_suit((int64_t)N * C * F, F, h, w) && backward_slabs_bytes(N, C, F, h, w) <= limit;
}
static size_t backward_workspace_within(int N, int C, int F, int h, int w, int need_mask, size_t limit)
{
    if (!sizes_ok(N, C, F, h, w) || any_empty(N, C, F, h, w) || !(need_mask & BC_NEED_ALL)) return 0;
    if (plane_path_fits_backward(F, h, w))
        return plane_partials_bytes(N, C, F);
    if (backward_on_slabs(N, C, F, h, w, limit)) return backward_slabs_bytes(N, C, F, h, w);
    if (band_path_fits_backward(F, h, w))
        return align_up(band_integral_floats((int64_t)N * C * F, h, w) * sizeof(float), 256) +
               align_up(band_partials_bytes(N, C, F, w), 256);
    return integral_bytes((int64_t)N * C * F, h, w) + align_up(backward_partials_bytes(N, C, F, h, w), 256);
}

size_t bc_boxconv2d_backward_workspace(int N, int C, int F, int h, int w, int need_mask)
{
    return backward_workspace_within(N, C, F, h, w, need_mask, SIZE_MAX);
}

// limit: as in backward_workspace_within()
static int backward_float(const float *input, const float *x_min, const float *x_max,
                          const float *y_min, const float *y_max, const float *grad_output,
                          float reparametrization_h, float reparametrization_w, int N, int C,
                          int F, int h, int w, int normalize, int exact, int need_mask,
                          float *grad_input, float *grad_params, void *workspace,
                          size_t workspace_bytes, unsigned *counters, bc_stream_t stream, size_t limit = SIZE_MAX)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    need_mask &= BC_NEED_ALL;
    if (!need_mask) return BC_OK;
    const bool need_params = (need_mask & ~BC_NEED_INPUT) != 0;
    if (any_empty(N, C, F, h, w)) {
        if (need_params && C > 0 && F > 0) {
            if (!grad_params) return BC_ERR_NULL_POINTER;
            for (int j = 0; j < 4; ++j)
                if (need_mask & (BC_NEED_X_MIN << j))
                    if (cudaError_t e = cudaMemsetAsync(grad_params + (size_t)j * C * F, 0, sizeof(float) * C * F, stream))
                        return cuda_failed(e, "memset");
        }
        return BC_OK;
    }
    if (!input || !x_min || !x_max || !y_min || !y_max || !grad_output) return BC_ERR_NULL_POINTER;
    if ((need_mask & BC_NEED_INPUT) && !grad_input) return BC_ERR_NULL_POINTER;
    if (need_params && !grad_params) return BC_ERR_NULL_POINTER;
    const BoxParams bp{x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, counters};
    const bool band = band_path_fits_backward(F, h, w);
    const size_t ib = band ? align_up(band_integral_floats((int64_t)N * C * F, h, w) * sizeof(float), 256)
                           : integral_bytes((int64_t)N * C * F, h, w);
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) ||
        workspace_bytes < backward_workspace_within(N, C, F, h, w, need_mask, limit))
        return BC_ERR_WORKSPACE;
    if (plane_path_fits_backward(F, h, w))
        return launch_backward_plane(input, grad_output, bp, reparametrization_h, reparametrization_w, N, C,
                                     F, h, w, normalize != 0, exact != 0, need_mask, grad_input,
                                     grad_params, static_cast<float *>(workspace), stream);
    if (backward_on_slabs(N, C, F, h, w, limit))
        return backward_slabs(input, nullptr, BC_IO_F32, grad_output, bp, reparametrization_h, reparametrization_w, N, C, F, h, w,
                              normalize != 0, exact != 0, need_mask, grad_input, grad_params, BC_IO_F32, workspace, stream);
    float *go_integ = static_cast<float *>(workspace);
    float *partials = reinterpret_cast<float *>(static_cast<char *>(workspace) + ib);
    if (band) {
        int st = launch_integral_image_f32(grad_output, go_integ, (int64_t)N * C * F, h, w, false, stream, band_lpad(),
                                           band_rpad(w));
        if (st != BC_OK) return st;
        return launch_backward_band(input, go_integ, bp, reparametrization_h, reparametrization_w, N, C, F, h, w,
                                    normalize != 0, exact != 0, need_mask, grad_input, grad_params, partials, stream);
    }
    int st = launch_integral_image<float>(grad_output, go_integ, (int64_t)N * C * F, h, w, stream);
    if (st != BC_OK) return st;
    return launch_backward_global<float>(input, nullptr, go_integ, bp, reparametrization_h,
                                  reparametrization_w, N, C, F, h, w, normalize != 0, exact != 0,
                                  need_mask, grad_input, grad_params, partials, stream);
}

int bc_boxconv2d_backward(const float *input, const float *x_min, const float *x_max,
                          const float *y_min, const float *y_max, const float *grad_output,
                          float reparametrization_h, float reparametrization_w, int N, int C,
                          int F, int h, int w, int normalize, int exact, int need_mask,
                          float *grad_input, float *grad_params, void *workspace,
                          size_t workspace_bytes, bc_stream_t stream)
{
    return backward_float(input, x_min, x_max, y_min, y_max, grad_output, reparametrization_h, reparametrization_w, N, C, F, h, w,
                          normalize, exact, need_mask, grad_input, grad_params, workspace, workspace_bytes, nullptr, stream);
}

// ---- float16 / bfloat16 tensors on the shared-memory kernels
int bc_boxconv2d_narrow_supported(int F, int h, int w)
{
    return (F > 0 && h > 0 && w > 0 && plane_path_fits_forward(F, h, w) && plane_path_fits_backward(F, h, w)) ? 1 : 0;
}

int bc_boxconv2d_forward_narrow(const void *input, int io_kind, const float *x_min, const float *x_max,
                                const float *y_min, const float *y_max, float reparametrization_h,
                                float reparametrization_w, void *output, int N, int C, int F, int h,
                                int w, int normalize, int exact, bc_stream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    if (io_kind != BC_IO_F16 && io_kind != BC_IO_BF16) return BC_ERR_UNSUPPORTED;
    if (any_empty(N, C, F, h, w)) return BC_OK;
    if (!input || !x_min || !x_max || !y_min || !y_max || !output) return BC_ERR_NULL_POINTER;
    if (!plane_path_fits_forward(F, h, w)) return BC_ERR_UNSUPPORTED;
    const BoxParams bp{x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w};
    return launch_forward_plane_narrow(input, io_kind, bp, output, N, C, F, h, w, normalize != 0, exact != 0, stream);
}

int bc_boxconv2d_narrow_all_supported(int F, int h, int w)
{
    return (F > 0 && h > 0 && w > 0 && ((plane_path_fits_forward(F, h, w) && plane_path_fits_backward(F, h, w)) || slab_path_fits(F, h, w))) ? 1 : 0;
}

size_t bc_boxconv2d_narrow_workspace(int N, int C, int F, int h, int w, int need_mask)
{
    if (!sizes_ok(N, C, F, h, w) || any_empty(N, C, F, h, w)) return 0;
    if (!(need_mask & BC_NEED_ALL))
        return plane_path_fits_forward(F, h, w) ? 0 : align_up(slab_integral_floats((int64_t)N * C, h, w) * sizeof(float), 256);
    if (plane_path_fits_backward(F, h, w)) return plane_partials_bytes(N, C, F);
    return align_up(slab_integral_floats((int64_t)N * C * F, h, w) * sizeof(float), 256) +
           align_up(slab_partials_bytes(N, C, F, h, w), 256);
}

int bc_boxconv2d_forward_narrow_all(const void *input, int io_kind, const float *x_min, const float *x_max,
                                    const float *y_min, const float *y_max, float reparametrization_h,
                                    float reparametrization_w, void *output, int N, int C, int F, int h,
                                    int w, int normalize, int exact, void *workspace, size_t workspace_bytes,
                                    bc_stream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    if (any_empty(N, C, F, h, w) || plane_path_fits_forward(F, h, w))
        return bc_boxconv2d_forward_narrow(input, io_kind, x_min, x_max, y_min, y_max, reparametrization_h,
                                           reparametrization_w, output, N, C, F, h, w, normalize, exact, stream);
    if (io_kind != BC_IO_F16 && io_kind != BC_IO_BF16) return BC_ERR_UNSUPPORTED;
    if (!input || !x_min || !x_max || !y_min || !y_max || !output) return BC_ERR_NULL_POINTER;
    if (!slab_path_fits(F, h, w)) return BC_ERR_UNSUPPORTED;
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) ||
        workspace_bytes < bc_boxconv2d_narrow_workspace(N, C, F, h, w, 0))
        return BC_ERR_WORKSPACE;
    const BoxParams bp{x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w};
    float *integ = static_cast<float *>(workspace);
    int st = launch_integral_quad(input, io_kind, integ, (int64_t)N * C, h, w, false, stream);
    if (st != BC_OK) return st;
    return launch_forward_slab(integ, bp, nullptr, output, io_kind, N, C, F, h, w, normalize != 0, exact != 0, stream);
}

// grad_params_kind: how the parameter gradients are stored (BC_IO_*)
static int backward_narrow(const void *input, int io_kind, const float *x_min, const float *x_max,
                           const float *y_min, const float *y_max, const void *grad_output,
                           float reparametrization_h, float reparametrization_w, int N, int C,
                           int F, int h, int w, int normalize, int exact, int need_mask,
                           void *grad_input, void *grad_params, int grad_params_kind, void *workspace,
                           size_t workspace_bytes, unsigned *counters, bc_stream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    if (io_kind != BC_IO_F16 && io_kind != BC_IO_BF16) return BC_ERR_UNSUPPORTED;
    need_mask &= BC_NEED_ALL;
    if (!need_mask) return BC_OK;
    const bool need_params = (need_mask & ~BC_NEED_INPUT) != 0;
    if (any_empty(N, C, F, h, w)) {
        if (need_params && C > 0 && F > 0) {
            if (!grad_params) return BC_ERR_NULL_POINTER;
            for (int j = 0; j < 4; ++j)
                if (need_mask & (BC_NEED_X_MIN << j)) {
                    const size_t bytes = (grad_params_kind == BC_IO_F32 ? 4 : 2) * (size_t)C * F;
                    if (cudaError_t e = cudaMemsetAsync(static_cast<char *>(grad_params) + j * bytes, 0, bytes, stream))
                        return cuda_failed(e, "memset");
                }
        }
        return BC_OK;
    }
    if (!input || !x_min || !x_max || !y_min || !y_max || !grad_output) return BC_ERR_NULL_POINTER;
    if ((need_mask & BC_NEED_INPUT) && !grad_input) return BC_ERR_NULL_POINTER;
    if (need_params && !grad_params) return BC_ERR_NULL_POINTER;
    const bool plane = plane_path_fits_backward(F, h, w);
    if (!plane && !slab_path_fits(F, h, w)) return BC_ERR_UNSUPPORTED;
    if (!workspace || (reinterpret_cast<uintptr_t>(workspace) & 255) ||
        workspace_bytes < bc_boxconv2d_narrow_workspace(N, C, F, h, w, need_mask))
        return BC_ERR_WORKSPACE;
    const BoxParams bp{x_min, x_max, y_min, y_max, reparametrization_h, reparametrization_w, counters};
    if (!plane)
        return backward_slabs(input, nullptr, io_kind, grad_output, bp, reparametrization_h, reparametrization_w, N, C, F, h, w,
                              normalize != 0, exact != 0, need_mask, grad_input, grad_params, grad_params_kind, workspace, stream);
    return launch_backward_plane_narrow(input, grad_output, io_kind, bp, reparametrization_h, reparametrization_w, N, C,
                                        F, h, w, normalize != 0, exact != 0, need_mask, grad_input, grad_params,
                                        grad_params_kind, static_cast<float *>(workspace), stream);
}

int bc_boxconv2d_backward_narrow(const void *input, int io_kind, const float *x_min, const float *x_max,
                                 const float *y_min, const float *y_max, const void *grad_output,
                                 float reparametrization_h, float reparametrization_w, int N, int C,
                                 int F, int h, int w, int normalize, int exact, int need_mask,
                                 void *grad_input, float *grad_params, void *workspace,
                                 size_t workspace_bytes, bc_stream_t stream)
{
    return backward_narrow(input, io_kind, x_min, x_max, y_min, y_max, grad_output, reparametrization_h, reparametrization_w,
                           N, C, F, h, w, normalize, exact, need_mask, grad_input, grad_params, BC_IO_F32, workspace,
                           workspace_bytes, nullptr, stream);
}

int bc_boxconv2d_backward_any(const void *input, int io_kind, const float *x_min, const float *x_max,
                              const float *y_min, const float *y_max, const void *grad_output,
                              float reparametrization_h, float reparametrization_w, int N, int C,
                              int F, int h, int w, int normalize, int exact, int need_mask,
                              void *grad_input, void *grad_params, void *workspace,
                              size_t workspace_bytes, unsigned *counters, bc_stream_t stream)
{
    if (io_kind == BC_IO_F32)
        return backward_float(static_cast<const float *>(input), x_min, x_max, y_min, y_max, static_cast<const float *>(grad_output),
                              reparametrization_h, reparametrization_w, N, C, F, h, w, normalize, exact, need_mask,
                              static_cast<float *>(grad_input), static_cast<float *>(grad_params), workspace, workspace_bytes,
                              counters, stream);
    return backward_narrow(input, io_kind, x_min, x_max, y_min, y_max, grad_output, reparametrization_h, reparametrization_w,
                           N, C, F, h, w, normalize, exact, need_mask, grad_input, grad_params, io_kind, workspace,
                           workspace_bytes, counters, stream);
}

// ---- backward pass on the library's own scratch array (see the header for who needs this)
static __device__ __align__(256) unsigned char g_static_scratch[BC_STATIC_SCRATCH_BYTES];

// In host code `g_static_scratch` is only a handle for the runtime; the address kernels can use
// comes from cudaGetSymbolAddress, once per device, with that device current.
static void *static_scratch_address(int *status)
{
    static std::mutex mutex;
    static void *address[64] = {nullptr};
    int device = -1;
    if (cudaError_t e = cudaGetDevice(&device)) {
        *status = cuda_failed(e, "bc_boxconv2d_backward_static: cudaGetDevice");
        return nullptr;
    }
    if (device < 0 || device >= 64) {
        *status = BC_ERR_UNSUPPORTED;
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mutex);
    if (!address[device]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p) {
            *status = cuda_failed(e, "bc_boxconv2d_backward_static: cudaGetSymbolAddress");
            return nullptr;
        }
        address[device] = p;
    }
    *status = BC_OK;
    return address[device];
}

int bc_boxconv2d_backward_static(const float *input, const float *x_min, const float *x_max,
                                 const float *y_min, const float *y_max, const float *grad_output,
                                 float reparametrization_h, float reparametrization_w, int N, int C,
                                 int F, int h, int w, int normalize, int exact, int need_mask,
                                 float *grad_input, float *grad_params, bc_stream_t stream)
{
    if (!sizes_ok(N, C, F, h, w)) return BC_ERR_BAD_SHAPE;
    const size_t need = backward_workspace_within(N, C, F, h, w, need_mask, BC_STATIC_SCRATCH_BYTES);
    if (need > BC_STATIC_SCRATCH_BYTES) {
        snprintf(g_last_error, sizeof(g_last_error),
                 "bc_boxconv2d_backward_static: this problem needs %zu bytes of scratch, the built-in array has %u",
                 need, (unsigned)BC_STATIC_SCRATCH_BYTES);
        return BC_ERR_WORKSPACE;
    }
    int status = BC_OK;
    void *scratch = static_scratch_address(&status);
    if (!scratch) return status;
    return backward_float(input, x_min, x_max, y_min, y_max, grad_output, reparametrization_h, reparametrization_w, N, C, F, h, w,
                          normalize, exact, need_mask, grad_input, grad_params, scratch, BC_STATIC_SCRATCH_BYTES, nullptr, stream,
                          BC_STATIC_SCRATCH_BYTES);
}

uint64_t bc_launch_count(void) { return g_launches.load(); }

int bc_wait_timeouts(int *count)
{
    if (!count) return BC_ERR_NULL_POINTER;
    return read_wait_timeouts(count);
}

int bc_profile_start(int capacity)
{
    if (capacity < 0) return BC_ERR_BAD_SHAPE;
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    while ((int)g_prof.size() < capacity) {
        ProfRecord r{0, nullptr, nullptr};
        cudaError_t e = cudaEventCreate(&r.a);
        if (e == cudaSuccess) e = cudaEventCreate(&r.b);
        if (e != cudaSuccess) return cuda_failed(e, "bc_profile_start");
        g_prof.push_back(r);
    }
    g_prof_used = 0;
    g_prof_on.store(true, std::memory_order_release);
    return BC_OK;
}

int bc_profile_stop(void)
{
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    g_prof_on.store(false, std::memory_order_release);
    return BC_OK;
}

int bc_profile_count(void)
{
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    return g_prof_used;
}

int bc_profile_get(int index, int *kernel_id, float *milliseconds)
{
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    if (index < 0 || index >= g_prof_used || !kernel_id || !milliseconds) return BC_ERR_BAD_SHAPE;
    *kernel_id = g_prof[index].kid;
    // (cudaErrorNotReady until the device has passed both events: synchronise first)
    if (cudaError_t e = cudaEventElapsedTime(milliseconds, g_prof[index].a, g_prof[index].b))
        return cuda_failed(e, "bc_profile_get");
    return BC_OK;
}

const char *bc_kernel_name(int kernel_id)
{
    switch (kernel_id) {
        case KID_INTEGRAL: return "integral_image_kernel";
        case KID_FORWARD_GLOBAL: return "forward_global_kernel";
        case KID_BACKWARD_GLOBAL: return "backward_global_kernel";
        case KID_FINISH_PARAM_GRADS: return "finish_param_grads_kernel";
        case KID_CLIP: return "clip_kernel";
        case KID_FORWARD_PLANE: return "forward_plane_kernel";
        case KID_BACKWARD_PLANE: return "backward_plane_kernel";
        case KID_SUM_CHUNKS: return "sum_chunk_grads_kernel";
        case KID_BACKWARD_BAND: return "backward_band_kernel";
        case KID_INTEGRAL_BANDS: return "integral_band_fixup_kernels";
        case KID_FORWARD_BAND: return "forward_band_kernel";
        case KID_FORWARD_SLAB: return "forward_slab_kernel";
        case KID_BACKWARD_SLAB: return "backward_slab_kernel";
        case KID_FORWARD_QUAD: return "forward_quad_kernel";
        case KID_BACKWARD_QUAD: return "backward_quad_kernel";
        case KID_FORWARD_TMEM: return "forward_tmem_kernel";
        case KID_FORWARD_TMEM_STREAM: return "forward_tmem_stream_kernel";
        case KID_BACKWARD_QUAD_PAIR: return "backward_quad_pair_kernel";
        case KID_BACKWARD_SQUARE: return "backward_square_kernel";
        case KID_FORWARD_FLAT: return "forward_flat_kernel";
        default: return "unknown";
    }
}

}  // extern "C"
