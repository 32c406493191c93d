// In-place projection of the stored box parameters (src/box_convolution.cpp:729-763,
// src/box_convolution_cuda_misc.cu:190-236): clamp both ends of every (min, max) pair to
// [-(max_size+1), max_size-1] pixels and widen pairs that have become narrower than the minimum
// size around their mean.  Arithmetic in double on the stored (reparametrized) values, like the
// reference.  One launch handles the x pair and the y pair.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "bc_common.cuh"

namespace bc {

namespace {

// Stored type S, arithmetic type T (what the reference rounds the mean to): 16-bit parameters are
// clipped as float32 and rounded when they are stored.
__device__ __forceinline__ float widen(float v) { return v; }
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ void put(float *p, float v) { *p = v; }
__device__ __forceinline__ void put(double *p, double v) { *p = v; }
__device__ __forceinline__ void put(__half *p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ void put(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

template <typename S, typename T>
__device__ __forceinline__ void clip_pair(S *pmin, S *pmax, double inv_rep, double min_size, double max_size)
{
    const double lo = -(max_size + 1) * inv_rep, hi = (max_size - 1) * inv_rep;
    double a = fmax(lo, fmin(hi, (double)widen(*pmin)));
    double b = fmax(lo, fmin(hi, (double)widen(*pmax)));
    if (a + (min_size - 0.9999) * inv_rep > b) {
        const T mean = (T)(0.5 * (a + b));   // rounded to the arithmetic type, as the reference does
        a = mean - 0.5 * (min_size - 0.9999) * inv_rep;
        b = mean + 0.5 * (min_size - 0.9999) * inv_rep;
    }
    put(pmin, (T)a);
    put(pmax, (T)b);
}

// `packed` (may be null): a (4, count) copy of the clipped values in the order x_min, x_max, y_min,
// y_max, written by the same threads: the snapshot of the parameters that a forward pass keeps for
// its backward pass, without a launch of its own.  `zeroed` (may be null): counters that the backward pass needs.
template <typename S, typename T>
__global__ void clip_kernel(S *x_min, S *x_max, S *y_min, S *y_max, int count,
                            double inv_rep_h, double inv_rep_w, double min_size, double max_h, double max_w,
                            T *packed, unsigned *zeroed, int zeroed_count)
{
    grid_dependency_release();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (zeroed && i < zeroed_count) zeroed[i] = 0u;      // (zeroed_count is at most 2 * count)
    if (i < count) {
        clip_pair<S, T>(x_min + i, x_max + i, inv_rep_h, min_size, max_h);
        if (packed) { packed[i] = widen(x_min[i]); packed[count + i] = widen(x_max[i]); }
    } else if (i < 2 * count) {
        const int j = i - count;
        clip_pair<S, T>(y_min + j, y_max + j, inv_rep_w, min_size, max_w);
        if (packed) { packed[2 * count + j] = widen(y_min[j]); packed[3 * count + j] = widen(y_max[j]); }
    }
}

// The copy alone, for calls that clip nothing.
template <typename S>
__global__ void pack_kernel(const S *x_min, const S *x_max, const S *y_min, const S *y_max, int count, float *packed,
                            unsigned *zeroed, int zeroed_count)
{
    grid_dependency_release();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    if (zeroed && i < zeroed_count) zeroed[i] = 0u;      // (at most count)
    packed[i] = widen(x_min[i]);
    packed[count + i] = widen(x_max[i]);
    packed[2 * count + i] = widen(y_min[i]);
    packed[3 * count + i] = widen(y_max[i]);
}

}  // namespace

template <typename S, typename T>
int launch_clip(S *x_min, S *x_max, S *y_min, S *y_max, int count, double rep_h,
                double rep_w, double max_h, double max_w, bool exact, cudaStream_t s, T *packed, unsigned *zeroed, int zeroed_count)
{
    if (count == 0) return BC_OK;
    // minimum sizes are single-precision constants in the reference (interface.cpp:405-406)
    const double min_size = (double)(exact ? 1.001f : 2.001f);
    const int threads = 128;
    const int blocks = (2 * count + threads - 1) / threads;
    {
        LaunchScope scope(KID_CLIP, s);
        clip_kernel<S, T><<<blocks, threads, 0, s>>>(x_min, x_max, y_min, y_max, count, 1.0 / rep_h, 1.0 / rep_w,
                                                     min_size, max_h, max_w, packed, zeroed, zeroed_count);
    }
    return check_launch("clip_parameters");
}

template int launch_clip<float, float>(float *, float *, float *, float *, int, double, double, double, double, bool, cudaStream_t,
                                       float *, unsigned *, int);
template int launch_clip<double, double>(double *, double *, double *, double *, int, double, double, double, double, bool,
                                         cudaStream_t, double *, unsigned *, int);

template <typename S>
static int clip_as(void *x_min, void *x_max, void *y_min, void *y_max, int count, double rep_h, double rep_w, double max_h, double max_w,
                   bool exact, cudaStream_t s, float *packed, unsigned *zeroed, int zeroed_count)
{
    return launch_clip<S, float>(static_cast<S *>(x_min), static_cast<S *>(x_max), static_cast<S *>(y_min), static_cast<S *>(y_max), count,
                                 rep_h, rep_w, max_h, max_w, exact, s, packed, zeroed, zeroed_count);
}

int launch_clip_any(void *x_min, void *x_max, void *y_min, void *y_max, int io_kind, int count, double rep_h, double rep_w,
                    double max_h, double max_w, bool exact, cudaStream_t s, float *packed, unsigned *zeroed, int zeroed_count)
{
    auto fn = io_kind == BC_IO_F32 ? clip_as<float> : io_kind == BC_IO_F16 ? clip_as<__half> : io_kind == BC_IO_BF16 ? clip_as<__nv_bfloat16> : nullptr;
    if (!fn) return BC_ERR_UNSUPPORTED;
    return fn(x_min, x_max, y_min, y_max, count, rep_h, rep_w, max_h, max_w, exact, s, packed, zeroed, zeroed_count);
}

template <typename S>
static void pack_as(const void *x_min, const void *x_max, const void *y_min, const void *y_max, int count, float *packed,
                    unsigned *zeroed, int zeroed_count, cudaStream_t s)
{
    pack_kernel<S><<<(count + 127) / 128, 128, 0, s>>>(static_cast<const S *>(x_min), static_cast<const S *>(x_max),
                                                       static_cast<const S *>(y_min), static_cast<const S *>(y_max), count, packed, zeroed,
                                                       zeroed_count);
}

int launch_pack(const void *x_min, const void *x_max, const void *y_min, const void *y_max, int io_kind, int count, float *packed,
                unsigned *zeroed, int zeroed_count, cudaStream_t s)
{
    if (count == 0) return BC_OK;
    {
        LaunchScope scope(KID_CLIP, s);
        if (io_kind == BC_IO_F32) pack_as<float>(x_min, x_max, y_min, y_max, count, packed, zeroed, zeroed_count, s);
        else if (io_kind == BC_IO_F16) pack_as<__half>(x_min, x_max, y_min, y_max, count, packed, zeroed, zeroed_count, s);
        else if (io_kind == BC_IO_BF16) pack_as<__nv_bfloat16>(x_min, x_max, y_min, y_max, count, packed, zeroed, zeroed_count, s);
        else return BC_ERR_UNSUPPORTED;
    }
    return check_launch("pack_parameters");
}

}  // namespace bc
