// From the five partial sums per (plane, filter) to the four parameter gradients.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "bc_common.cuh"

namespace bc {

template <typename T>
__device__ __forceinline__ T lane_sum(T v)
{
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// One warp: the gradients of box k from its `per_box` sets of partial sums, added in a fixed order.
template <typename T>
__device__ __forceinline__ void finish_box(const T *partials, const BoxParamsT<T> &bp, int k, int count, int per_box, bool normalize,
                                           bool exact, T rep_h, T rep_w, int need_mask, void *grad_params, int io_kind, int lane)
{
    const T *src = partials + (int64_t)k * per_box * kNumSums;
    T acc[kNumSums] = {T(0), T(0), T(0), T(0), T(0)};
    for (int i = lane; i < per_box; i += 32) {
#pragma unroll
        for (int j = 0; j < kNumSums; ++j) acc[j] += __ldcg(src + (int64_t)i * kNumSums + j);
    }
#pragma unroll
    for (int j = 0; j < kNumSums; ++j) acc[j] = lane_sum(acc[j]);
    if (lane == 0) {
        const BoxT<T> box = load_box(bp, k);
        const ParamSumsT<T> s = {acc[0], acc[1], acc[2], acc[3], acc[4]};
        T g[4];
        finish_param_grads(s, box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact, rep_h, rep_w, g);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (need_mask & (BC_NEED_X_MIN << j)) {
                const int64_t at = (int64_t)j * count + k;
                if (io_kind == BC_IO_F16) static_cast<__half *>(grad_params)[at] = __float2half_rn((float)g[j]);
                else if (io_kind == BC_IO_BF16) static_cast<__nv_bfloat16 *>(grad_params)[at] = __float2bfloat16_rn((float)g[j]);
                else static_cast<T *>(grad_params)[at] = g[j];
            }
    }
}

// The finishing step inside a backward kernel: the last of the `total` CTAs that work on channel c to get here does it
// for the channel's F boxes, in the same order of additions as the kernel of its own.  It saves a launch, 3 us of
// host time, which is worth it where a step is bound by the host.  Where it is bound by the GPU, the fence that
// every CTA pays for and the registers cost more than the launch ((8,16,4,128,256): 80 + 2.5 us in two launches, 88 in
// one), so kernels have it as a template parameter and launchers ask for it up to kFinishMaxOutputs outputs, and not
// while the stream is captured into a graph: a replay has no host time to save.
template <bool B>
struct Flag { static constexpr bool value = B; };      // (picks a kernel's instantiation)

struct Finish {
    void *grad_params;
    int io_kind, need_mask, per_box;
    float rep_h, rep_w;
    unsigned total;
};
constexpr int64_t kFinishMaxCtas = 4 * 148, kFinishMaxOutputs = 8 << 20;      // (a GPU time of about 45 us a step)

inline Finish finish_here(const BoxParams &bp, bool need_params, int64_t ctas, int64_t outputs, int C, void *grad_params, int io_kind,
                          int need_mask, int per_box, float rep_h, float rep_w, cudaStream_t stream)
{
    const bool here = need_params && bp.counters && ctas <= kFinishMaxCtas && outputs <= kFinishMaxOutputs && !is_capturing(stream);
    return Finish{grad_params, io_kind, need_mask, per_box, rep_h, rep_w, here ? (unsigned)(ctas / C) : 0u};
}

// Called by all threads of a CTA after it has written its partial sums.
__device__ __forceinline__ void finish_if_last(const Finish &fin, const float *partials, const BoxParams &bp, int c, int C, int F,
                                               bool normalize, bool exact)
{
    __shared__ unsigned last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(bp.counters + c, 1u) + 1u == fin.total;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) bp.counters[c] = 0u;      // ready for the next launch
    for (int f = threadIdx.x >> 5; f < F; f += blockDim.x >> 5)
        finish_box<float>(partials, bp, c * F + f, C * F, fin.per_box, normalize, exact, fin.rep_h, fin.rep_w, fin.need_mask,
                          fin.grad_params, fin.io_kind, threadIdx.x & 31);
}

}  // namespace bc
