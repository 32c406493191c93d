// Forward and backward for planes too large to keep in shared memory whole.
//
// Two kernels a pass.  integral_scan.cu writes the integral images of a batch of planes to a workspace,
// rows in the quad layout (bc_quad.cuh).  The gather kernels then work on slabs: R rows of one plane, full
// width.  What a slab of a box filter reads of the integral image is two runs of R + 1 adjacent rows, one on
// either side of the box, each a contiguous piece of memory: two bulk copies per filter bring them to shared
// memory.  A CTA has one stage and up to four warps wherever the plane's width allows; six of them on an SM
// (five in the backward) cover one another's copies.
//
// Against gathering from column bands (32 columns, full height) a slab costs 2 (R+1)/R words of L2 traffic an
// output instead of 2.5, two copy instructions instead of thousands of 16-byte ones, and reads shared
// memory with 5 (R+1)/R words an output instead of 8.
//
// Bound by the shared-memory pipe (77 % in the forward) and the issue slots (67 %); the data comes from L2.
// (8,16,4,256,512): forward 164 -> 86 us, backward 211 -> 121 us against column bands, 113 us with tensor memory.  A training step of
// (8,16,4,128,256) planes on whole-plane kernels takes the same time, so those stay there.
#include "bc_common.cuh"
#include "bc_finish.cuh"
#include "bc_quad.cuh"
#include "bc_tile_io.cuh"
#include "bc_tmem.cuh"

namespace bc {

namespace {

constexpr int kSlabMaxWarps = 16;
constexpr size_t kSlabMaxSmem = 200 * 1024;
constexpr int kStripRows = 8;              // rows per warp

// ---- gathers --------------------------------------------------------------------------------------
// The two runs of integral rows a slab needs for one filter, clamped to the plane.
struct SlabRows {
    int lo_first, lo_count, hi_first, hi_count;
};
__device__ __forceinline__ SlabRows slab_rows(const BoxTaps &t, int p0, int rows, int h)
{
    SlabRows s;
    s.lo_first = min(max(p0 + t.lo_r - 1, 0), h);
    s.lo_count = min(max(p0 + rows - 1 + t.lo_r, 0), h) - s.lo_first + 1;
    s.hi_first = min(max(p0 + t.hi_r, 0), h);
    s.hi_count = min(max(p0 + rows + t.hi_r, 0), h) - s.hi_first + 1;
    return s;
}

struct SlabShape {
    int R, slabs, col_tiles, stage_bytes;      // rows per slab, slabs per plane, 128-column tiles, bytes of one side's stage
};

__device__ __forceinline__ void slab_issue(const float *plane, int pitch, const BoxTaps &t, int p0, int rows, int h, uint32_t lo32,
                                           uint32_t hi32, uint32_t mbar)
{
    const SlabRows s = slab_rows(t, p0, rows, h);
    const uint32_t row_bytes = (uint32_t)pitch * 4u;
    bulk_load(lo32, plane + (int64_t)s.lo_first * pitch, (uint32_t)s.lo_count * row_bytes, mbar);
    bulk_load(hi32, plane + (int64_t)s.hi_first * pitch, (uint32_t)s.hi_count * row_bytes, mbar);
}

// FUSED: the inference steps of `Fusion` (the output may then alias the residual).
template <typename IO, bool VEC, bool FUSED, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 128 ? (FUSED ? 4 : 6) : 1)
forward_slab_kernel(const float *__restrict__ integ, BoxParams bp, IO *out, int C, int F, int h, int w, SlabShape sh, int fsplit,
                    bool normalize, bool exact, Fusion fu)
{
    extern __shared__ __align__(128) unsigned char slab_stage[];
    __shared__ __align__(8) unsigned long long mbar;
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5);
    // (32-bit: a 64-bit division would take what follows out of the uniform registers)
    const int part = blockIdx.x % fsplit, b = blockIdx.x / fsplit;
    const int slab = b % sh.slabs, plane_at = b / sh.slabs, c = plane_at % C;
    const int64_t nc = plane_at;
    const int f_begin = (F * part) / fsplit, f_end = (F * (part + 1)) / fsplit, nf = f_end - f_begin;
    const int cells = quad_cells(w), pitch = 4 * cells, row_bytes = pitch * 4;
    const int p_slab = slab * sh.R, rows = min(sh.R, h - p_slab);
    const uint32_t stage32 = smem_u32(slab_stage), mbar32 = smem_u32(&mbar);
    float *sTaps = reinterpret_cast<float *>(slab_stage + 2 * sh.stage_bytes);      // behind the stages: the boxes
    const float *plane = integ + nc * (int64_t)(h + 1) * pitch;

    if (threadIdx.x == 0) {
        mbar_init(mbar32, 2);
        fence_mbar_init();
    }
    if (FUSED && fu.residual) {      // hints only, while the integral images are still being written
        const int64_t npix = (int64_t)h * w;
        for (int f = f_begin; f < f_end; ++f)
            prefetch_l2(fu.residual + (nc * F + f) * npix + (int64_t)p_slab * w, (size_t)rows * w * sizeof(float));
    }
    grid_dependency_wait();
    if ((int)threadIdx.x < nf) {
        const Box box = load_box(bp, c * F + f_begin + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords, taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        fence_proxy_async();
        slab_issue(plane, pitch, load_taps(sTaps), p_slab, rows, h, stage32, stage32 + sh.stage_bytes, mbar32);
    }

    const int rg = warp / sh.col_tiles, ct = warp - rg * sh.col_tiles;
    const int q0 = ct * 128 + lane * kStrip, p0 = p_slab + rg * kStripRows;
    const int mine = min(kStripRows, p_slab + rows - p0);      // rows of this warp (may be <= 0)
    // (lanes past the plane gather too, from clamped columns, and store nothing)
    bool timed_out = false;
    for (int k = 0; k < nf; ++k) {
        const int f = f_begin + k;
        timed_out |= !mbar_wait(mbar32, k & 1);
        const BoxTaps t = load_taps_uniform(sTaps + k * kTapWords);
        if (mine > 0) {
            const SlabRows s = slab_rows(t, p_slab, rows, h);
            const uint32_t lo32 = stage32 - s.lo_first * row_bytes;
            const uint32_t hi32 = stage32 + sh.stage_bytes - s.hi_first * row_bytes;
            const QuadCols cols = quad_cols(t, q0 >> 2, cells, cells);
            const ColW2 cw = col_weights(t);
            const float sfl = t.scale * t.f_lo_r, sfh = t.scale * t.f_hi_r;
            const QuadRowsLater<kStripRows> q = quad_rows_later<kStripRows>(t, p0, h, lo32, hi32, row_bytes, lane);      // ((8,16,4,256,512): 91 -> 88 us)
            float mul = 1.0f, add = 0.0f;
            if (FUSED) {
                if (fu.scale) mul = __ldg(fu.scale + c * F + f);
                if (fu.shift) add = __ldg(fu.shift + c * F + f);
            }
            int64_t off = (nc * F + f) * (int64_t)h * w + (int64_t)p0 * w + q0;
            Rows8 skip;      // all residual rows in flight before the gather
            const float *res = FUSED && fu.residual ? fu.residual + off - q0 : nullptr;
            if (FUSED && res) rows8_load<float, VEC, true>(skip, res, w, q0, mine, lane);
            f2_t prev[kStrip];
            quad_pair(cols, q.lo(0), q.hi(0), cw, prev);
#pragma unroll
            for (int i = 0; i < kStripRows; ++i) {
                if (i < mine) {
                    f2_t cur[kStrip];
                    quad_pair(cols, q.lo(i + 1), q.hi(i + 1), cw, cur);
                    float v[kStrip];
                    quad_forward_row(prev, cur, t.scale, sfl, sfh, v);
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) prev[m] = cur[m];
                    if (FUSED) {
#pragma unroll
                        for (int m = 0; m < kStrip; ++m) v[m] = v[m] * mul + add;
                        if (res) {
                            const float4 e = rows8_get<float, VEC>(skip, res, w, q0, lane, i);
                            v[0] += e.x; v[1] += e.y; v[2] += e.z; v[3] += e.w;
                        }
                        if (fu.output_relu) {
#pragma unroll
                            for (int m = 0; m < kStrip; ++m) v[m] = fmaxf(v[m], 0.0f);
                        }
                    }
                    store_row4<IO, VEC>(out + off - q0, q0, w, v);
                    off += w;
                }
            }
        }
        __syncthreads();      // the stage has been read
        if (threadIdx.x == 0 && k + 1 < nf) {
            fence_proxy_async();
            slab_issue(plane, pitch, load_taps(sTaps + (k + 1) * kTapWords), p_slab, rows, h, stage32, stage32 + sh.stage_bytes, mbar32);
        }
    }
    if (timed_out && lane == 0) atomicAdd(&g_wait_timeouts, 1);
}

// The input values and the grad-input accumulators of a lane's rows wait in tensor memory (bc_tmem.cuh); the five sums
// are reduced per warp and filter, and per CTA at the end.
template <typename IO, bool VEC, bool NEED_PARAMS, bool COUNTED, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 128 ? 5 : 1)
backward_slab_kernel(const IO *__restrict__ x, const float *__restrict__ x_integ, const float *__restrict__ go_integ, BoxParams bp, IO *__restrict__ grad_input,
                     float *__restrict__ partials, int N, int C, int F, int h, int w, SlabShape sh, bool normalize, bool exact,
                     bool write_gin, Finish fin)
{
    extern __shared__ __align__(128) unsigned char slab_stage[];
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ uint32_t tmem_base;
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int slab = blockIdx.x % sh.slabs;
    const int64_t nc = blockIdx.x / sh.slabs;
    const int c = (int)(nc % C), n = (int)(nc / C);
    const int cells = quad_cells(w), pitch = 4 * cells, row_bytes = pitch * 4;
    const int p_slab = slab * sh.R, rows = min(sh.R, h - p_slab);
    const uint32_t stage32 = smem_u32(slab_stage), mbar32 = smem_u32(&mbar);
    float *sTaps = reinterpret_cast<float *>(slab_stage + 2 * sh.stage_bytes);      // behind the stages: the boxes, then
    float *red = sTaps + F * kTapWords;                                             // [F][warps][5] sums
    const int64_t ipl = (int64_t)(h + 1) * pitch;
    const float *planes = go_integ + nc * F * ipl;

    const int rg = warp / sh.col_tiles, ct = warp - rg * sh.col_tiles;
    const int q0 = ct * 128 + lane * kStrip, p0 = p_slab + rg * kStripRows;
    const int mine = min(kStripRows, p_slab + rows - p0);
    // (lanes past the plane gather too, from clamped columns, with x = 0)
    const int64_t pix = nc * (int64_t)h * w + (int64_t)p0 * w + q0;
    const IO *xrow = x + pix - q0;
    Rows8 g;
    if (threadIdx.x == 0) {
        mbar_init(mbar32, 2);
        fence_mbar_init();
    }
    grid_dependency_wait();
    if ((int)threadIdx.x < F) {
        const Box box = load_box(bp, c * F + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    if (NEED_PARAMS && x) rows8_load<IO, VEC>(g, xrow, w, q0, mine, lane);      // in flight meanwhile
    __syncwarp();
    if (warp == nwarps - 1) tmem_alloc(&tmem_base, tmem_columns(nwarps));
    __syncthreads();
    tmem_acquire();
    TmemRows<1> kept(tmem_base, warp);
    if (threadIdx.x == 0) {
        fence_proxy_async();
        slab_issue(planes, pitch, load_taps(sTaps), p_slab, rows, h, stage32, stage32 + sh.stage_bytes, mbar32);
    }

    if (NEED_PARAMS) {
        if (x) {
#pragma unroll
            for (int i = 0; i < kStripRows; ++i) kept.init(i, rows8_get<IO, VEC>(g, xrow, w, q0, lane, i));
        } else {      // the caller has only the input's integral image: its pixels are second differences
            const float *I = x_integ + nc * (int64_t)(h + 1) * (w + 1) + (int64_t)p0 * (w + 1);
            pixels_of_integral(I, w, q0, q0 < w ? mine : 0, [&](int i, const float4 &e) { kept.init(i, e); });
        }
    } else {
#pragma unroll
        for (int i = 0; i < kStripRows; ++i) kept.init(i, make_float4(0.f, 0.f, 0.f, 0.f));
    }
    kept.sync();
    bool timed_out = false;
    for (int f = 0; f < F; ++f) {
        timed_out |= !mbar_wait(mbar32, f & 1);
        float sums[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
        const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
        if (mine > 0) {
            const SlabRows s = slab_rows(t, p_slab, rows, h);
            const uint32_t lo32 = stage32 - s.lo_first * row_bytes;
            const uint32_t hi32 = stage32 + sh.stage_bytes - s.hi_first * row_bytes;
            const QuadCols cols = quad_cols(t, q0 >> 2, cells, cells);
            const QuadRows<kStripRows> q = quad_rows<kStripRows>(t, p0, h, lo32, hi32, row_bytes, lane);
            if (mine == kStripRows)
                quad_backward_strip<kStripRows, NEED_PARAMS, true>(t, cols, q, col_weights(t), kept, sums, mine);
            else
                quad_backward_strip<kStripRows, NEED_PARAMS, false>(t, cols, q, col_weights(t), kept, sums, mine);
            kept.sync();
        }
        if (NEED_PARAMS) {
            const float s = warp_sum5(sums, lane);
            const int slot = sum5_slot(lane);
            if (slot >= 0) red[(f * nwarps + warp) * kNumSums + slot] = s;
        }
        __syncthreads();      // the stage has been read
        if (threadIdx.x == 0 && f + 1 < F) {
            fence_proxy_async();
            slab_issue(planes + (f + 1) * ipl, pitch, load_taps(sTaps + (f + 1) * kTapWords), p_slab, rows, h, stage32,
                       stage32 + sh.stage_bytes, mbar32);
        }
    }
    if (timed_out && lane == 0) atomicAdd(&g_wait_timeouts, 1);

    if (NEED_PARAMS) {
        for (int i = threadIdx.x; i < F * kNumSums; i += blockDim.x) {
            const int f = i / kNumSums, j = i - f * kNumSums;
            float s = 0.0f;
            for (int k = 0; k < nwarps; ++k) s += red[(f * nwarps + k) * kNumSums + j];
            partials[(((int64_t)(c * F + f) * N + n) * sh.slabs + slab) * kNumSums + j] = s;
        }
    }
    if (write_gin && mine > 0) {
        IO *row = grad_input + pix - q0;
#pragma unroll
        for (int i = 0; i < kStripRows; ++i, row += w)
            if (i < mine) {
                const float4 g = kept.grad_input(i);
                float v[kStrip] = {g.x, g.y, g.z, g.w};
                store_row4<IO, VEC>(row, q0, w, v);
            }
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, tmem_columns(nwarps));
    if (COUNTED) finish_if_last(fin, partials, bp, c, C, F, normalize, exact);
}

inline SlabShape slab_shape(int h, int w)
{
    SlabShape s;
    s.col_tiles = (w + 127) / 128;
    const int groups = 4 / s.col_tiles > 1 ? 4 / s.col_tiles : 1;      // about four warps a CTA
    s.R = groups * kStripRows;
    s.slabs = (h + s.R - 1) / s.R;
    s.stage_bytes = ((s.R + 1) * quad_pitch(w) * 4 + 127) & ~127;
    return s;
}
inline int slab_threads(const SlabShape &s) { return 32 * s.col_tiles * (s.R / kStripRows); }
// (the table of boxes and the per-warp sums of up to 32 filters sit behind the stage)
inline size_t slab_smem(const SlabShape &s, int F, bool sums)
{
    return 2 * (size_t)s.stage_bytes + (size_t)F * kTapWords * sizeof(float) +
           (sums ? (size_t)F * (slab_threads(s) / 32) * kNumSums * sizeof(float) : 0);
}

template <typename IO>
int forward_slab_t(const float *integ, const BoxParams &bp, const Fusion *fu, IO *out, int N, int C, int F, int h, int w,
                   bool normalize, bool exact, cudaStream_t s)
{
    const SlabShape sh = slab_shape(h, w);
    const int64_t base = (int64_t)N * C * sh.slabs;
    // one CTA a slab takes all its filters in turn; fewer each when there are not enough CTAs for two on every SM
    int fsplit = 1;
    while (fsplit < F && base * fsplit < 2 * 148) fsplit = fsplit * 2 < F ? fsplit * 2 : F;
    if (base * fsplit > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool vec = w % 4 == 0 && aligned_to(out, Io<IO>::kVecBytes) && (!fu || !fu->residual || aligned_to(fu->residual, 16));
    void (*kern)(const float *, BoxParams, IO *, int, int, int, int, SlabShape, int, bool, bool, Fusion);
    constexpr bool FU = IsFloat<IO>::value;
    constexpr int S = 128, L = 32 * kSlabMaxWarps;
    if (slab_threads(sh) <= S) {
        if (fu) kern = vec ? forward_slab_kernel<IO, true, FU, S> : forward_slab_kernel<IO, false, FU, S>;
        else kern = vec ? forward_slab_kernel<IO, true, false, S> : forward_slab_kernel<IO, false, false, S>;
    } else {
        if (fu) kern = vec ? forward_slab_kernel<IO, true, FU, L> : forward_slab_kernel<IO, false, FU, L>;
        else kern = vec ? forward_slab_kernel<IO, true, false, L> : forward_slab_kernel<IO, false, false, L>;
    }
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kSlabMaxSmem);
    if (st != BC_OK) return st;
    const Fusion none{0, nullptr, nullptr, nullptr, 0};
    {
        LaunchScope scope(KID_FORWARD_SLAB, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)(base * fsplit), slab_threads(sh), slab_smem(sh, (F + fsplit - 1) / fsplit, false), s, integ, bp, out, C,
                                              F, h, w, sh, fsplit, normalize, exact, fu ? *fu : none))
            return cuda_failed(e, "forward_slab");
    }
    return check_launch("forward_slab");
}

template <typename IO>
int backward_slab_t(const IO *x, const float *x_integ, const float *go_integ, const BoxParams &bp, float rep_h, float rep_w, int N, int C, int F, int h,
                    int w, bool normalize, bool exact, int need_mask, IO *grad_input, void *grad_params, int grad_params_kind,
                    float *partials, cudaStream_t s)
{
    const SlabShape sh = slab_shape(h, w);
    const int64_t blocks = (int64_t)N * C * sh.slabs;
    if (blocks > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool need_params = (need_mask & (BC_NEED_ALL & ~BC_NEED_INPUT)) != 0;
    const bool write_gin = (need_mask & BC_NEED_INPUT) != 0;
    const bool vec = w % 4 == 0 && aligned_to(x, Io<IO>::kVecBytes) && (!write_gin || aligned_to(grad_input, Io<IO>::kVecBytes));
    void (*kern)(const IO *, const float *, const float *, BoxParams, IO *, float *, int, int, int, int, int, SlabShape, bool, bool, bool, Finish);
    const Finish fin = finish_here(bp, need_params, blocks, (int64_t)N * C * F * h * w, C, grad_params, grad_params_kind, need_mask, N * sh.slabs, rep_h, rep_w, s);
    auto pick = [&](auto counted) {
        constexpr int S = 128, L = 32 * kSlabMaxWarps;
        constexpr bool K = decltype(counted)::value;
        if (slab_threads(sh) <= S) {
            if (need_params) kern = vec ? backward_slab_kernel<IO, true, true, K, S> : backward_slab_kernel<IO, false, true, K, S>;
            else kern = vec ? backward_slab_kernel<IO, true, false, false, S> : backward_slab_kernel<IO, false, false, false, S>;
        } else {
            if (need_params) kern = vec ? backward_slab_kernel<IO, true, true, K, L> : backward_slab_kernel<IO, false, true, K, L>;
            else kern = vec ? backward_slab_kernel<IO, true, false, false, L> : backward_slab_kernel<IO, false, false, false, L>;
        }
    };
    if (fin.total) pick(Flag<true>{});
    else pick(Flag<false>{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kSlabMaxSmem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_SLAB, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)blocks, slab_threads(sh), slab_smem(sh, F, need_params), s, x, x_integ, go_integ, bp, grad_input,
                                              partials, N, C, F, h, w, sh, normalize, exact, write_gin, fin))
            return cuda_failed(e, "backward_slab");
    }
    st = check_launch("backward_slab");
    if (st != BC_OK || !need_params || fin.total) return st;
    return launch_finish_param_grads<float>(partials, bp, C * F, N * sh.slabs, normalize, exact, rep_h, rep_w, need_mask,
                                            grad_params, s, grad_params_kind);
}

}  // namespace

bool slab_path_fits(int F, int h, int w)
{
    return h >= 1 && w >= 1 && F <= kMaxFilters && (w + 127) / 128 <= kSlabMaxWarps && slab_smem(slab_shape(h, w), F, true) <= kSlabMaxSmem;
}
size_t slab_integral_floats(int64_t planes, int h, int w) { return (size_t)planes * (size_t)(h + 1) * (size_t)quad_pitch(w); }
size_t slab_partials_bytes(int N, int C, int F, int h, int w)
{
    return (size_t)C * F * N * slab_shape(h, w).slabs * kNumSums * sizeof(float);
}

int launch_forward_slab(const float *integ, const BoxParams &bp, const Fusion *fu, void *out, int io_kind, int N, int C, int F,
                        int h, int w, bool normalize, bool exact, cudaStream_t s)
{
    if (io_kind == BC_IO_F16) return forward_slab_t(integ, bp, nullptr, static_cast<__half *>(out), N, C, F, h, w, normalize, exact, s);
    if (io_kind == BC_IO_BF16)
        return forward_slab_t(integ, bp, nullptr, static_cast<__nv_bfloat16 *>(out), N, C, F, h, w, normalize, exact, s);
    return forward_slab_t(integ, bp, fu, static_cast<float *>(out), N, C, F, h, w, normalize, exact, s);
}

int launch_backward_slab(const void *x, const float *x_integ, int io_kind, const float *go_integ, const BoxParams &bp, float rep_h, float rep_w, int N,
                         int C, int F, int h, int w, bool normalize, bool exact, int need_mask, void *grad_input, void *grad_params,
                         int grad_params_kind, float *partials, cudaStream_t s)
{
    if (io_kind == BC_IO_F16)
        return backward_slab_t(static_cast<const __half *>(x), nullptr, go_integ, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact, need_mask,
                               static_cast<__half *>(grad_input), grad_params, grad_params_kind, partials, s);
    if (io_kind == BC_IO_BF16)
        return backward_slab_t(static_cast<const __nv_bfloat16 *>(x), nullptr, go_integ, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact,
                               need_mask, static_cast<__nv_bfloat16 *>(grad_input), grad_params, grad_params_kind, partials, s);
    return backward_slab_t(static_cast<const float *>(x), x_integ, go_integ, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact, need_mask,
                           static_cast<float *>(grad_input), grad_params, grad_params_kind, partials, s);
}

int read_wait_timeouts_slab(int *count) { return read_wait_timeouts_here(count); }

}  // namespace bc
