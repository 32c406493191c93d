// Whole-plane kernels for planes of any width: strips dealt out to lanes in one sequence (bc_flat.cuh).
//
// What kernels with fixed tiles lose on such planes is lanes: of a tile of 8 x 128 or 32 x 32 pixels they work on those inside the
// plane.  Here all of them have pixels, and samples of one channel share a CTA where a plane alone would not fill it, so
// that its barriers and latencies are shared too.  The gather is the quad kernels', with row offsets of a lane's own (four
// integer operations a tap row more).
//
// Bound by issue slots: 1820 instructions a strip tile and filter, where the quad backward has 1440 ((1480,1,4,40,128): 85 us, 72).  Against the 32 x 32-tile kernel
// that served these planes, over 310 drawn ones (20 to 280 rows, 24 to 560 columns, 1 to 4000 planes): 0.61 of the time.
#include <type_traits>

#include "bc_cluster.cuh"
#include "bc_common.cuh"
#include "bc_finish.cuh"
#include "bc_flat.cuh"
#include "bc_tmem.cuh"

namespace bc {

namespace {

// A lane's rows of a tile in tensor memory, every filter's contribution rounded before it is added: a sum that starts with it, in a
// CTA that has no other filter, is then the same to the last bit.  (`zero` comes from memory: a product and a sum the compiler
// makes one operation of.)  `to`: where the sums of a filter go.
template <int T>
struct FlatKept : TmemRows<1, T> {
    uint32_t to;
    f2_t zero;
    __device__ __forceinline__ FlatKept(uint32_t cta_base, int warp, int k, uint32_t offset, float nil)
        : TmemRows<1, T>(cta_base, warp, k), to(this->base + offset), zero(pack2(nil, nil)) {}
    __device__ __forceinline__ void add(int i, f2_t g01, f2_t g23, f2_t scale)
    {
        float4 v;
        unpack2(add2(pack2(this->g.x, this->g.y), fma2(g01, scale, zero)), v.x, v.y);
        unpack2(add2(pack2(this->g.z, this->g.w), fma2(g23, scale, zero)), v.z, v.w);
        tmem_store4(to + 8 * i, v);
    }
};

// Backward: as backward_quad_kernel, a CTA for `sh.planes` samples of a channel, T tiles a warp.  Few planes: `sh.split` CTAs, a cluster, take
// some of the filters each and keep every filter's contribution to grad-input by itself (the last one's where the others'
// sums would be); they meet in shared memory, where each CTA adds up an eighth or more of the rows in the order of the filters, to the same bits as one
// CTA alone.  (Tensor memory is given back before the cluster's barrier: a CTA that waits for its neighbours must not hold
// what a neighbour may be waiting for.)
template <typename IO, bool VEC, int T, bool NEED_PARAMS, bool COUNTED>
__global__ void __launch_bounds__(T == 1 ? 768 : 512, 1)
backward_plane_kernel(const IO *__restrict__ x, const float *__restrict__ x_integ, const IO *__restrict__ grad_output, BoxParams bp, IO *__restrict__ grad_input,
                     float *__restrict__ partials, int N, int C, int F, int h, int w, const __grid_constant__ FlatShape sh, bool normalize, bool exact, bool write_gin, Finish fin)
{
    constexpr bool kPacked = T == 1;
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int rank = blockIdx.x % sh.split, b = blockIdx.x / sh.split;
    const int c = b % C, team = b / C, n0 = team * sh.planes, planes = min(sh.planes, N - n0);
    const int f_begin = F * rank / sh.split, f_end = F * (rank + 1) / sh.split;
    const int npix = h * w;
    const FlatSmem s = flat_smem_at<T>(smem4, sh);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));
    float *red = sTaps + F * kTapWords;                                                        // [F][warps][5]
    __shared__ uint32_t tmem_base;

    auto cell_of = [&](int k) { return flat_cell(sh, (warp + k * nwarps) * 32 + lane, planes, h); };
    // the strip's first row in the input (and grad-input), and in filter 0's grad_output
    auto pixel_of = [&](const FlatCell &cell) { return ((int64_t)(n0 + cell.plane) * C + c) * npix + cell.group * kFlatRows * w; };
    auto grad_of = [&](const FlatCell &cell) { return ((int64_t)(n0 + cell.plane) * C + c) * F * npix + cell.group * kFlatRows * w; };
    auto request = [&](int f) {
        for (int g = 0; g < planes; ++g) prefetch_l2(grad_output + (((int64_t)(n0 + g) * C + c) * F + f) * npix, (size_t)npix * sizeof(IO));
    };

    if (f_begin < f_end) request(f_begin);      // (a hint, whatever the kernel in front still does)
    flat_zero_padding(s.image, sh, planes, h);
    grid_dependency_wait();
    __syncwarp();
    if (warp == nwarps - 1) tmem_alloc(&tmem_base, sh.columns);
    if ((int)threadIdx.x < F) {
        const Box box = load_box(bp, c * F + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    __syncthreads();
    tmem_acquire();
    uint32_t packed[T];
    int row_first[T];      // the tile in which the tile's first row begins
#pragma unroll
    for (int k = 0; k < T; ++k) {
        const FlatCell mine = cell_of(k);
        packed[k] = flat_pack(mine);
        row_first[k] = (warp + k * nwarps) * 32 / sh.strips * sh.strips / 32;
        TmemRows<1, T> kept(tmem_base, warp, k);
        if (!NEED_PARAMS) {
#pragma unroll
            for (int i = 0; i < kFlatRows; ++i) kept.init(i, make_float4(0.f, 0.f, 0.f, 0.f));
        } else if (!x) {
            // the caller has only the input's integral image: its pixels are second differences
            const FlatCell &cell = mine;
            const float *I = x_integ + ((int64_t)(n0 + cell.plane) * C + c) * (h + 1) * (w + 1) + cell.group * kFlatRows * (w + 1);
            pixels_of_integral(I, w, cell.strip * 4, cell.rows, [&](int i, const float4 &e) { kept.init(i, e); });
        } else {
            FlatBlock v;
            flat_load<IO, VEC>(v, x + pixel_of(mine), w, mine, lane, sh.strips);
#pragma unroll
            for (int i = 0; i < kFlatRows; ++i) {
                float4 e;
                unpack2(v.a[i], e.x, e.y);
                unpack2(v.b[i], e.z, e.w);
                kept.init(i, e);
            }
        }
        kept.sync();
    }
#pragma unroll 1
    for (int f = f_begin; f < f_end; ++f) {
        {
            FlatBlock v[T];
            float carry[T][kFlatRows];
            uint32_t starts[T];
#pragma unroll
            for (int k = 0; k < T; ++k) {
                const FlatCell cell = flat_unpack(packed[k]);
                flat_load<IO, VEC>(v[k], grad_output + grad_of(cell) + f * (int64_t)npix, w, cell, lane, sh.strips);
                starts[k] = __ballot_sync(0xffffffffu, cell.strip == 0);
            }
            if (f + 1 < f_end) request(f + 1);
#pragma unroll
            for (int k = 0; k < T; ++k) flat_scan<T>(v[k], carry[k], s, warp + k * nwarps, starts[k], sh.spans, warp, nwarps, lane);
            if (sh.spans) __syncthreads();
#pragma unroll
            for (int k = 0; k < T; ++k) flat_publish(v[k], carry[k], s, row_first[k], warp + k * nwarps, starts[k], lane);
            __syncthreads();      // (also: every gather of the previous filter is done)
            if (sh.groups > kFlatTall) {
                flat_sum_above(s, sh);
                __syncthreads();
            }
#pragma unroll
            for (int k = 0; k < T; ++k) flat_put(v[k], flat_unpack(packed[k]), s, sh, warp + k * nwarps, lane);
        }
        __syncthreads();
        const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
        const ColW2 cw = col_weights(t);
        float all[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
            const FlatCell cell = flat_unpack(T == 1 || k == 0 ? packed[0] : packed[T - 1]);
            FlatKept<T> kept(tmem_base, warp, k, sh.split == 1 || f + 1 == f_end ? 0 : (f - f_begin + 1) * flat_slot_columns(T, nwarps),
                             lds<9 * 4>(s.taps + f * kTapWords * 4));
            float sums[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
            const FlatCols cols = flat_cols<false>(t, cell, s.image, sh);
            // Of small CTAs, of which an SM runs several, all warps take the same of the two paths: 1300 instructions each, and with both
            // warps wait for instructions longer than for anything else (2.3 of 8.5 cycles an instruction, (300,4,4,134,33)): cut planes
            // of up to 8 tiles, 148 or more, 0.88 of the time (35 drawn ones), fewer 1.02, of more tiles 1.00 to 1.01.
            if (h % kFlatRows == 0 || ((sh.tiles > 8 || gridDim.x < 148) && __all_sync(0xffffffffu, cell.rows == kFlatRows || cell.rows == 0)))
                quad_backward_strip<kFlatRows, NEED_PARAMS, true, kPacked>(t, cols, flat_rows<false>(t, cell, h, sh), cw, kept, sums, kFlatRows);
            else
                quad_backward_strip<kFlatRows, NEED_PARAMS, true, kPacked, true>(t, cols, flat_rows<true>(t, cell, h, sh), cw, kept, sums, cell.rows);
            __syncwarp();
            kept.sync();
#pragma unroll
            for (int j = 0; j < kNumSums; ++j) all[j] += sums[j];
        }
        if (NEED_PARAMS) {
            const float sum = warp_sum5(all, lane);
            const int slot = sum5_slot(lane);
            if (slot >= 0) red[(f * nwarps + warp) * kNumSums + slot] = sum;
        }
    }
    if (NEED_PARAMS) {
        const int teams = (N + sh.planes - 1) / sh.planes;
        __syncthreads();
        for (int i = threadIdx.x; i < (f_end - f_begin) * kNumSums; i += blockDim.x) {
            const int k = i / kNumSums, j = i - k * kNumSums, f = f_begin + k;
            float sum = 0.0f;
            for (int k = 0; k < nwarps; ++k) sum += red[(f * nwarps + k) * kNumSums + j];
            partials[((int64_t)(c * F + f) * teams + team) * kNumSums + j] = sum;
        }
    }
    const bool together = write_gin && sh.split > 1;
    if (together) {
        __syncthreads();      // the sums have been read, which the rows may lie over
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
#pragma unroll 1
            for (int f = f_begin; f < f_end; ++f) {
                TmemRows<1, T> kept(tmem_base + (f + 1 == f_end ? 0 : (f - f_begin + 1) * flat_slot_columns(T, nwarps)), warp, k);
                const uint32_t at = s.image + (((f - f_begin) * kFlatRows * sh.tiles + warp + k * nwarps) * 32 + lane) * 16;
#pragma unroll
                for (int i = 0; i < kFlatRows; ++i) sts128(at + i * sh.tiles * 512, kept.grad_input(i));
            }
        }
    } else if (write_gin) {
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
            const FlatCell cell = flat_unpack(T == 1 || k == 0 ? packed[0] : packed[T - 1]);
            TmemRows<1, T> kept(tmem_base, warp, k);
            IO *row = grad_input + pixel_of(cell);
#pragma unroll
            for (int i = 0; i < kFlatRows; ++i, row += w) {
                const float4 g = kept.grad_input(i);
                const float v[kStrip] = {g.x, g.y, g.z, g.w};
                if (i < cell.rows) store_row4<IO, VEC>(row, cell.strip * 4, w, v);
                __syncwarp();
            }
        }
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, sh.columns);
    if (together) {
        __syncwarp();
        cluster_sync();
        const int row_begin = kFlatRows * rank / sh.split, row_end = kFlatRows * (rank + 1) / sh.split;
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
            const FlatCell cell = flat_unpack(T == 1 || k == 0 ? packed[0] : packed[T - 1]);
            IO *row = grad_input + pixel_of(cell) + row_begin * w;
            for (int i = row_begin; i < row_end; ++i, row += w) {
                const uint32_t at = s.image + ((i * sh.tiles + warp + k * nwarps) * 32 + lane) * 16;
                float v[kStrip] = {0.f, 0.f, 0.f, 0.f};
                for (int r = 0; r < sh.split; ++r) {
                    const uint32_t there = cluster_map(at, r);
                    for (int j = F * (r + 1) / sh.split - F * r / sh.split - 1, k = 0; k <= j; ++k) {
                        const float4 g = cluster_load4(there + k * kFlatRows * sh.tiles * 512);
                        v[0] += g.x; v[1] += g.y; v[2] += g.z; v[3] += g.w;
                    }
                }
                if (i < cell.rows) store_row4<IO, VEC>(row, cell.strip * 4, w, v);
                __syncwarp();
            }
        }
        cluster_sync();      // nobody leaves while another still reads its rows
    }
    if (COUNTED) finish_if_last(fin, partials, bp, c, C, F, normalize, exact);
}

// Forward: a CTA for `sh.planes` samples of a channel, a part of the filters and of the tiles (`fsplit`, `tsplit`).  It builds all integral images, a
// tile a warp (64 registers: up to 32 warps, or 16 twice an SM), then its warps gather tile by tile and filter by filter.
// A null `x`: `integ` holds the planes' integral images, plain rows of w + 1 floats, which are only copied (INTEG).
// FUSED: the inference steps of `Fusion` (the output may then alias the residual); the planes travel to L2 while the CTA still waits for the
// kernel in front, and all residual rows of a tile are in flight before its gather.
template <typename IO, bool VEC, bool FUSED, bool INTEG, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
forward_flat_kernel(const IO *__restrict__ x, const float *__restrict__ integ, BoxParams bp, IO *out, int N, int C, int F, int h, int w,
                    const __grid_constant__ FlatShape sh, int fsplit, int tsplit, bool tight, bool normalize, bool exact, Fusion fu)
{
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int tpart = blockIdx.x % tsplit, rest = blockIdx.x / tsplit, part = rest % fsplit, b = rest / fsplit;
    const int c = b % C, n0 = b / C * sh.planes, planes = min(sh.planes, N - n0);
    const int f_begin = F * part / fsplit, nf = F * (part + 1) / fsplit - f_begin;
    const int npix = h * w;
    FlatSmem s = flat_smem_at<1>(smem4, sh);
    if (tight) {      // the scans' corners where the images will be, whose padding is written behind them
        s.taps = s.scan;
        s.scan = s.image;
    }
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));
    // tiles that have strips, and this CTA's share of them
    const int have = (sh.cells * planes + 31) / 32, t_begin = have * tpart / tsplit, nt = have * (tpart + 1) / tsplit - t_begin;

    if (!INTEG)      // a hint
        for (int g = 0; g < planes; ++g) prefetch_l2(x + ((int64_t)(n0 + g) * C + c) * npix, (size_t)npix * sizeof(IO));
    if (!tight) flat_zero_padding(s.image, sh, planes, h);
    // registers and shared memory only up to here; now what the kernel in front of this one may have written
    grid_dependency_wait();
    auto boxes = [&]() {
        if ((int)threadIdx.x < nf) {
            const Box box = load_box(bp, c * F + f_begin + threadIdx.x);
            store_taps(sTaps + threadIdx.x * kTapWords, taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
        }
    };
    if constexpr (INTEG) {
        if (tight) flat_zero_padding(s.image, sh, planes, h);
        boxes();
        __syncthreads();      // (the zero padding has been written)
        for (int g = 0; g < planes; ++g) {
            const float *I = integ + ((int64_t)(n0 + g) * C + c) * (h + 1) * (w + 1);
            copy_integral_rows(I, h, w, 4 * sh.strips + 8, warp, nwarps, lane, [&](int a, int col, float e) {
                sts<8>(s.image + g * sh.plane + flat_row_at(a, sh.row, sh.skew) + (col & 3) * sh.sub + (col >> 2) * 4, e);
            });
        }
    } else {
        FlatBlock v;
        float carry[kFlatRows];
        const FlatCell mine = flat_cell(sh, warp * 32 + lane, planes, h);
        flat_load<IO, VEC>(v, x + ((int64_t)(n0 + mine.plane) * C + c) * npix + mine.group * kFlatRows * w, w, mine, lane, sh.strips);
        const uint32_t starts = __ballot_sync(0xffffffffu, mine.strip == 0);
        boxes();
        __syncwarp();
        if (FUSED && fu.input_relu) {
#pragma unroll
            for (int i = 0; i < kFlatRows; ++i) {
                float e0, e1;
                unpack2(v.a[i], e0, e1);
                v.a[i] = pack2(fmaxf(e0, 0.f), fmaxf(e1, 0.f));
                unpack2(v.b[i], e0, e1);
                v.b[i] = pack2(fmaxf(e0, 0.f), fmaxf(e1, 0.f));
            }
        }
        flat_scan<1>(v, carry, s, warp, starts, sh.spans, warp, nwarps, lane);
        if (sh.spans) __syncthreads();
        flat_publish(v, carry, s, warp * 32 / sh.strips * sh.strips / 32, warp, starts, lane);
        __syncthreads();
        if (tight) flat_zero_padding(s.image, sh, planes, h);
        if (sh.groups > kFlatTall) {
            flat_sum_above(s, sh);
            __syncthreads();
        }
        flat_put(v, mine, s, sh, warp, lane);
    }
    __syncthreads();

    FlatCell cell;
    int at = -1;
    for (int task = warp; task < nt * nf; task += nwarps) {
        const int k = task / nt, tile = t_begin + task - k * nt, f = f_begin + k;
        if (tile != at) cell = flat_cell(sh, tile * 32 + lane, planes, h);
        at = tile;
        const BoxTaps t = load_taps_uniform(sTaps + k * kTapWords);
        const FlatCols cols = flat_cols<true>(t, cell, s.image, sh);
        const FlatRows<false> q = flat_rows<false>(t, cell, h, sh);
        const ColW2 cw = col_weights(t);
        const float sfl = t.scale * t.f_lo_r, sfh = t.scale * t.f_hi_r;
        float mul = 1.0f, add = 0.0f;
        if (FUSED) {
            if (fu.scale) mul = __ldg(fu.scale + c * F + f);
            if (fu.shift) add = __ldg(fu.shift + c * F + f);
        }
        const int64_t first = (((int64_t)(n0 + cell.plane) * C + c) * F + f) * npix + cell.group * kFlatRows * w;
        IO *row = out + first;
        FlatBlock skip;
        if constexpr (FUSED) {
            if (fu.residual) flat_load<float, VEC, true>(skip, fu.residual + first, w, cell, lane, sh.strips);
        }
        f2_t prev[kStrip];
        quad_pair(cols, q.lo(0), q.hi(0), cw, prev);
#pragma unroll
        for (int i = 0; i < kFlatRows; ++i) {
            f2_t cur[kStrip];
            quad_pair(cols, q.lo(i + 1), q.hi(i + 1), cw, cur);
            float v[kStrip];
            quad_forward_row(prev, cur, t.scale, sfl, sfh, v);
#pragma unroll
            for (int m = 0; m < kStrip; ++m) prev[m] = cur[m];
            if constexpr (FUSED) {
#pragma unroll
                for (int m = 0; m < kStrip; ++m) v[m] = v[m] * mul + add;
                if (fu.residual) {
                    float e0, e1, e2, e3;
                    unpack2(skip.a[i], e0, e1);
                    unpack2(skip.b[i], e2, e3);
                    v[0] += e0; v[1] += e1; v[2] += e2; v[3] += e3;
                }
                if (fu.output_relu) {
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) v[m] = fmaxf(v[m], 0.0f);
                }
            }
            if (i < cell.rows) store_row4<IO, VEC>(row, cell.strip * 4, w, v);
            row += w;
        }
    }
}

template <typename IO>
int launch_backward_flat_t(const IO *x, const float *x_integ, const IO *grad_output, const BoxParams &bp, float rep_h, float rep_w, int N, int C, int F,
                           int h, int w, bool normalize, bool exact, int need_mask, IO *grad_input, void *grad_params, int grad_params_kind,
                           float *partials, cudaStream_t s)
{
    const bool need_params = (need_mask & (BC_NEED_ALL & ~BC_NEED_INPUT)) != 0, write_gin = (need_mask & BC_NEED_INPUT) != 0;
    const FlatPlan plan = flat_backward_plan(N, C, F, h, w, write_gin);
    const int teams = (N + plan.sh.planes - 1) / plan.sh.planes;
    const int64_t ctas = (int64_t)teams * C * plan.sh.split;
    if (ctas > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const int vec = Io<IO>::kVecBytes;
    const bool fast = w % 4 == 0 && aligned_to(x, vec) && aligned_to(grad_output, vec) && (!write_gin || aligned_to(grad_input, vec));
    const Finish fin = finish_here(bp, need_params, ctas, (int64_t)N * C * F * h * w, C, grad_params, grad_params_kind, need_mask, teams, rep_h, rep_w, s);
    void (*kern)(const IO *, const float *, const IO *, BoxParams, IO *, float *, int, int, int, int, int, FlatShape, bool, bool, bool, Finish);
    auto pick = [&](auto vecs, auto tiles) {
        constexpr bool V = decltype(vecs)::value;
        constexpr int T = decltype(tiles)::value;
        kern = !need_params ? backward_plane_kernel<IO, V, T, false, false>
               : fin.total  ? backward_plane_kernel<IO, V, T, true, true>
                            : backward_plane_kernel<IO, V, T, true, false>;
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    if (plan.tiles_a_warp == 1) fast ? pick(Flag<true>{}, One{}) : pick(Flag<false>{}, One{});
    else fast ? pick(Flag<true>{}, Two{}) : pick(Flag<false>{}, Two{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kFlatMaxSmem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_PLANE, s);
        if (cudaError_t e = launch_overlapped_cluster(kern, (unsigned)ctas, plan.warps * 32, plan.smem, plan.sh.split, s, x, x_integ, grad_output, bp, grad_input, partials, N, C, F,
                                              h, w, plan.sh, normalize, exact, write_gin, fin))
            return cuda_failed(e, "backward_plane");
    }
    st = check_launch("backward_plane");
    if (st != BC_OK || !need_params || fin.total) return st;
    return launch_finish_param_grads<float>(partials, bp, C * F, teams, normalize, exact, rep_h, rep_w, need_mask, grad_params, s, grad_params_kind);
}

template <typename IO>
int launch_forward_flat_t(const IO *x, const float *integ, const BoxParams &bp, const Fusion *fu, IO *out, int N, int C, int F, int h, int w,
                          bool normalize, bool exact, cudaStream_t s)
{
    const FlatForwardPlan plan = flat_forward_plan(N, C, F, h, w);
    const int64_t ctas = (int64_t)((N + plan.sh.planes - 1) / plan.sh.planes) * C * plan.fsplit;
    // No parts of a plane where the output lies over the input (one filter, in place): a CTA that starts late would integrate
    // rows that another has already replaced.
    const bool in_place = x && ranges_overlap(x, (size_t)N * C * h * w * sizeof(IO), out, (size_t)N * C * F * h * w * sizeof(IO));
    const int tsplit = in_place ? 1 : plan.tsplit;
    if (ctas * tsplit > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool fast = w % 4 == 0 && aligned_to(x, Io<IO>::kVecBytes) && aligned_to(out, Io<IO>::kVecBytes) && (!fu || !fu->residual || aligned_to(fu->residual, 16));
    void (*kern)(const IO *, const float *, BoxParams, IO *, int, int, int, int, int, FlatShape, int, int, bool, bool, bool, Fusion);
    auto pick = [&](auto vecs) {
        constexpr bool V = decltype(vecs)::value, FL = IsFloat<IO>::value;
        if constexpr (FL) {      // (the fused steps are float's)
            // residual rows in flight want registers, unless they cost an SM its second CTA
            if (fu) {
                kern = plan.warps <= 10 || (plan.warps <= 20 && ctas * tsplit <= 148) ? forward_flat_kernel<IO, V, true, false, 640> : forward_flat_kernel<IO, V, true, false, 1024>;
                return;
            }
        }
        kern = x ? forward_flat_kernel<IO, V, false, false, 1024> : forward_flat_kernel<IO, V, false, FL, 1024>;
    };
    if (fast) pick(Flag<true>{});
    else pick(Flag<false>{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kFlatMaxSmem);
    if (st != BC_OK) return st;
    const Fusion none{0, nullptr, nullptr, nullptr, 0};
    {
        LaunchScope scope(KID_FORWARD_FLAT, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)(ctas * tsplit), plan.warps * 32, plan.smem, s, x, integ, bp, out, N, C, F, h, w, plan.sh, plan.fsplit,
                                              tsplit, plan.tight, normalize, exact, fu ? *fu : none))
            return cuda_failed(e, "forward_flat");
    }
    return check_launch("forward_flat");
}

}  // namespace

bool flat_fits_backward(int F, int h, int w)
{
    if (F > kMaxFilters || (int64_t)flat_strips(w) * flat_groups(h) > 32 * kFlatMaxTiles) return false;
    return flat_backward_plan(1, 1, F, h, w, true).smem <= kFlatMaxSmem;
}

// (Samples share a CTA only up to eight tiles of them and 56 KB of images: what holds one plane of more holds those.)
bool flat_fits_forward(int F, int h, int w)
{
    if (F > kMaxFilters || (int64_t)flat_strips(w) * flat_groups(h) > 32 * kFlatMaxTiles) return false;
    return flat_forward_plan(1, 1, F, h, w).smem <= kFlatMaxSmem;
}

int launch_forward_flat(const void *x, const float *integ, int io_kind, const BoxParams &bp, const Fusion *fu, void *out, int N, int C, int F, int h, int w,
                        bool normalize, bool exact, cudaStream_t s)
{
    auto launch = [&](auto zero) {
        using IO = decltype(zero);
        return launch_forward_flat_t(static_cast<const IO *>(x), integ, bp, fu, static_cast<IO *>(out), N, C, F, h, w, normalize, exact, s);
    };
    if (io_kind == BC_IO_F32) return launch(0.0f);
    if (fu) return BC_ERR_UNSUPPORTED;
    return io_kind == BC_IO_F16 ? launch(__half{}) : launch(__nv_bfloat16{});
}

int launch_backward_flat(const void *x, const float *x_integ, int io_kind, const void *grad_output, const BoxParams &bp, float rep_h, float rep_w, int N,
                         int C, int F, int h, int w, bool normalize, bool exact, int need_mask, void *grad_input, void *grad_params,
                         int grad_params_kind, float *partials, cudaStream_t s)
{
    auto launch = [&](auto zero) {
        using IO = decltype(zero);
        return launch_backward_flat_t(static_cast<const IO *>(x), x_integ, static_cast<const IO *>(grad_output), bp, rep_h, rep_w, N, C, F, h, w, normalize,
                                      exact, need_mask, static_cast<IO *>(grad_input), grad_params, grad_params_kind, partials, s);
    };
    if (io_kind == BC_IO_F16) return launch(__half{});
    if (io_kind == BC_IO_BF16) return launch(__nv_bfloat16{});
    return launch(0.0f);
}

}  // namespace bc
