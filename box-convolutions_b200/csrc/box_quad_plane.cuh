// Whole-plane kernels with the integral image in the quad layout (bc_quad.cuh): planes that are wide enough to
// fill a warp's 128 columns and small enough for shared memory.  HBM traffic is the compulsory minimum: no
// integral image ever goes to global memory.
//
// A tile is 8 rows x 128 columns of a plane, one per warp, lane = 4 columns.  The integral image is built from
// registers: a warp loads its tile with one vector load a lane and row, publishes the tile's column sums, takes
// those of the tiles above as the start of its running column sums, scans the rows across the warp and
// stores four conflict-free words a lane and row.  That is two barriers a plane (one more where a plane has
// several column tiles), against three and 35 % more instructions for 32 x 32 tiles.
// The gather is that of the slab kernels: five words of shared memory an output and side, no bank conflicts.
#pragma once
#include "bc_common.cuh"
#include "bc_quad.cuh"
#include "bc_tile_io.cuh"

namespace bc {

namespace {

constexpr int kTileRows = 8;
constexpr int kQuadMaxWarps = 16;
constexpr size_t kQuadMaxSmem = 200 * 1024;
template <int I>
struct Index { static constexpr int value = I; };

// A sub-row has the cells of CT full column tiles whatever the plane's width, so that the layout's strides are
// compile-time constants and a tile's 32 stores and its row addresses need no arithmetic.
template <int CT>
struct QuadImage {
    static constexpr int kCells = 32 * CT + 3;
    static constexpr int kSub = kCells * 4;            // bytes of a sub-row
    static constexpr int kRow = kSub * 4;              // bytes of a row
};
__host__ __device__ inline int quad_image_bytes(int h, int ct) { return (h + 1) * (32 * ct + 3) * 16; }

// Shared memory behind the image: column sums (512 bytes a tile), row sums (32 bytes a tile), then the boxes.
struct QuadSmem {
    uint32_t image, col, row, taps;
};
__device__ __forceinline__ QuadSmem quad_smem(const void *base, int h, int ct, int ntiles)
{
    QuadSmem s;
    s.image = smem_u32(base);
    asm volatile("" : "+r"(s.image));      // opaque: the compiler would rather work the window's base out again at every use
    s.col = s.image + quad_image_bytes(h, ct);
    s.row = s.col + ntiles * 512;
    s.taps = s.row + ntiles * 32;
    return s;
}

__device__ __forceinline__ void sts128(uint32_t a, float4 v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// A warp's tile: 8 rows x 128 columns, 4 columns a lane.
struct QuadTile {
    int rt, ct, p0, c, rows;       // rows inside the plane (0: no tile)
};
template <int CT>
__device__ __forceinline__ QuadTile quad_tile(int tile, int lane, int h)
{
    QuadTile t;
    t.rt = tile / CT;
    t.ct = tile - t.rt * CT;
    t.p0 = t.rt * kTileRows;
    t.c = t.ct * 128 + lane * 4;
    t.rows = max(min(kTileRows, h - t.p0), 0);
    return t;
}

// Zeroes what never changes in the integral image: row 0, and the first cell and column 0 of every row.
template <int CT>
__device__ __forceinline__ void quad_zero_padding(uint32_t image, int h)
{
    using Q = QuadImage<CT>;
    for (int i = threadIdx.x; i < Q::kRow / 16; i += blockDim.x) sts128(image + i * 16, make_float4(0.f, 0.f, 0.f, 0.f));
    for (int a = 1 + threadIdx.x; a <= h; a += blockDim.x) {
        const uint32_t row = image + a * Q::kRow;
        sts<0>(row, 0.f); sts<4>(row, 0.f);
        sts<Q::kSub>(row, 0.f); sts<2 * Q::kSub>(row, 0.f); sts<3 * Q::kSub>(row, 0.f);
    }
}

// FULL: the tile has all its rows.
template <typename IO, bool VEC, bool FULL>
__device__ __forceinline__ void quad_load_tile(float4 (&v)[kTileRows], const QuadTile &t, const IO *plane, int w, int lane)
{
    const IO *row = plane + t.p0 * w;
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) v[i] = load_row4<IO, VEC>(row + i * w, t.c, w, FULL || i < t.rows, lane);
}

// Build, first part: the tile's own 2-D prefix sums; with several column tiles only down its columns and along
// its rows within the tile, the rows' totals being published (followed by a barrier, then quad_join_rows()).
template <int CT>
__device__ __forceinline__ void quad_scan(float4 (&v)[kTileRows], float (&carry)[kTileRows], const QuadTile &t, const QuadSmem &s, int lane)
{
#pragma unroll
    for (int i = 1; i < kTileRows; ++i) { v[i].x += v[i - 1].x; v[i].y += v[i - 1].y; v[i].z += v[i - 1].z; v[i].w += v[i - 1].w; }
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) {
        v[i].y += v[i].x;
        v[i].z += v[i].y;
        v[i].w += v[i].z;
        const float incl = warp_scan(v[i].w);
        carry[i] = incl - v[i].w;
        if (CT > 1 && lane == 31) sts<0>(s.row + (t.rt * CT + t.ct) * 32 + i * 4, incl);
    }
}
// Second part: carries joined, the tile's last row published as what it adds to the tiles below.  Followed by a
// barrier.
template <int CT>
__device__ __forceinline__ void quad_publish(float4 (&v)[kTileRows], float (&carry)[kTileRows], const QuadTile &t, const QuadSmem &s, int lane)
{
    if (CT > 1) {
        for (int k = 0; k < t.ct; ++k) {
            const float4 a = lds128(s.row + (t.rt * CT + k) * 32), b = lds128(s.row + (t.rt * CT + k) * 32 + 16);
            carry[0] += a.x; carry[1] += a.y; carry[2] += a.z; carry[3] += a.w;
            carry[4] += b.x; carry[5] += b.y; carry[6] += b.z; carry[7] += b.w;
        }
    }
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) { v[i].x += carry[i]; v[i].y += carry[i]; v[i].z += carry[i]; v[i].w += carry[i]; }
    sts128(s.col + (t.rt * CT + t.ct) * 512 + lane * 16, v[kTileRows - 1]);
}
// Third part: what the tiles above add, and the stores.  Followed by a barrier.
template <int CT, bool FULL>
__device__ __forceinline__ void quad_store(const float4 (&v)[kTileRows], const QuadTile &t, const QuadSmem &s, int w, int lane)
{
    using Q = QuadImage<CT>;
    float4 up = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t above = s.col + t.ct * 512 + lane * 16;
    for (int r = 0; r < t.rt; ++r, above += CT * 512) {
        const float4 u = lds128(above);
        up.x += u.x; up.y += u.y; up.z += u.z; up.w += u.w;
    }
    // column c+1 of integral row p0+1: sub-row 1, cell c/4 + 1
    const uint32_t at = s.image + (t.p0 + 1) * Q::kRow + ((t.c >> 2) + 1) * 4;
    auto put = [&](auto I) {
        constexpr int kI = decltype(I)::value;
        if (FULL || kI < t.rows) {
            sts<kI * Q::kRow + Q::kSub>(at, v[kI].x + up.x);
            sts<kI * Q::kRow + 2 * Q::kSub>(at, v[kI].y + up.y);
            sts<kI * Q::kRow + 3 * Q::kSub>(at, v[kI].z + up.z);
            sts<kI * Q::kRow + 4>(at, v[kI].w + up.w);
        }
    };
    put(Index<0>{}); put(Index<1>{}); put(Index<2>{}); put(Index<3>{});
    put(Index<4>{}); put(Index<5>{}); put(Index<6>{}); put(Index<7>{});
    // Cells of columns past the last lane's (planes whose width comes within eight columns of the tiles'): seven
    // words a row, one lane each.
    if (t.ct == CT - 1 && (w >> 2) + 2 > 32 * CT) {
        const int sub = lane < 3 ? lane + 1 : lane - 3, cell = lane < 3 ? 32 * CT + 1 : 32 * CT + 2;
        const uint32_t extra = s.image + (t.p0 + 1) * Q::kRow + sub * Q::kSub + cell * 4;
        auto copy = [&](auto I) {
            constexpr int i = decltype(I)::value;
            const float last = __shfl_sync(0xffffffffu, v[i].w + up.w, 31);
            if (lane < 7 && (FULL || i < t.rows)) sts<i * Q::kRow>(extra, last);
        };
        copy(Index<0>{}); copy(Index<1>{}); copy(Index<2>{}); copy(Index<3>{});
        copy(Index<4>{}); copy(Index<5>{}); copy(Index<6>{}); copy(Index<7>{});
    }
}

// Forward: one CTA per (plane, part of the filters).  T: tiles a warp holds while it builds.  The gather is cut
// into tasks of one filter, one column tile and `chunk` row tiles, walked top to bottom so that a tap-row pair
// is loaded once per row and once more per task.
// FAST: rows and tensors aligned for vector accesses, heights a multiple of 8.
template <typename IO, int CT, int T, bool FAST, bool FUSED, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 3 : 1)
forward_quad_kernel(const IO *__restrict__ x, BoxParams bp, IO *out, int C, int F, int h, int w, int row_tiles, int fsplit, int chunk,
                    bool normalize, bool exact, Fusion fu)
{
    using Q = QuadImage<CT>;
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int part = blockIdx.x % fsplit, plane_at = blockIdx.x / fsplit, c = plane_at % C;
    const int f_begin = (F * part) / fsplit, nf = (F * (part + 1)) / fsplit - f_begin;
    const int64_t npix = (int64_t)h * w, nc = plane_at;
    const int cells = quad_cells(w), ntiles = row_tiles * CT;
    const QuadSmem s = quad_smem(smem4, h, CT, ntiles);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));

    quad_zero_padding<CT>(s.image, h);
    // registers and shared memory only up to here; now what the kernel in front of this one may have written
    grid_dependency_wait();
    {
        QuadTile tile[T];
        float4 v[T][kTileRows];
        float carry[T][kTileRows];
#pragma unroll
        for (int k = 0; k < T; ++k) {
            tile[k] = quad_tile<CT>(warp + k * nwarps, lane, h);
            if (tile[k].rows) quad_load_tile<IO, FAST, FAST>(v[k], tile[k], x + nc * npix, w, lane);
        }
        if ((int)threadIdx.x < nf) {
            const Box box = load_box(bp, c * F + f_begin + threadIdx.x);
            store_taps(sTaps + threadIdx.x * kTapWords, taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
        }
#pragma unroll
        for (int k = 0; k < T; ++k) {
            if (!tile[k].rows) continue;
            if (FUSED && fu.input_relu) {
#pragma unroll
                for (int i = 0; i < kTileRows; ++i)
                    v[k][i] = make_float4(fmaxf(v[k][i].x, 0.f), fmaxf(v[k][i].y, 0.f), fmaxf(v[k][i].z, 0.f), fmaxf(v[k][i].w, 0.f));
            }
            quad_scan<CT>(v[k], carry[k], tile[k], s, lane);
        }
        if (CT > 1) __syncthreads();
#pragma unroll
        for (int k = 0; k < T; ++k)
            if (tile[k].rows) quad_publish<CT>(v[k], carry[k], tile[k], s, lane);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < T; ++k)
            if (tile[k].rows) quad_store<CT, FAST>(v[k], tile[k], s, w, lane);
    }
    __syncthreads();

    const int groups = (row_tiles + chunk - 1) / chunk, ntasks = nf * groups * CT;
    for (int task = warp; task < ntasks; task += nwarps) {
        const int rest = task / nf, k = task - rest * nf, f = f_begin + k;
        const int g = rest / CT, ct = rest - g * CT;
        const BoxTaps t = load_taps_uniform(sTaps + k * kTapWords);
        const int q0 = ct * 128 + lane * kStrip;
        const QuadCols cols = quad_cols(t, q0 >> 2, cells, Q::kCells);
        const ColW2 cw = col_weights(t);
        const float sfl = t.scale * t.f_lo_r, sfh = t.scale * t.f_hi_r;
        float mul = 1.0f, add = 0.0f;
        if (FUSED) {
            if (fu.scale) mul = __ldg(fu.scale + c * F + f);
            if (fu.shift) add = __ldg(fu.shift + c * F + f);
        }
        const int p_begin = g * chunk * kTileRows, p_end = min(p_begin + chunk * kTileRows, h);
        const int64_t first = (nc * F + f) * npix + (int64_t)p_begin * w;
        IO *row = out + first;
        const float *res = FUSED && fu.residual ? fu.residual + first + q0 : nullptr;
        f2_t prev[kStrip];
        for (int p0 = p_begin; p0 < p_end; p0 += kTileRows) {
            const QuadRows<kTileRows> r = quad_rows<kTileRows>(t, p0, h, s.image, s.image, Q::kRow, lane);
            if (p0 == p_begin) quad_pair(cols, r.lo[0], r.hi[0], cw, prev);
#pragma unroll
            for (int i = 0; i < kTileRows; ++i) {
                if (FAST || p0 + i < p_end) {
                    f2_t cur[kStrip];
                    quad_pair(cols, r.lo[i + 1], r.hi[i + 1], cw, cur);
                    float v[kStrip];
                    quad_forward_row(prev, cur, t.scale, sfl, sfh, v);
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) prev[m] = cur[m];
                    if (FUSED) {
#pragma unroll
                        for (int m = 0; m < kStrip; ++m) v[m] = v[m] * mul + add;
                        if (res) {      // plain loads: the residual may be the output
                            if (FAST) {
                                const float4 e = q0 < w ? *reinterpret_cast<const float4 *>(res) : make_float4(0.f, 0.f, 0.f, 0.f);
                                v[0] += e.x; v[1] += e.y; v[2] += e.z; v[3] += e.w;
                            } else {
#pragma unroll
                                for (int m = 0; m < kStrip; ++m)
                                    if (q0 + m < w) v[m] += res[m];
                            }
                            res += w;
                        }
                        if (fu.output_relu) {
#pragma unroll
                            for (int m = 0; m < kStrip; ++m) v[m] = fmaxf(v[m], 0.0f);
                        }
                    }
                    store_row4<IO, FAST>(row, q0, w, v, lane);
                    row += w;
                }
            }
        }
    }
}

// Backward: one CTA per plane, one tile per warp.  Per filter the grad_output plane is integrated in shared
// memory and gathered with the mirrored box.  The grad-input accumulators of a lane's 8 x 4 pixels stay in
// registers; its input values wait in shared memory, where only their own warp touches them.  The next
// grad_output plane is requested into L2 while the current one is gathered.
template <typename IO, int CT, bool FAST, bool NEED_PARAMS, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 2 : 1)
backward_quad_kernel(const IO *__restrict__ x, const IO *__restrict__ grad_output, BoxParams bp, IO *__restrict__ grad_input,
                     float *__restrict__ partials, int N, int C, int F, int h, int w, int row_tiles, bool normalize, bool exact,
                     bool write_gin)
{
    using Q = QuadImage<CT>;
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int64_t nc = blockIdx.x;
    const int c = blockIdx.x % C, n = blockIdx.x / C;
    const int npix = h * w, cells = quad_cells(w), ntiles = row_tiles * CT;
    const QuadSmem s = quad_smem(smem4, h, CT, ntiles);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));
    float *red = sTaps + F * kTapWords;                                                        // [F][warps][5]
    const uint32_t sx = s.taps + ((F * (kTapWords + ntiles * kNumSums) * 4 + 15) & ~15) + warp * (kTileRows * 512) + lane * 16;
    const IO *gbase = grad_output + nc * F * (int64_t)npix;
    const QuadTile tile = quad_tile<CT>(warp, lane, h);

    if (FAST && threadIdx.x == 0) bulk_prefetch_l2(gbase, (uint32_t)npix * (uint32_t)sizeof(IO));
    quad_zero_padding<CT>(s.image, h);
    grid_dependency_wait();
    if (NEED_PARAMS) {
        float4 v[kTileRows];
        quad_load_tile<IO, FAST, FAST>(v, tile, x + nc * npix, w, lane);
#pragma unroll
        for (int i = 0; i < kTileRows; ++i) sts128(sx + i * 512, v[i]);
    }
    if ((int)threadIdx.x < F) {
        const Box box = load_box(bp, c * F + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    float gin[kTileRows][kStrip];
#pragma unroll
    for (int i = 0; i < kTileRows; ++i)
#pragma unroll
        for (int m = 0; m < kStrip; ++m) gin[i][m] = 0.0f;
    for (int f = 0; f < F; ++f) {
        {
            float4 v[kTileRows];
            float carry[kTileRows];
            quad_load_tile<IO, FAST, FAST>(v, tile, gbase + f * (int64_t)npix, w, lane);
            if (FAST && threadIdx.x == 0 && f + 1 < F)
                bulk_prefetch_l2(gbase + (f + 1) * (int64_t)npix, (uint32_t)npix * (uint32_t)sizeof(IO));
            quad_scan<CT>(v, carry, tile, s, lane);
            if (CT > 1) __syncthreads();
            quad_publish<CT>(v, carry, tile, s, lane);
            __syncthreads();      // (also: every gather of the previous filter is done)
            quad_store<CT, FAST>(v, tile, s, w, lane);
        }
        __syncthreads();
        float sums[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
        const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
        quad_backward_strip<kTileRows, NEED_PARAMS, FAST>(t, quad_cols(t, tile.c >> 2, cells, Q::kCells),
                                                          quad_rows<kTileRows>(t, tile.p0, h, s.image, s.image, Q::kRow, lane),
                                                          col_weights(t), [&](int i) { return lds128(sx + i * 512); }, gin, sums,
                                                          tile.rows);
        if (NEED_PARAMS) {
            const float sum = warp_sum5(sums, lane);
            const int slot = sum5_slot(lane);
            if (slot >= 0) red[(f * nwarps + warp) * kNumSums + slot] = sum;
        }
    }
    if (NEED_PARAMS) {
        __syncthreads();
        for (int i = threadIdx.x; i < F * kNumSums; i += blockDim.x) {
            const int f = i / kNumSums, j = i - f * kNumSums;
            float sum = 0.0f;
            for (int k = 0; k < nwarps; ++k) sum += red[(f * nwarps + k) * kNumSums + j];
            partials[((int64_t)(c * F + f) * N + n) * kNumSums + j] = sum;
        }
    }
    if (write_gin) {
        IO *row = grad_input + nc * npix + tile.p0 * w;
#pragma unroll
        for (int i = 0; i < kTileRows; ++i, row += w)
            if (FAST || i < tile.rows) store_row4<IO, FAST>(row, tile.c, w, gin[i], lane);
    }
}

inline int quad_row_tiles(int h) { return (h + kTileRows - 1) / kTileRows; }
inline int quad_col_tiles(int w) { return (w + 127) / 128; }
inline size_t quad_forward_smem(int F, int h, int w)
{
    const int ct = quad_col_tiles(w), tiles = quad_row_tiles(h) * ct;
    return (size_t)quad_image_bytes(h, ct) + tiles * 544 + F * kTapWords * 4;
}
inline size_t quad_backward_smem(int F, int h, int w)
{
    const size_t tiles = (size_t)quad_row_tiles(h) * quad_col_tiles(w);
    return quad_forward_smem(F, h, w) + F * tiles * kNumSums * 4 + 16 + tiles * kTileRows * 512;
}
#ifndef QMINW
#define QMINW 65
#endif
inline bool quad_fits_forward(int F, int h, int w)
{
    return w >= QMINW && w <= 256 && F <= kMaxFilters && quad_row_tiles(h) * quad_col_tiles(w) <= 2 * kQuadMaxWarps &&
           quad_forward_smem(F, h, w) <= kQuadMaxSmem;
}
inline bool quad_fits_backward(int F, int h, int w)
{
    return w >= QMINW && w <= 256 && F <= kMaxFilters && quad_row_tiles(h) * quad_col_tiles(w) <= kQuadMaxWarps &&
           quad_backward_smem(F, h, w) <= kQuadMaxSmem;
}

template <typename IO>
int launch_forward_quad_t(const IO *x, const BoxParams &bp, const Fusion *fu, IO *out, int N, int C, int F, int h, int w,
                          bool normalize, bool exact, cudaStream_t s)
{
    const int row_tiles = quad_row_tiles(h), col_tiles = quad_col_tiles(w), tiles = row_tiles * col_tiles;
    const int64_t planes = (int64_t)N * C;
    int fsplit = 1;
    if (F % 2 == 0 && planes < 148 * 6) fsplit = 2;
    while (fsplit < F && F % (fsplit * 2) == 0 && planes * fsplit * 2 <= 148 * 2) fsplit *= 2;
    if (planes * fsplit > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const int T = tiles > 8 ? 2 : 1;
    const int warps = (tiles + T - 1) / T, nf = (F + fsplit - 1) / fsplit;
    // rows per task: few long tasks read fewer tap rows twice, but every warp should get the same share
    int chunk = 1;
    double best = 1e30;
    for (int k = 1; k <= row_tiles; ++k) {
        const int tasks = nf * ((row_tiles + k - 1) / k) * col_tiles;
        const double cost = ((tasks + warps - 1) / warps) * (k * kTileRows + 2.0);
        if (cost < best) { best = cost; chunk = k; }
    }
    const bool fast = w % 4 == 0 && h % kTileRows == 0 && aligned_to(x, Io<IO>::kVecBytes) && aligned_to(out, Io<IO>::kVecBytes) &&
                     (!fu || !fu->residual || aligned_to(fu->residual, 16));
    void (*kern)(const IO *, BoxParams, IO *, int, int, int, int, int, int, int, bool, bool, Fusion);
    auto pick = [&](auto ct) {
        constexpr int CT = decltype(ct)::value, S = 256, L = 512;
        constexpr bool FU = IsFloat<IO>::value;
        if (T == 1) {
            if (fu) kern = fast ? forward_quad_kernel<IO, CT, 1, true, FU, S> : forward_quad_kernel<IO, CT, 1, false, FU, S>;
            else kern = fast ? forward_quad_kernel<IO, CT, 1, true, false, S> : forward_quad_kernel<IO, CT, 1, false, false, S>;
        } else {
            if (fu) kern = fast ? forward_quad_kernel<IO, CT, 2, true, FU, L> : forward_quad_kernel<IO, CT, 2, false, FU, L>;
            else kern = fast ? forward_quad_kernel<IO, CT, 2, true, false, L> : forward_quad_kernel<IO, CT, 2, false, false, L>;
        }
    };
    if (col_tiles == 1) pick(Index<1>{});
    else pick(Index<2>{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kQuadMaxSmem);
    if (st != BC_OK) return st;
    const Fusion none{0, nullptr, nullptr, nullptr, 0};
    {
        LaunchScope scope(KID_FORWARD_QUAD, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)(planes * fsplit), warps * 32, quad_forward_smem(nf, h, w), s, x, bp, out,
                                              C, F, h, w, row_tiles, fsplit, chunk, normalize, exact, fu ? *fu : none))
            return cuda_failed(e, "forward_quad");
    }
    return check_launch("forward_quad");
}

template <typename IO>
int launch_backward_quad_t(const IO *x, const IO *grad_output, const BoxParams &bp, float rep_h, float rep_w, int N, int C, int F,
                           int h, int w, bool normalize, bool exact, int need_mask, IO *grad_input, void *grad_params,
                           int grad_params_kind, float *partials, cudaStream_t s)
{
    const int row_tiles = quad_row_tiles(h), col_tiles = quad_col_tiles(w), tiles = row_tiles * col_tiles;
    const int64_t planes = (int64_t)N * C;
    if (planes > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool need_params = (need_mask & (BC_NEED_ALL & ~BC_NEED_INPUT)) != 0;
    const bool write_gin = (need_mask & BC_NEED_INPUT) != 0;
    const bool fast = w % 4 == 0 && h % kTileRows == 0 && ((size_t)h * w * sizeof(IO)) % 16 == 0 && aligned_to(x, Io<IO>::kVecBytes) &&
                     aligned_to(grad_output, 16) && (!write_gin || aligned_to(grad_input, Io<IO>::kVecBytes));
    void (*kern)(const IO *, const IO *, BoxParams, IO *, float *, int, int, int, int, int, int, bool, bool, bool);
    auto pick = [&](auto ct) {
        constexpr int CT = decltype(ct)::value, S = 256, L = 512;
        if (tiles <= 8) {
            if (need_params) kern = fast ? backward_quad_kernel<IO, CT, true, true, S> : backward_quad_kernel<IO, CT, false, true, S>;
            else kern = fast ? backward_quad_kernel<IO, CT, true, false, S> : backward_quad_kernel<IO, CT, false, false, S>;
        } else {
            if (need_params) kern = fast ? backward_quad_kernel<IO, CT, true, true, L> : backward_quad_kernel<IO, CT, false, true, L>;
            else kern = fast ? backward_quad_kernel<IO, CT, true, false, L> : backward_quad_kernel<IO, CT, false, false, L>;
        }
    };
    if (col_tiles == 1) pick(Index<1>{});
    else pick(Index<2>{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kQuadMaxSmem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_QUAD, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)planes, tiles * 32, quad_backward_smem(F, h, w), s, x, grad_output, bp,
                                              grad_input, partials, N, C, F, h, w, row_tiles, normalize, exact, write_gin))
            return cuda_failed(e, "backward_quad");
    }
    st = check_launch("backward_quad");
    if (st != BC_OK || !need_params) return st;
    return launch_finish_param_grads<float>(partials, bp, C * F, N, normalize, exact, rep_h, rep_w, need_mask, grad_params, s,
                                            grad_params_kind);
}

}  // namespace

}  // namespace bc
