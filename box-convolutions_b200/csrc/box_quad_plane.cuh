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
#include <type_traits>

#include "bc_common.cuh"
#include "bc_finish.cuh"
#include "bc_quad.cuh"
#include "bc_tile_io.cuh"
#include "bc_tmem.cuh"

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

// Shared memory behind the image: last rows (512 bytes a tile), row sums (32 bytes a tile), a scan corner per warp
// (kScanBytes), then the boxes.
struct QuadSmem {
    uint32_t image, col, row, scan, taps;
};
__device__ __forceinline__ QuadSmem quad_smem(const void *base, int h, int ct, int ntiles, int nwarps)
{
    QuadSmem s;
    s.image = smem_u32(base);
    asm volatile("" : "+r"(s.image));      // opaque: the compiler would rather work the window's base out again at every use
    s.col = s.image + quad_image_bytes(h, ct);
    s.row = s.col + ntiles * 512;
    s.scan = s.row + ntiles * 32;
    s.taps = s.scan + nwarps * (kTileRows * 36 * 4);
    return s;
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

// A lane's 8 x 4 values, each row as two packed pairs (columns c, c+1 and c+2, c+3).
struct QuadBlock {
    f2_t a[kTileRows], b[kTileRows];
};

// FULL: the tile has all its rows.
template <typename IO, bool VEC, bool FULL>
__device__ __forceinline__ void quad_load_tile(QuadBlock &v, const QuadTile &t, const IO *plane, int w, int lane)
{
    const IO *row = plane + t.p0 * w;
    Rows8 g;
    rows8_load<IO, VEC>(g, row, w, t.c, FULL ? kTileRows : t.rows, lane);
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) {
        const float4 e = rows8_get<IO, VEC>(g, row, w, t.c, lane, i);
        v.a[i] = pack2(e.x, e.y);
        v.b[i] = pack2(e.z, e.w);
    }
}

// Build, first part: the tile's own 2-D prefix sums; with several column tiles only down its columns and along
// its rows within the tile, the rows' totals being published (followed by a barrier).
// The sums of a row's 32 lanes are scanned eight rows at once through a corner of shared memory: four lanes a
// row, each with eight of its values, then two shuffle steps.  Shuffling every row by itself takes five
// shuffles and five additions a row, twice the instructions.
constexpr int kScanPitch = 36;      // words per row: eight lanes' 16-byte accesses fall into distinct banks
constexpr int kScanBytes = kTileRows * kScanPitch * 4;
template <int CT>
__device__ __forceinline__ void quad_scan(QuadBlock &v, float (&carry)[kTileRows], const QuadTile &t, const QuadSmem &s, int warp, int lane)
{
    const uint32_t scan = s.scan + warp * kScanBytes;
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) {
        if (i) { v.a[i] = add2(v.a[i], v.a[i - 1]); v.b[i] = add2(v.b[i], v.b[i - 1]); }
    }
    __syncwarp();
    auto row_of = [&](auto I) {
        constexpr int i = decltype(I)::value;
        float x, y, z, u;
        unpack2(v.a[i], x, y);
        unpack2(v.b[i], z, u);
        y += x; z += y; u += z;
        v.a[i] = pack2(x, y);
        v.b[i] = pack2(z, u);
        sts<i * kScanPitch * 4>(scan + lane * 4, u);
    };
    row_of(Index<0>{}); row_of(Index<1>{}); row_of(Index<2>{}); row_of(Index<3>{});
    row_of(Index<4>{}); row_of(Index<5>{}); row_of(Index<6>{}); row_of(Index<7>{});
    __syncwarp();
    const int k = lane & 3;
    const uint32_t mine = scan + (lane >> 2) * (kScanPitch * 4) + k * 32;
    float4 p = lds128(mine), q = lds128(mine + 16);
    p.y += p.x; p.z += p.y; p.w += p.z;
    q.x += p.w; q.y += q.x; q.z += q.y; q.w += q.z;
    // What the row has in front of the four lanes' shares, added up by itself: taking a lane's own share off an inclusive
    // sum again would leave its infinity or its rounding in the 32 columns to its left.
    const float one = __shfl_up_sync(0xffffffffu, q.w, 1);
    float before = k >= 1 ? one : 0.0f;
    const float two = __shfl_up_sync(0xffffffffu, q.w + before, 2);
    if (k >= 2) before += two;
    if (CT > 1 && k == 3) sts<0>(s.row + (t.rt * CT + t.ct) * 32 + (lane >> 2) * 4, before + q.w);
    sts128(mine, make_float4(before, before + p.x, before + p.y, before + p.z));
    sts128(mine + 16, make_float4(before + p.w, before + q.x, before + q.y, before + q.z));
    __syncwarp();
    auto carry_of = [&](auto I) { constexpr int i = decltype(I)::value; carry[i] = lds<i * kScanPitch * 4>(scan + lane * 4); };
    carry_of(Index<0>{}); carry_of(Index<1>{}); carry_of(Index<2>{}); carry_of(Index<3>{});
    carry_of(Index<4>{}); carry_of(Index<5>{}); carry_of(Index<6>{}); carry_of(Index<7>{});
}
// Second part: carries joined, the tile's last row published as what it adds to the tiles below.  Followed by a
// barrier.
template <int CT>
__device__ __forceinline__ void quad_publish(QuadBlock &v, float (&carry)[kTileRows], const QuadTile &t, const QuadSmem &s, int lane)
{
    if (CT > 1) {
        for (int k = 0; k < t.ct; ++k) {
            const float4 a = lds128(s.row + (t.rt * CT + k) * 32), b = lds128(s.row + (t.rt * CT + k) * 32 + 16);
            carry[0] += a.x; carry[1] += a.y; carry[2] += a.z; carry[3] += a.w;
            carry[4] += b.x; carry[5] += b.y; carry[6] += b.z; carry[7] += b.w;
        }
    }
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) {
        const f2_t c = pack2(carry[i], carry[i]);
        v.a[i] = add2(v.a[i], c);
        v.b[i] = add2(v.b[i], c);
    }
    float4 e;
    unpack2(v.a[kTileRows - 1], e.x, e.y);
    unpack2(v.b[kTileRows - 1], e.z, e.w);
    sts128(s.col + (t.rt * CT + t.ct) * 512 + lane * 16, e);
}
// Third part: what the tiles above add, and the stores.  Followed by a barrier.
template <int CT, bool FULL>
__device__ __forceinline__ void quad_store(QuadBlock &v, const QuadTile &t, const QuadSmem &s, int w, int lane)
{
    using Q = QuadImage<CT>;
    f2_t up_a = pack2(0.f, 0.f), up_b = up_a;
    uint32_t above = s.col + t.ct * 512 + lane * 16;
    for (int r = 0; r < t.rt; ++r, above += CT * 512) {
        const float4 u = lds128(above);
        up_a = add2(up_a, pack2(u.x, u.y));
        up_b = add2(up_b, pack2(u.z, u.w));
    }
#pragma unroll
    for (int i = 0; i < kTileRows; ++i) { v.a[i] = add2(v.a[i], up_a); v.b[i] = add2(v.b[i], up_b); }
    // column c+1 of integral row p0+1: sub-row 1, cell c/4 + 1
    const uint32_t at = s.image + (t.p0 + 1) * Q::kRow + ((t.c >> 2) + 1) * 4;
    const bool inside = t.c < w;
    auto put = [&](auto I) {
        constexpr int kI = decltype(I)::value;
        if (inside && (FULL || kI < t.rows)) {
            float x, y, z, u;
            unpack2(v.a[kI], x, y);
            unpack2(v.b[kI], z, u);
            sts<kI * Q::kRow + Q::kSub>(at, x);
            sts<kI * Q::kRow + 2 * Q::kSub>(at, y);
            sts<kI * Q::kRow + 3 * Q::kSub>(at, z);
            sts<kI * Q::kRow + 4>(at, u);
        }
    };
    put(Index<0>{}); put(Index<1>{}); put(Index<2>{}); put(Index<3>{});
    put(Index<4>{}); put(Index<5>{}); put(Index<6>{}); put(Index<7>{});
    // Columns past w hold exactly what column w holds (a box border out there contributes nothing): the seven words behind the last strip,
    // four lanes a row.  (Adding the rows up in every lane past the plane and copying the value there took 40 instructions more, 2.5 % of the backward.)
    if (t.ct == CT - 1) {
        const int k = lane & 3, i = lane >> 2;
        const uint32_t end = s.image + (t.p0 + 1 + i) * Q::kRow + (((w - 1) >> 2) + 2) * 4;
        __syncwarp();
        if (FULL || i < t.rows) {
            const float u = lds<0>(end);
            sts<0>(end + (k ? k * Q::kSub : 4), u);
            if (k) sts<4>(end + k * Q::kSub, u);
        }
    }
}

// Forward: one CTA per (plane, part of the filters).  T: tiles a warp holds while it builds.  The gather is cut
// into tasks of one filter, one column tile and `chunk` row tiles, walked top to bottom so that a tap-row pair
// is loaded once per row and once more per task.
// FAST: rows and tensors aligned for vector accesses, heights a multiple of 8.
// A null `x`: `integ` holds the plane's integral image, plain rows of w + 1 floats, which is only copied.
// FUSED: the inference steps of `Fusion` (the output may then alias the residual).  Such calls are single frames, a
// few CTAs an SM at most: registers are there to have all residual rows of a task in flight before its gather,
// and the planes travel to L2 while the CTA still waits for the kernel in front.
// Row parts (rsplit): few large planes, a CTA gathers only some of the rows for its filters.
template <typename IO, int CT, int T, bool FAST, bool FUSED, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? (FUSED ? 2 : 3) : 1)
forward_quad_kernel(const IO *__restrict__ x, const float *__restrict__ integ, BoxParams bp, IO *out, int C, int F, int h, int w, int row_tiles, int fsplit,
                    int rsplit, int chunk, bool normalize, bool exact, Fusion fu)
{
    using Q = QuadImage<CT>;
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int row_part = blockIdx.x % rsplit, b = blockIdx.x / rsplit;
    const int part = b % fsplit, plane_at = b / fsplit, c = plane_at % C;
    const int f_begin = (F * part) / fsplit, nf = (F * (part + 1)) / fsplit - f_begin;
    const int first_tile = (row_tiles * row_part) / rsplit, end_tile = (row_tiles * (row_part + 1)) / rsplit;
    const int64_t npix = (int64_t)h * w, nc = plane_at;
    const int cells = quad_cells(w), ntiles = row_tiles * CT;
    const QuadSmem s = quad_smem(smem4, h, CT, ntiles, nwarps);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));

    if (FUSED) {      // hints only
        prefetch_l2(x + nc * npix, npix * sizeof(IO));
        if (fu.residual) {
            const int64_t p0 = first_tile * kTileRows * w, p1 = min(end_tile * kTileRows, h) * w;
            if (rsplit == 1) prefetch_l2(fu.residual + (nc * F + f_begin) * npix, (size_t)nf * npix * sizeof(float));
            else
                for (int k = 0; k < nf; ++k) prefetch_l2(fu.residual + (nc * F + f_begin + k) * npix + p0, (size_t)(p1 - p0) * sizeof(float));
        }
    }
    quad_zero_padding<CT>(s.image, h);
    // registers and shared memory only up to here; now what the kernel in front of this one may have written
    grid_dependency_wait();
    if (!x) {
        if ((int)threadIdx.x < nf) {
            const Box box = load_box(bp, c * F + f_begin + threadIdx.x);
            store_taps(sTaps + threadIdx.x * kTapWords, taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
        }
        const float *I = integ + nc * (int64_t)(h + 1) * (w + 1);
        __syncthreads();      // (the zero padding has been written)
        for (int a = warp; a <= h; a += nwarps) {
            for (int col = lane; col < 4 * (cells - 1); col += 32) {
                const float e = __ldg(I + (int64_t)a * (w + 1) + min(col, w));
                sts<0>(s.image + a * Q::kRow + (col & 3) * Q::kSub + ((col >> 2) + 1) * 4, e);
            }
        }
    } else {
        QuadTile tile[T];
        QuadBlock v[T];
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
                for (int i = 0; i < kTileRows; ++i) {
                    float e0, e1;
                    unpack2(v[k].a[i], e0, e1);
                    v[k].a[i] = pack2(fmaxf(e0, 0.f), fmaxf(e1, 0.f));
                    unpack2(v[k].b[i], e0, e1);
                    v[k].b[i] = pack2(fmaxf(e0, 0.f), fmaxf(e1, 0.f));
                }
            }
            quad_scan<CT>(v[k], carry[k], tile[k], s, warp, lane);
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

    const int groups = (end_tile - first_tile + chunk - 1) / chunk, ntasks = nf * groups * CT;
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
        const int p_begin = (first_tile + g * chunk) * kTileRows, p_end = min(min(first_tile + (g + 1) * chunk, end_tile) * kTileRows, h);
        const int64_t first = (nc * F + f) * npix + (int64_t)p_begin * w;
        IO *row = out + first;
        const float *res = FUSED && fu.residual ? fu.residual + first : nullptr;
        f2_t prev[kStrip];
        for (int p0 = p_begin; p0 < p_end; p0 += kTileRows) {
            Rows8 skip;
            if (FUSED && res) rows8_load<float, FAST, true>(skip, res, w, q0, FAST ? kTileRows : p_end - p0, lane);
            const QuadRows<kTileRows> r = quad_rows<kTileRows>(t, p0, h, s.image, s.image, Q::kRow, lane);
            if (p0 == p_begin) quad_pair(cols, r.lo(0), r.hi(0), cw, prev);
#pragma unroll
            for (int i = 0; i < kTileRows; ++i) {
                if (FAST || p0 + i < p_end) {
                    f2_t cur[kStrip];
                    quad_pair(cols, r.lo(i + 1), r.hi(i + 1), cw, cur);
                    float v[kStrip];
                    quad_forward_row(prev, cur, t.scale, sfl, sfh, v);
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) prev[m] = cur[m];
                    if (FUSED) {
#pragma unroll
                        for (int m = 0; m < kStrip; ++m) v[m] = v[m] * mul + add;
                        if (res) {
                            const float4 e = rows8_get<float, FAST>(skip, res, w, q0, lane, i);
                            v[0] += e.x; v[1] += e.y; v[2] += e.z; v[3] += e.w;
                        }
                        if (fu.output_relu) {
#pragma unroll
                            for (int m = 0; m < kStrip; ++m) v[m] = fmaxf(v[m], 0.0f);
                        }
                    }
                    store_row4<IO, FAST>(row, q0, w, v);
                    row += w;
                }
            }
            if (FUSED && res) res += kTileRows * w;
        }
    }
}

// Backward: one CTA per plane, one tile per warp.  Per filter the grad_output plane is integrated in shared
// memory and gathered with the mirrored box.  The grad-input accumulators of a lane's 8 x 4 pixels and its input
// values wait in tensor memory (bc_tmem.cuh).  The next grad_output plane is requested into L2 while the
// current one is gathered.
// Bound by the latencies of its phases, which other CTAs of the SM have to cover: (256,32,4,64,128) with accumulators in
// registers and input values in shared memory, two CTAs an SM: 564 us; like this, three: 504 us.
template <typename IO, int CT, bool FAST, bool NEED_PARAMS, bool COUNTED, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT > 384 ? 1 : MAXT > 256 ? 2 : FAST || NEED_PARAMS ? 3 : 2)
backward_quad_kernel(const IO *__restrict__ x, const float *__restrict__ x_integ, const IO *__restrict__ grad_output, BoxParams bp, IO *__restrict__ grad_input,
                     float *__restrict__ partials, int N, int C, int F, int h, int w, int row_tiles, bool normalize, bool exact,
                     bool write_gin, Finish fin)
{
    using Q = QuadImage<CT>;
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int64_t nc = blockIdx.x;
    const int c = blockIdx.x % C, n = blockIdx.x / C;
    const int npix = h * w, cells = quad_cells(w), ntiles = row_tiles * CT;
    const QuadSmem s = quad_smem(smem4, h, CT, ntiles, nwarps);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));
    float *red = sTaps + F * kTapWords;                                                        // [F][warps][5]
    __shared__ uint32_t tmem_base;
    const IO *gbase = grad_output + nc * F * (int64_t)npix;
    const QuadTile tile = quad_tile<CT>(warp, lane, h);

    if (FAST && threadIdx.x == 0) bulk_prefetch_l2(gbase, (uint32_t)npix * (uint32_t)sizeof(IO));
    quad_zero_padding<CT>(s.image, h);
    grid_dependency_wait();
    const IO *xrow = x + nc * npix + tile.p0 * w;
    Rows8 g;
    if (NEED_PARAMS && x) rows8_load<IO, FAST>(g, xrow, w, tile.c, FAST ? kTileRows : tile.rows, lane);      // in flight meanwhile
    __syncwarp();
    if (warp == nwarps - 1) tmem_alloc(&tmem_base, tmem_columns(nwarps));
    if ((int)threadIdx.x < F) {
        const Box box = load_box(bp, c * F + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    __syncthreads();
    tmem_acquire();
    TmemRows<1> kept(tmem_base, warp);
    if (NEED_PARAMS) {
        if (!x) {
            // the caller has only the input's integral image: its pixels are second differences
            const float *I = x_integ + nc * (int64_t)(h + 1) * (w + 1) + (int64_t)tile.p0 * (w + 1);
            pixels_of_integral(I, w, tile.c, tile.c < w ? tile.rows : 0, [&](int i, const float4 &e) { kept.init(i, e); });
        } else {
#pragma unroll
            for (int i = 0; i < kTileRows; ++i) kept.init(i, rows8_get<IO, FAST>(g, xrow, w, tile.c, lane, i));
        }
    } else {
#pragma unroll
        for (int i = 0; i < kTileRows; ++i) kept.init(i, make_float4(0.f, 0.f, 0.f, 0.f));
    }
    kept.sync();
    for (int f = 0; f < F; ++f) {
        {
            QuadBlock v;
            float carry[kTileRows];
            quad_load_tile<IO, FAST, FAST>(v, tile, gbase + f * (int64_t)npix, w, lane);
            if (FAST && threadIdx.x == 0 && f + 1 < F)
                bulk_prefetch_l2(gbase + (f + 1) * (int64_t)npix, (uint32_t)npix * (uint32_t)sizeof(IO));
            quad_scan<CT>(v, carry, tile, s, warp, lane);
            if (CT > 1) __syncthreads();
            quad_publish<CT>(v, carry, tile, s, lane);
            __syncthreads();      // (also: every gather of the previous filter is done)
            quad_store<CT, FAST>(v, tile, s, w, lane);
        }
        __syncthreads();
        float sums[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
        const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
        quad_backward_strip<kTileRows, NEED_PARAMS, FAST, FAST && CT == 1 && MAXT <= 384>(t, quad_cols(t, tile.c >> 2, cells, Q::kCells),
                                                                                          quad_rows<kTileRows>(t, tile.p0, h, s.image, s.image, Q::kRow, lane),
                                                                                          col_weights(t), kept, sums, tile.rows);
        kept.sync();
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
            if (FAST || i < tile.rows) {
                const float4 g = kept.grad_input(i);
                float v[kStrip] = {g.x, g.y, g.z, g.w};
                store_row4<IO, FAST>(row, tile.c, w, v);
            }
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, tmem_columns(nwarps));
    if (COUNTED) finish_if_last(fin, partials, bp, c, C, F, normalize, exact);
}

// Backward of larger aligned planes (FAST in the kernel above), two tiles a warp: 18 to 32 tiles, two column tiles wide, take the
// whole of tensor memory for their input values and grad-input accumulators, and the SM; 14 and 16 tiles half of either.
// The 32 x 32-tile kernel, which had the former before, keeps accumulators in registers and reads the input plane again from L2 for every
// filter, and its tap loads conflict where rows are clamped at the plane's border.
// (8,16,4,128,256): 71 -> 51 us, bfloat16 (10,16,4,80,240): 105 -> 68.  Every warp has two whole tiles; asked whether it has, the compiler
// ran out of registers (456 bytes of spills, 64 us).
template <typename IO, int CT, bool NEED_PARAMS, bool COUNTED, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 2 : 1)
backward_quad_pair_kernel(const IO *__restrict__ x, const IO *__restrict__ grad_output, BoxParams bp, IO *__restrict__ grad_input,
                          float *__restrict__ partials, int N, int C, int F, int h, int w, int row_tiles, bool normalize, bool exact, bool write_gin, Finish fin)
{
    constexpr int T = 2;
    // (the scalar form spills 44 bytes here: with pairs 0.97 of the time over 5 sizes of up to 16 tiles, 0.995 over 73 larger ones; float 1.014)
    constexpr bool kPacked = CT == 2 && std::is_same<IO, __nv_bfloat16>::value;
    using Q = QuadImage<CT>;
    extern __shared__ float4 smem4[];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int64_t nc = blockIdx.x;
    const int c = blockIdx.x % C, n = blockIdx.x / C;
    const int npix = h * w, cells = quad_cells(w), ntiles = row_tiles * CT;
    const QuadSmem s = quad_smem(smem4, h, CT, ntiles, nwarps);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));
    float *red = sTaps + F * kTapWords;                                                        // [F][warps][5]
    __shared__ uint32_t tmem_base;
    const IO *gbase = grad_output + nc * F * (int64_t)npix;
    auto tile_of = [&](int k) { return quad_tile<CT>(warp + k * nwarps, lane, h); };      // (all of them exist, with all their rows)

    if (threadIdx.x == 0) bulk_prefetch_l2(gbase, (uint32_t)npix * (uint32_t)sizeof(IO));
    quad_zero_padding<CT>(s.image, h);
    grid_dependency_wait();
    __syncwarp();
    if (warp == nwarps - 1) tmem_alloc(&tmem_base, tmem_columns<T>(nwarps));
    if ((int)threadIdx.x < F) {
        const Box box = load_box(bp, c * F + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    __syncthreads();
    tmem_acquire();
#pragma unroll 1
    for (int k = 0; k < T; ++k) {
        const QuadTile t = tile_of(k);
        TmemRows<1, T> kept(tmem_base, warp, k);
        const IO *xrow = x + nc * npix + t.p0 * w;
        Rows8 g;
        if (NEED_PARAMS) rows8_load<IO, true>(g, xrow, w, t.c, kTileRows, lane);
#pragma unroll
        for (int i = 0; i < kTileRows; ++i)
            kept.init(i, NEED_PARAMS ? rows8_get<IO, true>(g, xrow, w, t.c, lane, i) : make_float4(0.f, 0.f, 0.f, 0.f));
        kept.sync();
    }
#pragma unroll 1
    for (int f = 0; f < F; ++f) {
        {
            QuadTile tile[T];
            QuadBlock v[T];
            float carry[T][kTileRows];
#pragma unroll
            for (int k = 0; k < T; ++k) {
                tile[k] = tile_of(k);
                quad_load_tile<IO, true, true>(v[k], tile[k], gbase + f * (int64_t)npix, w, lane);
            }
            if (threadIdx.x == 0 && f + 1 < F) bulk_prefetch_l2(gbase + (f + 1) * (int64_t)npix, (uint32_t)npix * (uint32_t)sizeof(IO));
#pragma unroll
            for (int k = 0; k < T; ++k)
                quad_scan<CT>(v[k], carry[k], tile[k], s, warp, lane);
            if (CT > 1) __syncthreads();
#pragma unroll
            for (int k = 0; k < T; ++k)
                quad_publish<CT>(v[k], carry[k], tile[k], s, lane);
            __syncthreads();      // (also: every gather of the previous filter is done)
#pragma unroll
            for (int k = 0; k < T; ++k)
                quad_store<CT, true>(v[k], tile[k], s, w, lane);
        }
        __syncthreads();
        const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
        float all[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
            const QuadTile tile = tile_of(k);
            TmemRows<1, T> kept(tmem_base, warp, k);
            float sums[kNumSums] = {0.f, 0.f, 0.f, 0.f, 0.f};
            quad_backward_strip<kTileRows, NEED_PARAMS, true, kPacked>(t, quad_cols(t, tile.c >> 2, cells, Q::kCells),
                                                                       quad_rows_later<kTileRows>(t, tile.p0, h, s.image, s.image, Q::kRow, lane),
                                                                       col_weights(t), kept, sums, kTileRows);
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
        __syncthreads();
        for (int i = threadIdx.x; i < F * kNumSums; i += blockDim.x) {
            const int f = i / kNumSums, j = i - f * kNumSums;
            float sum = 0.0f;
            for (int k = 0; k < nwarps; ++k) sum += red[(f * nwarps + k) * kNumSums + j];
            partials[((int64_t)(c * F + f) * N + n) * kNumSums + j] = sum;
        }
    }
    if (write_gin) {
#pragma unroll 1
        for (int k = 0; k < T; ++k) {
            const QuadTile tile = tile_of(k);
            TmemRows<1, T> kept(tmem_base, warp, k);
            IO *row = grad_input + nc * npix + tile.p0 * w;
#pragma unroll
            for (int i = 0; i < kTileRows; ++i, row += w) {
                const float4 g = kept.grad_input(i);
                if (tile.c < w) Io<IO>::store4(row + tile.c, g.x, g.y, g.z, g.w);
            }
        }
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, tmem_columns<T>(nwarps));
    if (COUNTED) finish_if_last(fin, partials, bp, c, C, F, normalize, exact);
}

inline int quad_row_tiles(int h) { return (h + kTileRows - 1) / kTileRows; }
inline int quad_col_tiles(int w) { return (w + 127) / 128; }
inline size_t quad_forward_smem(int F, int h, int w)
{
    const int ct = quad_col_tiles(w), tiles = quad_row_tiles(h) * ct;
    return (size_t)quad_image_bytes(h, ct) + tiles * (544 + kScanBytes) + F * kTapWords * 4;
}
inline size_t quad_backward_smem(int F, int h, int w)
{
    const size_t tiles = (size_t)quad_row_tiles(h) * quad_col_tiles(w);
    return quad_forward_smem(F, h, w) + F * tiles * kNumSums * 4;
}
// Narrower planes leave more than half of a warp's lanes idle and are better off in 32 x 32 tiles.
constexpr int kQuadMinWidth = 65;
// How many CTAs share a plane's filters, and its rows: planes of more than 16 tiles that leave SMs idle, CTAs that each
// gather a part of the rows from integral images of their own ((1,16,4,128,256), 64 -> 128 CTAs: 12.0 -> 9.8 us a block tail).
struct QuadSplit {
    int filters, rows;
};
inline QuadSplit quad_forward_split(int64_t planes, int F, int tiles)
{
    QuadSplit s{1, 1};
    if (F % 2 == 0 && planes < 148 * 6) s.filters = 2;
    while (s.filters < F && F % (s.filters * 2) == 0 && planes * s.filters * 2 <= 148 * 2) s.filters *= 2;
    while (tiles > 16 && planes * s.filters * s.rows * 2 <= 148 && s.rows < 4) s.rows *= 2;
    return s;
}

// Forward in tiles of 8 x 128 or of 32 x 32, where both fit?  A tile of either kind is 1024 pixels and a warp's work.
// Rows that vector accesses fit, and all rows of the tiles: as many tiles or fewer, which compares what is wasted past
// the plane ((8,16,4,128,256), 32 to 32: 31 us against 34; 448 planes of 48 x 120, F = 4, 6 to 8: 18 against 23; (4,16,4,96,160), 24 to
// 15: 16 against 11; 1032 planes of 64 x 80, F = 4, 8 to 6: 37 against 34), and launches that leave SMs idle, for the shorter
// chain of the 8 x 128 build.  Rows that no vector access fits are loaded and stored through shuffles, and cut rows at
// the bottom take guarded code: work that a single and nearly full column tile repays ((7,63,4,244,125), float16: 135 us
// against 170, (3,56,2,78,99): 13.5 against 17.5, (56,9,4,35,104): 21 against 23) and others do not ((27,26,4,31,162): 46 against 35;
// (5,7,3,37,69): 11 against 7.4; (37,5,4,34,68): 10.7 against 9.4), unless the CTA has its SM to itself either way, the rows are
// aligned and three quarters of the tiles' pixels exist ((3,38,6,63,216): 24 against 25; (117,5,8,68,92): 78 against 67).  A
// split by rows, which 32 x 32 tiles do not have, pays whatever the rows ((3,5,3,116,186): 12 against 21).
inline bool quad_prefers_forward(int64_t planes, int F, int h, int w)
{
    const int tiles = quad_row_tiles(h) * quad_col_tiles(w), square = ((h + 31) / 32) * ((w + 31) / 32);
    if (quad_forward_split(planes, F, tiles).rows > 1) return true;
    const bool few = planes * F <= 148, full = 4 * (int64_t)h * w >= 3 * (int64_t)tiles * 1024;
    if (w % 4 == 0 && h % kTileRows == 0) return tiles <= square || few;
    return (w > 96 && w <= 128 && (tiles <= 8 || full)) || (w % 4 == 0 && tiles > 8 && (full || few));
}
// The same from the plane's integral image, which both kernels copy, this one a row a warp at a time: large planes of two
// column tiles, and small ones of full rows (684 planes of 80 x 248, F = 3: 92 us against 110; 448 of 48 x 120, F = 4: 21
// against 25; (97,9,4,112,104): 177 against 107; 1024 planes of 64 x 128, F = 4: 62 against 55).
inline bool quad_prefers_forward_integ(int64_t planes, int F, int h, int w)
{
    if (!quad_prefers_forward(planes, F, h, w)) return false;
    const int tiles = quad_row_tiles(h) * quad_col_tiles(w), square = ((h + 31) / 32) * ((w + 31) / 32);
    if (quad_col_tiles(w) == 2) return tiles <= 8 || tiles > 16;
    return tiles <= 8 && tiles < square && w % 4 == 0 && h % kTileRows == 0;
}
inline bool quad_fits_forward(int F, int h, int w)
{
    const int tiles = quad_row_tiles(h) * quad_col_tiles(w);
    return w >= kQuadMinWidth && w <= 256 && F <= kMaxFilters && tiles <= 2 * kQuadMaxWarps && quad_forward_smem(F, h, w) <= kQuadMaxSmem;
}
inline bool quad_fits_backward(int F, int h, int w)
{
    return w >= kQuadMinWidth && w <= 256 && F <= kMaxFilters && quad_row_tiles(h) * quad_col_tiles(w) <= kQuadMaxWarps &&
           quad_backward_smem(F, h, w) <= kQuadMaxSmem;
}

// Threads at most of the pair kernel that is launched for a CTA of `warps` warps; 0: there is none.
inline int quad_pair_max_threads(int col_tiles, int warps)
{
    if (warps <= 8) return 256;
    return col_tiles == 2 && warps <= kQuadMaxWarps ? 512 : 0;
}

// Aligned planes with two tiles a warp, so with an even number of tiles.
// 18 to 32 tiles in two columns (one column of them has no kernel of more than eight warps: strips).  In 16 bits not where these tiles waste
// half as much again as square ones ((10,16,4,96,160), 24 tiles for 15: 67 us against 58 in those; (10,16,4,80,240), 20 for 24: 68 against 105); float
// always ((55,16,4,128,156): 274, 351; (30,16,2,88,188): 83, 121; (40,16,4,104,224): 215, 330).  Of at most 16 tiles of 32 x 32 (72 to 96 rows, 132 to 160
// columns) strips take 0.60 to 1.00 of the time for any number of planes ((37,1,4,80,132) 34.0 us, 21.5; (1300,1,4,80,144) 306, 198), and with three filters
// or more they have them (flat_beats_pair()).  With one or two the line by the number of planes is the one that was measured against 32 x 32 tiles, two
// planes an SM at about half the rate, where a round of 148 planes here has to save half a round there: the first and the third do.  Strips would gain
// there too: (148,1,2,72,136) 20.9, 18.2; (370,1,1,72,156) 36.6, 27.4.
// 14 and 16 tiles, which as one tile a warp have an SM to themselves: two CTAs of half the warps, if there are planes for two
// ((16,32,4,128,128): 94, 105; (16,32,4,64,256): 91, 108; (64,32,4,112,96): 258, 329).  Not of 10 and 12 tiles, two CTAs an SM either
// way ((16,32,4,96,128): 73, 68; (16,32,4,40,248): 71, 65).
// Two rules: of which sides and filters the kernel holds planes, and for how many planes it is the faster one of those with fixed tiles.
inline bool quad_pair_fits_backward(int F, int h, int w, bool wide)
{
    const int col_tiles = quad_col_tiles(w), tiles = quad_row_tiles(h) * col_tiles, square = ((h + 31) / 32) * ((w + 31) / 32);
    if (w < kQuadMinWidth || w > 256 || w % 4 || h % kTileRows || F > kMaxFilters || tiles % 2 || quad_backward_smem(F, h, w) > kQuadMaxSmem) return false;
    if (tiles <= kQuadMaxWarps) return tiles > 12;
    return col_tiles == 2 && tiles <= 2 * kQuadMaxWarps && (wide || 2 * tiles <= 3 * square);
}
inline bool quad_pair_suits_backward(int64_t planes, int F, int h, int w, bool wide)
{
    const int tiles = quad_row_tiles(h) * quad_col_tiles(w), square = ((h + 31) / 32) * ((w + 31) / 32);
    if (!quad_pair_fits_backward(F, h, w, wide)) return false;
    if (tiles <= kQuadMaxWarps) return planes > 148;
    return square > 16 || F >= 8 || planes <= 148 || (planes > 296 && planes <= 444);
}

template <typename IO>
int launch_forward_quad_t(const IO *x, const float *integ, const BoxParams &bp, const Fusion *fu, IO *out, int N, int C, int F, int h, int w,
                          bool normalize, bool exact, cudaStream_t s)
{
    const int row_tiles = quad_row_tiles(h), col_tiles = quad_col_tiles(w), tiles = row_tiles * col_tiles;
    const int64_t planes = (int64_t)N * C;
    const QuadSplit split = quad_forward_split(planes, F, tiles);
    const int fsplit = split.filters;
    if (planes * fsplit > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool fast = w % 4 == 0 && h % kTileRows == 0 && aligned_to(x, Io<IO>::kVecBytes) && aligned_to(out, Io<IO>::kVecBytes) &&
                      (!fu || !fu->residual || aligned_to(fu->residual, 16));
    const int T = tiles > 8 ? 2 : 1;
    // No row parts where the output lies over the input (one filter, in place): a CTA that starts late would integrate rows
    // that another has already replaced.
    const bool in_place = x && ranges_overlap(x, (size_t)planes * h * w * sizeof(IO), out, (size_t)planes * F * h * w * sizeof(IO));
    const int rsplit = in_place ? 1 : split.rows;
    const int warps = (tiles + T - 1) / T, nf = (F + fsplit - 1) / fsplit;
    // rows per task: few long tasks read fewer tap rows twice, but every warp should get the same share
    int chunk = 1;
    double best = 1e30;
    const int part_tiles = (row_tiles + rsplit - 1) / rsplit;
    for (int k = 1; k <= part_tiles; ++k) {
        const int tasks = nf * ((part_tiles + k - 1) / k) * col_tiles;
        const double cost = ((tasks + warps - 1) / warps) * (k * kTileRows + 2.0);
        if (cost < best) { best = cost; chunk = k; }
    }
    void (*kern)(const IO *, const float *, BoxParams, IO *, int, int, int, int, int, int, int, int, bool, bool, Fusion);
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
        if (cudaError_t e = launch_overlapped(kern, (unsigned)(planes * fsplit * rsplit), warps * 32, quad_forward_smem(nf, h, w), s, x, integ, bp, out,
                                              C, F, h, w, row_tiles, fsplit, rsplit, chunk, normalize, exact, fu ? *fu : none))
            return cuda_failed(e, "forward_quad");
    }
    return check_launch("forward_quad");
}

template <typename IO>
int launch_backward_quad_t(const IO *x, const float *x_integ, const IO *grad_output, const BoxParams &bp, float rep_h, float rep_w, int N, int C, int F,
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
    void (*kern)(const IO *, const float *, const IO *, BoxParams, IO *, float *, int, int, int, int, int, int, bool, bool, bool, Finish);
    const Finish fin = finish_here(bp, need_params, planes, planes * F * h * w, C, grad_params, grad_params_kind, need_mask, N, rep_h, rep_w, s);
    auto pick = [&](auto ct, auto counted) {
        constexpr int CT = decltype(ct)::value;
        constexpr bool K = decltype(counted)::value;
        auto sized = [&](auto threads) {
            constexpr int T = decltype(threads)::value;
            if (need_params) kern = fast ? backward_quad_kernel<IO, CT, true, true, K, T> : backward_quad_kernel<IO, CT, false, true, K, T>;
            else kern = fast ? backward_quad_kernel<IO, CT, true, false, false, T> : backward_quad_kernel<IO, CT, false, false, false, T>;
        };
        if (tiles <= 8) sized(Index<256>{});
        else if (tiles <= 12) sized(Index<384>{});      // registers for two CTAs an SM
        else sized(Index<512>{});
    };
    if (fin.total) col_tiles == 1 ? pick(Index<1>{}, Flag<true>{}) : pick(Index<2>{}, Flag<true>{});
    else col_tiles == 1 ? pick(Index<1>{}, Flag<false>{}) : pick(Index<2>{}, Flag<false>{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kQuadMaxSmem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_QUAD, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)planes, tiles * 32, quad_backward_smem(F, h, w), s, x, x_integ, grad_output, bp,
                                              grad_input, partials, N, C, F, h, w, row_tiles, normalize, exact, write_gin, fin))
            return cuda_failed(e, "backward_quad");
    }
    st = check_launch("backward_quad");
    if (st != BC_OK || !need_params || fin.total) return st;
    return launch_finish_param_grads<float>(partials, bp, C * F, N, normalize, exact, rep_h, rep_w, need_mask, grad_params, s,
                                            grad_params_kind);
}

template <typename IO>
int launch_backward_quad_pair_t(const IO *x, const IO *grad_output, const BoxParams &bp, float rep_h, float rep_w, int N, int C, int F, int h, int w,
                                bool normalize, bool exact, int need_mask, IO *grad_input, void *grad_params, int grad_params_kind, float *partials,
                                cudaStream_t s)
{
    const int row_tiles = quad_row_tiles(h);
    const int64_t planes = (int64_t)N * C;
    if (planes > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool need_params = (need_mask & (BC_NEED_ALL & ~BC_NEED_INPUT)) != 0, write_gin = (need_mask & BC_NEED_INPUT) != 0;
    const Finish fin = finish_here(bp, need_params, planes, planes * F * h * w, C, grad_params, grad_params_kind, need_mask, N, rep_h, rep_w, s);
    void (*kern)(const IO *, const IO *, BoxParams, IO *, float *, int, int, int, int, int, int, bool, bool, bool, Finish);
    auto pick = [&](auto ct, auto threads) {
        constexpr int CT = decltype(ct)::value, T = decltype(threads)::value;
        kern = !need_params ? backward_quad_pair_kernel<IO, CT, false, false, T>
               : fin.total  ? backward_quad_pair_kernel<IO, CT, true, true, T>
                            : backward_quad_pair_kernel<IO, CT, true, false, T>;
    };
    const int col_tiles = quad_col_tiles(w), warps = row_tiles * col_tiles / 2, bound = quad_pair_max_threads(col_tiles, warps);
    if (!bound) return BC_ERR_UNSUPPORTED;
    if (bound == 512) pick(Index<2>{}, Index<512>{});
    else if (col_tiles == 2) pick(Index<2>{}, Index<256>{});
    else pick(Index<1>{}, Index<256>{});
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), (int)kQuadMaxSmem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_QUAD_PAIR, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)planes, warps * 32, quad_backward_smem(F, h, w), s, x, grad_output, bp, grad_input, partials,
                                              N, C, F, h, w, row_tiles, normalize, exact, write_gin, fin))
            return cuda_failed(e, "backward_quad_pair");
    }
    st = check_launch("backward_quad_pair");
    if (st != BC_OK || !need_params || fin.total) return st;
    return launch_finish_param_grads<float>(partials, bp, C * F, N, normalize, exact, rep_h, rep_w, need_mask, grad_params, s, grad_params_kind);
}

}  // namespace

}  // namespace bc
