// Whole-plane forward with the column-combined rows in tensor memory.
//
// The gather of the quad kernels reads five words of shared memory an output: ten taps of a pair of tap rows give four
// outputs, and every tap row is read twice, once as the row at the box's upper border and, rows later, as the one at its
// lower border.  Here a filter's combination of the ten taps, D(a, q), is worked out once per row a and kept, so that an
// output costs half the words of the shared-memory pipe, which bounds that kernel.  D is the size of a plane; written to
// shared memory and read back it would cost what it saves, but tensor memory (bc_tmem.cuh) has a pipe of its own: a
// row's four columns a lane are stored as they are made and loaded twice, by rows of any offset, since the row is the
// tensor memory's column.
//
// What tensor memory asks for: a warp reaches the 32 lanes of its number modulo 4, so all rows of a (filter, column tile
// of 128) have to be made and read by warps of the same number modulo 4.  Four such units are worked on at a time, each
// by a quarter of the CTA's warps, which split the rows; a barrier among them stands between the rows' making and their
// use.  A unit occupies 4 h columns of its lanes: planes of up to 128 rows.  CTAs allocate after they have built the
// integral image and free behind the last unit, so CTAs that wait for tensor memory have their planes on the way.
#pragma once
#include <algorithm>

#include "box_quad_plane.cuh"

namespace bc {

namespace {

constexpr int kTmemMaxRows = 128;

// Barrier among `threads` threads of the CTA; those that only arrive do not wait.  The instructions count whole warps and ask for
// converged ones, and some lanes come from a store that others, past the plane, did not make.
__device__ __forceinline__ void unit_barrier(int id, int threads)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void unit_arrive(int id, int threads)
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// What the warps of a unit share: integral row a (1 .. h) of the unit is at the columns 4 (a - 1) .. of `rows32`.
struct TmemUnit {
    uint32_t rows32;
    int r_begin, r_end, h;      // the warp's rows
};

// The warp's rows of D for the columns from q0 on.
template <int CT>
__device__ __forceinline__ void tmem_make_rows(const TmemUnit &n, const BoxTaps &t, uint32_t image, int q0, int cells)
{
    using Q = QuadImage<CT>;
    const QuadCols cols = quad_cols(t, q0 >> 2, cells, Q::kCells);
    const ColW2 cw = col_weights(t);
    const float nfl = -t.f_lo_c;
    for (int r = n.r_begin; r < n.r_end; r += kTileRows) {
        QuadCols at = cols;
#pragma unroll
        for (int m = 0; m <= kStrip; ++m) {
            at.lo[m] += image + (r + 1) * Q::kRow;
            at.hi[m] += image + (r + 1) * Q::kRow;
        }
        auto two_rows = [&](auto I) {
            constexpr int i = decltype(I)::value;
            f2_t l[kStrip + 1], g[kStrip + 1];
            float lo[2][kStrip], sum[2][kStrip];
#pragma unroll
            for (int m = 0; m <= kStrip; ++m) {
                l[m] = pack2(lds<i * Q::kRow>(at.lo[m]), lds<(i + 1) * Q::kRow>(at.lo[m]));
                g[m] = pack2(lds<i * Q::kRow>(at.hi[m]), lds<(i + 1) * Q::kRow>(at.hi[m]));
            }
            // (the last step by itself for either row: its results go where the store wants them)
#pragma unroll
            for (int m = 0; m < kStrip; ++m) {
                unpack2(l[m], lo[0][m], lo[1][m]);
                unpack2(fma2(cw.nwl, l[m + 1], fma2(cw.fh, g[m + 1], mul2(cw.wh, g[m]))), sum[0][m], sum[1][m]);
            }
            float4 a, b;
            a.x = fmaf(nfl, lo[0][0], sum[0][0]); a.y = fmaf(nfl, lo[0][1], sum[0][1]);
            a.z = fmaf(nfl, lo[0][2], sum[0][2]); a.w = fmaf(nfl, lo[0][3], sum[0][3]);
            b.x = fmaf(nfl, lo[1][0], sum[1][0]); b.y = fmaf(nfl, lo[1][1], sum[1][1]);
            b.z = fmaf(nfl, lo[1][2], sum[1][2]); b.w = fmaf(nfl, lo[1][3], sum[1][3]);
            __syncwarp();
            tmem_store8(n.rows32 + 4 * (r + i), a, b);
        };
        two_rows(Index<0>{}); two_rows(Index<2>{}); two_rows(Index<4>{}); two_rows(Index<6>{});
    }
    tmem_wait_store();
}

// The warp's output rows from the unit's rows of D; `row`: the first of them.
template <typename IO>
__device__ __forceinline__ void tmem_use_rows(const TmemUnit &n, const BoxTaps &t, IO *row, int q0, int w)
{
    const float sfl = t.scale * t.f_lo_r, sfh = t.scale * t.f_hi_r;
    const f2_t scale2 = pack2(t.scale, t.scale), sfl2 = pack2(sfl, sfl), sfh2 = pack2(sfh, sfh);
    // The integral rows a .. a+3 combined (row 0 is zero, rows past the plane repeat its last).  Zero times the columns' weights:
    // a box whose sides are no numbers gives none in the rows above the plane either.
    const float none = 0.0f * t.f_lo_c + 0.0f * t.f_hi_c;
    const float4 row0 = make_float4(none, none, none, none);
    auto fetch = [&](float4 (&v)[4], int a) {
        __syncwarp();
        if (a >= 1 && a + 3 <= n.h) {
            tmem_load16(n.rows32 + 4 * (a - 1), v);
            tmem_wait_load(v);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) tmem_load4(n.rows32 + 4 * (min(max(a + i, 1), n.h) - 1), v[i]);
            tmem_wait_load(v);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (a + i < 1) v[i] = row0;
        }
    };
    if (n.r_begin >= n.r_end) return;
    float4 A, B;      // the rows at lo-1 and hi, which are those at lo and hi+1 of the row above
    {
        const int a = n.r_begin + t.lo_r - 1, b = n.r_begin + t.hi_r;
        __syncwarp();
        tmem_load4(n.rows32 + 4 * (min(max(a, 1), n.h) - 1), A);
        tmem_load4(n.rows32 + 4 * (min(max(b, 1), n.h) - 1), B);
        tmem_wait_load(A, B);
        if (a < 1) A = row0;
        if (b < 1) B = row0;
    }
#pragma unroll 1
    for (int p = n.r_begin; p < n.r_end; p += 4) {
        float4 L[4], H[4];      // those at lo and hi+1
        fetch(L, p + t.lo_r);
        fetch(H, p + t.hi_r + 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float v[kStrip];
            auto pair = [&](f2_t a, f2_t b, f2_t lo, f2_t hi, float &v0, float &v1) {
                const f2_t mid = mul2(sub2(b, lo), scale2);
                unpack2(fma2(sfl2, sub2(lo, a), fma2(sfh2, sub2(hi, b), mid)), v0, v1);
            };
            pair(pack2(A.x, A.y), pack2(B.x, B.y), pack2(L[i].x, L[i].y), pack2(H[i].x, H[i].y), v[0], v[1]);
            pair(pack2(A.z, A.w), pack2(B.z, B.w), pack2(L[i].z, L[i].w), pack2(H[i].z, H[i].w), v[2], v[3]);
            if (q0 < w) Io<IO>::store4(row + q0, v[0], v[1], v[2], v[3]);
            row += w;
            A = L[i];
            B = H[i];
        }
    }
}

__device__ __forceinline__ TmemUnit tmem_unit(uint32_t tmem_base, int lanes, int part, int parts, int row_tiles, int h)
{
    const int part_rows = (row_tiles + parts - 1) / parts * kTileRows, r_begin = part * part_rows;
    return TmemUnit{tmem_base + ((uint32_t)lanes << 21), r_begin, min(r_begin + part_rows, h), h};
}

// One plane a CTA: planes of which an SM's shared memory holds one.  T: tiles a warp holds while it builds.
template <typename IO, int CT, int T>
__global__ void __launch_bounds__(512)
forward_tmem_kernel(const IO *__restrict__ x, BoxParams bp, IO *__restrict__ out, int C, int F, int h, int w, int row_tiles, uint32_t tmem_columns,
                    bool normalize, bool exact)
{
    extern __shared__ float4 smem4[];
    __shared__ uint32_t tmem_base;
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int c = blockIdx.x % C;
    const int64_t npix = (int64_t)h * w, nc = blockIdx.x;
    const int cells = quad_cells(w), ntiles = row_tiles * CT;
    const QuadSmem s = quad_smem(smem4, h, CT, ntiles, nwarps);
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + (s.taps - s.image));

    quad_zero_padding<CT>(s.image, h);
    grid_dependency_wait();
    {
        QuadTile tile[T];
        QuadBlock v[T];
        float carry[T][kTileRows];
#pragma unroll
        for (int k = 0; k < T; ++k) {
            tile[k] = quad_tile<CT>(warp + k * nwarps, lane, h);
            if (tile[k].rows) quad_load_tile<IO, true, true>(v[k], tile[k], x + nc * npix, w, lane);
        }
        if ((int)threadIdx.x < F) {
            const Box box = load_box(bp, c * F + threadIdx.x);
            store_taps(sTaps + threadIdx.x * kTapWords, taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
        }
#pragma unroll
        for (int k = 0; k < T; ++k)
            if (tile[k].rows) quad_scan<CT>(v[k], carry[k], tile[k], s, warp, lane);
        if (CT > 1) __syncthreads();
#pragma unroll
        for (int k = 0; k < T; ++k)
            if (tile[k].rows) quad_publish<CT>(v[k], carry[k], tile[k], s, lane);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < T; ++k)
            if (tile[k].rows) quad_store<CT, true>(v[k], tile[k], s, w, lane);
    }
    __syncwarp();
    if (warp == nwarps - 1) tmem_alloc(&tmem_base, tmem_columns);
    __syncthreads();
    tmem_acquire();

    const int lanes = warp & 3, parts = nwarps >> 2;
    const TmemUnit unit = tmem_unit(tmem_base, lanes, warp >> 2, parts, row_tiles, h);
    for (int u = lanes; u < F * CT; u += 4) {
        const int f = u / CT, q0 = (u - f * CT) * 128 + lane * kStrip;
        const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
        if (u != lanes) {      // the rows of the unit before have been read
            tmem_release();
            unit_barrier(1 + lanes, parts * 32);
            tmem_acquire();
        }
        tmem_make_rows<CT>(unit, t, s.image, q0, cells);
        tmem_release();
        unit_barrier(1 + lanes, parts * 32);
        tmem_acquire();
        tmem_use_rows<IO>(unit, t, out + (nc * F + f) * npix + (int64_t)unit.r_begin * w, q0, w);
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, tmem_columns);
}

// A stream of planes a CTA: half of its warps build integral images, one ahead of the other half, which gather.  An SM
// runs no more CTAs than tensor memory holds, two here, so a CTA has to cover by itself what a plane's way from memory takes (5000 of
// the 18000 cycles a plane took one after the other).
// W: warps of either half, and tiles of a plane at most.  Named barriers: 1 .. 4 units, 5 the building warps', 6 and 7 image built,
// 8 and 9 image read.
template <typename IO, int CT, int W>
__global__ void __launch_bounds__(64 * W, W == 8 ? 2 : 1)
forward_tmem_stream_kernel(const IO *__restrict__ x, BoxParams bp, IO *__restrict__ out, int planes, int C, int F, int h, int w, int row_tiles,
                           uint32_t tmem_columns, bool normalize, bool exact)
{
    extern __shared__ float4 smem4[];
    __shared__ uint32_t tmem_base;
    __shared__ __align__(16) float sTaps[2][kMaxFilters * kTapWords];
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5);
    const int64_t npix = (int64_t)h * w;
    const int cells = quad_cells(w), ntiles = row_tiles * CT, image_bytes = quad_image_bytes(h, CT);
    QuadSmem s = quad_smem(smem4, h, CT, ntiles, W);      // of the first image; behind it the second one's, then the scan corners
    const uint32_t other = image_bytes + ntiles * 544;
    s.scan = s.image + 2 * other;

    quad_zero_padding<CT>(s.image, h);
    quad_zero_padding<CT>(s.image + other, h);
    grid_dependency_wait();
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmem_base, tmem_columns);
    __syncthreads();
    tmem_acquire();

    const int count = (planes - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    if (warp >= W) {
        const QuadTile tile = quad_tile<CT>(warp - W, lane, h);
        for (int k = 0; k < count; ++k) {
            const int64_t nc = blockIdx.x + (int64_t)k * gridDim.x;
            const int b = k & 1;
            if (k + 1 == count) grid_dependency_release();      // (any earlier, and the next kernel's CTAs would wait on SMs that are still at work)
            QuadSmem at = s;
            at.image += b * other; at.col += b * other; at.row += b * other;
            QuadBlock v;
            float carry[kTileRows];
            if (tile.rows) {
                quad_load_tile<IO, true, true>(v, tile, x + nc * npix, w, lane);
                quad_scan<CT>(v, carry, tile, at, warp - W, lane);
            }
            if (CT > 1) unit_barrier(5, W * 32);
            if (tile.rows) quad_publish<CT>(v, carry, tile, at, lane);
            unit_barrier(5, W * 32);
            if (k >= 2) unit_barrier(8 + b, 64 * W);
            if (tile.rows) quad_store<CT, true>(v, tile, at, w, lane);
            const int f = threadIdx.x - W * 32;
            if (f < F) {
                const Box box = load_box(bp, (int)(nc % C) * F + f);
                store_taps(sTaps[b] + f * kTapWords, taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
            }
            unit_arrive(6 + b, 64 * W);
        }
    } else {
        const int lanes = warp & 3, parts = W >> 2;
        const TmemUnit unit = tmem_unit(tmem_base, lanes, warp >> 2, parts, row_tiles, h);
        for (int k = 0; k < count; ++k) {
            const int64_t nc = blockIdx.x + (int64_t)k * gridDim.x;
            const int b = k & 1;
            tmem_release();
            unit_barrier(6 + b, 64 * W);      // (also: the rows of the plane before have been read)
            tmem_acquire();
            if (lanes >= F * CT && k + 2 < count) unit_arrive(8 + b, 64 * W);
            for (int u = lanes; u < F * CT; u += 4) {
                const int f = u / CT, q0 = (u - f * CT) * 128 + lane * kStrip;
                const BoxTaps t = load_taps_uniform(sTaps[b] + f * kTapWords);
                if (u != lanes) {
                    tmem_release();
                    unit_barrier(1 + lanes, parts * 32);
                    tmem_acquire();
                }
                tmem_make_rows<CT>(unit, t, s.image + b * other, q0, cells);
                if (u + 4 >= F * CT && k + 2 < count) unit_arrive(8 + b, 64 * W);
                tmem_release();
                unit_barrier(1 + lanes, parts * 32);
                tmem_acquire();
                tmem_use_rows<IO>(unit, t, out + (nc * F + f) * npix + (int64_t)unit.r_begin * w, q0, w);
            }
        }
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, tmem_columns);
}

inline int tmem_forward_warps(int h, int w) { return quad_row_tiles(h) * quad_col_tiles(w) <= 8 ? 8 : 16; }
// (every warp that builds has a scan corner, whether it has a tile or not)
inline size_t tmem_forward_smem(int F, int h, int w)
{
    const int ct = quad_col_tiles(w);
    return (size_t)quad_image_bytes(h, ct) + quad_row_tiles(h) * ct * 544 + tmem_forward_warps(h, w) * kScanBytes + F * kTapWords * 4;
}
inline size_t tmem_stream_smem(int h, int w)
{
    const int ct = quad_col_tiles(w);
    return 2 * ((size_t)quad_image_bytes(h, ct) + quad_row_tiles(h) * ct * 544) + tmem_forward_warps(h, w) * kScanBytes;
}

// Which planes: rows and tensors aligned for vector accesses, heights a multiple of 8 (with guarded rows the quad kernel is
// as fast: (110,16,4,41,116): 63 us here, 59 there; (129,16,4,32,104): 33 and 37).  Enough planes, as their filters are not
// split over CTAs ((4,16,4,48,216): 10.9 us, 8.3; (5,16,4,40,232): 10.4, 11.8), and where an SM runs one streaming CTA not a little
// more than one round of them ((13,16,4,64,228): 23.9 us, 22.8; (154,16,4,72,120): 93, 108).  (256,32,4,64,128): 273 -> 230 us;
// (8,16,4,128,256): 30.5 -> 22.
// A second column tile that is not mostly empty: up to 160 columns 32 x 32 tiles waste less (planes x filters x rows x columns,
// here and there: 2878 x 4 x 96 x 160: 318 us, 205; 340 x 6 x 80 x 160: 56, 44; 510 x 6 x 32 x 160: 26, 23; 1321 x 8 x 104 x 160 the other way:
// 248, 262; from 164 to 192 columns 0.90 of the time at the median of 148 sizes).
// At least three of the four quarters of tensor memory at work.  Three of them, over more than one plane an SM, only where few
// lanes idle as well, or the plane has but three units (1171 x 3 x 128 x 172, bfloat16: 164 us, 124; 2332 x 6 x 24 x 84: 52, 41;
// 191 x 3 x 24 x 228: 10.8, 8.2; but 147 x 3 x 104 x 72: 9.5, 12.9).
// One or two rows of tiles, which leave a gathering warp eight rows or none, in two columns: many filters, or the
// quad kernel's shorter chain wins (228 x 2 x 8 x 188: 5.7 us, 4.8; 188 x 4 x 8 x 208: 7.3, 6.2; 184 x 2 x 16 x 244: 7.0, 6.1; 260 x 16 x 8 x 256: 13.9, 19.5;
// 604 x 6 x 16 x 164: 18.9, 20.9).
inline bool tmem_suits_forward(int64_t planes, int F, int h, int w)
{
    const int ct = quad_col_tiles(w), tiles = quad_row_tiles(h) * ct, units = F * ct;
    if (h % kTileRows || w % 4 || w < kQuadMinWidth || w > 256 || (ct > 1 && w <= 160) || h > kTmemMaxRows || F > kMaxFilters || planes < 74) return false;
    if (4 * units < 3 * ((units + 3) / 4 * 4)) return false;
    if (units % 4 && planes > 148 && !(units == 3 && w > 96) && 10 * w < 9 * 128 * ct) return false;
    if (ct > 1 && h <= 2 * kTileRows && (F < 6 || (h == kTileRows && w <= 200))) return false;
    if (tiles > 16) return tiles <= 2 * kQuadMaxWarps && tmem_forward_smem(F, h, w) <= kQuadMaxSmem;
    return tmem_stream_smem(h, w) <= kQuadMaxSmem && (tiles <= 8 || planes <= 148 || planes > 222);
}

template <typename IO>
int launch_forward_tmem_t(const IO *x, const BoxParams &bp, IO *out, int N, int C, int F, int h, int w, bool normalize, bool exact, cudaStream_t s)
{
    const int row_tiles = quad_row_tiles(h), col_tiles = quad_col_tiles(w), tiles = row_tiles * col_tiles;
    const int64_t planes = (int64_t)N * C;
    if (planes > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const int warps = tmem_forward_warps(h, w);
    uint32_t columns = 32;      // (a power of two)
    while (columns < (uint32_t)(h * kStrip)) columns *= 2;
    void (*kern)(const IO *, BoxParams, IO *, int, int, int, int, int, uint32_t, bool, bool) = nullptr;
    void (*flow)(const IO *, BoxParams, IO *, int, int, int, int, int, int, uint32_t, bool, bool) = nullptr;
    auto pick = [&](auto ct) {
        constexpr int CT = decltype(ct)::value;
        if (tiles <= 8) flow = forward_tmem_stream_kernel<IO, CT, 8>;
        else if (tiles <= 16) flow = forward_tmem_stream_kernel<IO, CT, 16>;
        else if constexpr (CT == 2) kern = forward_tmem_kernel<IO, CT, 2>;      // (128 rows of one column tile are 16 tiles)
    };
    if (col_tiles == 1) pick(Index<1>{});
    else pick(Index<2>{});
    int st = raise_smem_limit(flow ? reinterpret_cast<const void *>(flow) : reinterpret_cast<const void *>(kern), (int)kQuadMaxSmem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(flow ? KID_FORWARD_TMEM_STREAM : KID_FORWARD_TMEM, s);
        const int64_t ctas = std::min<int64_t>(planes, warps == 8 ? 2 * 148 : 148);
        const cudaError_t e = flow ? launch_overlapped(flow, (unsigned)ctas, 2 * warps * 32, tmem_stream_smem(h, w), s, x, bp, out, (int)planes, C, F, h, w,
                                                       row_tiles, columns, normalize, exact)
                                   : launch_overlapped(kern, (unsigned)planes, warps * 32, tmem_forward_smem(F, h, w), s, x, bp, out, C, F, h, w, row_tiles,
                                                       columns, normalize, exact);
        if (e) return cuda_failed(e, "forward_tmem");
    }
    return check_launch("forward_tmem");
}

}  // namespace

}  // namespace bc
