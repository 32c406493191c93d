// Strips of 8 rows x 4 columns dealt out to lanes in one sequence: sample after sample of a channel, row group after row
// group of a plane, strip after strip of a row group.  A warp's tile is 32 of them, whatever the plane's width: no lane works
// past the plane's last column and only the last row group's and the last tile's lanes on nothing, where tiles of 8 x 128 or 32 x 32 pixels
// leave up to three quarters of a warp idle (34 x 49 pixels: 65 strips, 2.03 tiles; 2 x 2 = 4 tiles of 32 x 32).
//
// Integral images have the quad layout's sub-rows (bc_quad.cuh): column c of a row is word (c & 3) * P + (c >> 2) + 2 of it,
// P = strips + 4 cells: two zero cells in front (columns -8 .. -1), two that repeat the value at w behind, so that of a
// window of five taps the clamped first cell fixes all.  Rows of a row group are 4 P words apart and row groups 8 rows and S mod 32
// words (S strips a row), planes such that the next plane's first strip goes on where the last one ended: the 32 lanes of a
// warp read and write 32 different banks although they work on several rows or planes.
#pragma once
#include "bc_quad.cuh"
#include "bc_tile_io.cuh"
#include "bc_tmem.cuh"

namespace bc {

namespace {

constexpr int kFlatRows = 8;

struct FlatShape {
    int strips, groups, cells;      // a row's strips, a plane's row groups, their product
    int planes, tiles;              // planes a CTA works on together, tiles of its warps
    int sub, row, skew, plane;      // bytes of a sub-row, from row to row, added from row group to row group, from plane to plane
    int last;                       // offset of the plane's last row
    bool spans;                     // a row may reach over several tiles
    int split, columns;             // CTAs that share a plane's filters, a cluster; columns of tensor memory of each
    int offset[16];                 // of rows 0 .. 15: kernels read it from their parameters, one load instead of two or three operations
};

__host__ __device__ inline int flat_strips(int w) { return (w + 3) / 4; }
__host__ __device__ inline int flat_groups(int h) { return (h + kFlatRows - 1) / kFlatRows; }
__host__ __device__ inline int flat_row_at(int a, int row, int skew) { return a * row + (a >> 3) * skew; }      // (a may be negative)

inline FlatShape flat_shape(int h, int w, int planes)
{
    FlatShape s;
    s.strips = flat_strips(w);
    s.groups = flat_groups(h);
    s.cells = s.strips * s.groups;
    s.planes = planes;
    s.tiles = (s.cells * planes + 31) / 32;
    s.sub = (s.strips + 4) * 4;
    s.row = 4 * s.sub;
    s.skew = 4 * (s.strips & 31);
    s.last = flat_row_at(h, s.row, s.skew);
    const int words = (s.last + s.row) / 4;
    s.plane = 4 * (words + ((s.cells - words) & 31));
    s.spans = 32 % s.strips != 0;
    s.split = 1;
    s.columns = 0;
    for (int a = 0; a < 16; ++a) s.offset[a] = flat_row_at(a, s.row, s.skew);
    return s;
}

// Shared memory: images, what a tile's columns add to the tiles below (512 bytes), its last row's part (32), a scan corner a warp, boxes.
// With two tiles a warp its corner is where it will publish both tiles' columns.
constexpr int kFlatScanPitch = 144, kFlatScanBytes = 8 * kFlatScanPitch;
__host__ __device__ inline int flat_image_bytes(const FlatShape &s) { return (s.planes * s.plane + 15) & ~15; }
inline size_t flat_smem(const FlatShape &s, int tiles_a_warp, int F)
{
    return (size_t)flat_image_bytes(s) + s.tiles * (544 + (tiles_a_warp == 1 ? kFlatScanBytes : 0)) + F * kTapWords * 4;
}
struct FlatSmem {
    uint32_t image, col, row, scan, taps;
};
template <int T>
__device__ __forceinline__ FlatSmem flat_smem_at(const void *base, const FlatShape &sh)
{
    FlatSmem s;
    s.image = smem_u32(base);
    asm volatile("" : "+r"(s.image));
    s.col = s.image + flat_image_bytes(sh);
    s.row = s.col + sh.tiles * 512;
    s.scan = s.row + sh.tiles * 32;
    s.taps = s.scan + (T == 1 ? sh.tiles * kFlatScanBytes : 0);
    return s;
}

// A lane's strip.
struct FlatCell {
    int plane, group, strip, rows;      // rows inside the plane; 0: there is no such strip
};
__device__ __forceinline__ FlatCell flat_cell(const FlatShape &sh, int q, int planes, int h)
{
    FlatCell c;
    c.plane = q / sh.cells;
    const int rest = q - c.plane * sh.cells;
    c.group = rest / sh.strips;
    c.strip = rest - c.group * sh.strips;
    c.rows = min(kFlatRows, h - c.group * kFlatRows);
    if (c.plane >= planes) c.plane = c.group = c.rows = 0;
    return c;
}

// In one register, for kernels with several a lane (at most 1024 strips a plane and 255 planes).
__device__ __forceinline__ uint32_t flat_pack(const FlatCell &c) { return (uint32_t)c.strip | (uint32_t)c.group << 10 | (uint32_t)c.plane << 20 | (uint32_t)c.rows << 28; }
__device__ __forceinline__ FlatCell flat_unpack(uint32_t v)
{
    return FlatCell{(int)(v >> 20 & 0xff), (int)(v >> 10 & 0x3ff), (int)(v & 0x3ff), (int)(v >> 28)};
}

// What never changes in the images: row 0, and the first two cells and column 0 of every row.
__device__ __forceinline__ void flat_zero_padding(uint32_t image, const FlatShape &sh, int planes, int h)
{
    for (int g = 0; g < planes; ++g, image += sh.plane) {
        for (int i = threadIdx.x; i < sh.row / 4; i += blockDim.x) sts<0>(image + i * 4, 0.f);
        for (int i = threadIdx.x; i < h * 4; i += blockDim.x) {
            const uint32_t at = image + flat_row_at(1 + (i >> 2), sh.row, sh.skew) + (i & 3) * sh.sub;
            sts<0>(at, 0.f); sts<4>(at, 0.f);
            if ((i & 3) == 0) sts<8>(at, 0.f);
        }
    }
}

// ---- a strip's eight rows of four columns from and to memory ----------------------------------------
// Rows of any alignment as in bc_tile_io.cuh: a lane loads the aligned groups in which its columns begin and the k elements that it lacks come
// from the next lane by shuffle; the last lane of a row, or of the warp, loads the next group itself.
struct FlatBlock {
    f2_t a[kFlatRows], b[kFlatRows];      // columns c, c+1 and c+2, c+3
};
// PLAIN: the kernel may write the rows later.
template <typename IO, bool VEC, bool PLAIN = false>
__device__ __forceinline__ void flat_load(FlatBlock &v, const IO *row0, int w, const FlatCell &cell, int lane, int strips)
{
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const int c = cell.strip * 4;
    const IO *p = row0 + c;
    auto load = [](const IO *at) {
        if constexpr (PLAIN) return Io<IO>::load4_plain(at);
        else return Io<IO>::load4(at);
    };
    if (VEC) {
        float4 e[kFlatRows];
#pragma unroll
        for (int i = 0; i < kFlatRows; ++i, p += w) e[i] = i < cell.rows ? load(p) : zero;
#pragma unroll
        for (int i = 0; i < kFlatRows; ++i) { v.a[i] = pack2(e[i].x, e[i].y); v.b[i] = pack2(e[i].z, e[i].w); }
        return;
    }
    const bool end = lane == 31 || cell.strip == strips - 1;
    const int k0 = row_shift(row0);
    float4 e[kFlatRows], next[kFlatRows];
#pragma unroll
    for (int i = 0; i < kFlatRows; ++i, p += w) {
        const int k = (k0 + i * w) & 3;
        e[i] = i < cell.rows ? load(p - k) : zero;
        next[i] = end && k && i < cell.rows && c + 4 - k < w ? load(p + 4 - k) : zero;
    }
#pragma unroll
    for (int i = 0; i < kFlatRows; ++i) {
        const int k = (k0 + i * w) & 3;
        const bool one = k & 1, two = k & 2;
        float4 a = e[i];
        float n0 = __shfl_down_sync(0xffffffffu, a.x, 1);
        if (end) n0 = next[i].x;
        if (one) a = make_float4(a.y, a.z, a.w, n0);
        float m0 = __shfl_down_sync(0xffffffffu, a.x, 1), m1 = __shfl_down_sync(0xffffffffu, a.y, 1);
        if (end) {
            m0 = one ? next[i].y : next[i].x;
            m1 = one ? next[i].z : next[i].y;
        }
        if (two) a = make_float4(a.z, a.w, m0, m1);
        if (c + 1 >= w) a.y = 0.f;
        if (c + 2 >= w) a.z = 0.f;
        if (c + 3 >= w) a.w = 0.f;
        v.a[i] = pack2(a.x, a.y);
        v.b[i] = pack2(a.z, a.w);
    }
}

// ---- building the integral images -------------------------------------------------------------------
// First part: a strip's own prefix sums, and `carry`: what the strips to its left add to its rows, as far as they are in the same tile.  Eight
// rows at once through the warp's corner, four lanes a row with eight strips each; `starts`: the lanes that begin a row.
// With rows over several tiles the sum of the tile's last row part is published (followed by a barrier).
template <int T>
__device__ __forceinline__ void flat_scan(FlatBlock &v, float (&carry)[kFlatRows], const FlatSmem &s, int tile, uint32_t starts, bool spans, int warp, int nwarps, int lane)
{
    constexpr int kPitch = T == 1 ? kFlatScanPitch : 128;
    const uint32_t half[2] = {T == 1 ? s.scan + warp * kFlatScanBytes : s.col + warp * 512,
                              T == 1 ? s.scan + warp * kFlatScanBytes + 4 * kPitch : s.col + (warp + nwarps) * 512};
#pragma unroll
    for (int i = 1; i < kFlatRows; ++i) { v.a[i] = add2(v.a[i], v.a[i - 1]); v.b[i] = add2(v.b[i], v.b[i - 1]); }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kFlatRows; ++i) {
        float x, y, z, u;
        unpack2(v.a[i], x, y);
        unpack2(v.b[i], z, u);
        y += x; z += y; u += z;
        v.a[i] = pack2(x, y);
        v.b[i] = pack2(z, u);
        sts<0>(half[i >> 2] + (i & 3) * kPitch + lane * 4, u);
    }
    __syncwarp();
    const int k = lane & 3;
    const uint32_t mine = half[lane >> 4] + (lane >> 2 & 3) * kPitch + k * 32;
    const float4 p = lds128(mine), q = lds128(mine + 16);
    float e[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
    const uint32_t begin = (starts >> (8 * k)) & 0xffu;
    // (sums of what is in front, never an inclusive sum less a strip's own: that would leave its infinity or its rounding to its left)
    float run = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float own = e[j];
        if (begin & (1u << j)) run = 0.f;
        e[j] = run;
        run += own;
    }
    const int row_lane = lane & ~3;
    const float r0 = __shfl_sync(0xffffffffu, run, row_lane), r1 = __shfl_sync(0xffffffffu, run, row_lane + 1), r2 = __shfl_sync(0xffffffffu, run, row_lane + 2);
    const float b2 = (starts & 0xff00u) ? r1 : r0 + r1, b3 = (starts & 0xff0000u) ? r2 : b2 + r2;
    const float before = k == 0 ? 0.f : k == 1 ? r0 : k == 2 ? b2 : b3;
    if (spans && k == 3) sts<0>(s.row + tile * 32 + (lane >> 2) * 4, begin ? run : before + run);
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (!(begin & ((2u << j) - 1u))) e[j] += before;
    sts128(mine, make_float4(e[0], e[1], e[2], e[3]));
    sts128(mine + 16, make_float4(e[4], e[5], e[6], e[7]));
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kFlatRows; ++i) carry[i] = lds<0>(half[i >> 2] + (i & 3) * kPitch + lane * 4);
    if (T > 1) __syncwarp();      // with two tiles a warp flat_publish() stores over these words
}
// Second part: the parts of the row in other tiles, and the strip's last row as what it adds to those below.  Followed by a barrier.
__device__ __forceinline__ void flat_publish(FlatBlock &v, float (&carry)[kFlatRows], const FlatSmem &s, int first, int tile, uint32_t starts, int lane)
{
    if (!(starts & 1u)) {      // (`first`: the tile in which this tile's first row begins)
        const bool head = !(starts & ((2u << lane) - 1u));
        for (int t = first; t < tile; ++t) {
            const float4 a = lds128(s.row + t * 32), b = lds128(s.row + t * 32 + 16);
            if (head) {
                carry[0] += a.x; carry[1] += a.y; carry[2] += a.z; carry[3] += a.w;
                carry[4] += b.x; carry[5] += b.y; carry[6] += b.z; carry[7] += b.w;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kFlatRows; ++i) {
        const f2_t c = pack2(carry[i], carry[i]);
        v.a[i] = add2(v.a[i], c);
        v.b[i] = add2(v.b[i], c);
    }
    float4 e;
    unpack2(v.a[kFlatRows - 1], e.x, e.y);
    unpack2(v.b[kFlatRows - 1], e.z, e.w);
    sts128(s.col + (tile * 32 + lane) * 16, e);
}
// Many row groups: the sums of what is above, a column a thread, instead of every strip adding up what is above it.  Barriers on either side.
constexpr int kFlatTall = 8;
__device__ __forceinline__ void flat_sum_above(const FlatSmem &s, const FlatShape &sh)
{
    const int columns = sh.strips * 4, step = sh.strips * 16;
    for (int i = threadIdx.x; i < sh.planes * columns; i += blockDim.x) {
        const int g = i / columns;
        uint32_t at = s.col + g * sh.cells * 16 + (i - g * columns) * 4;
        float run = 0.f;
#pragma unroll 4
        for (int r = 0; r < sh.groups; ++r, at += step) {
            const float own = lds<0>(at);
            sts<0>(at, run);
            run += own;
        }
    }
}
// Store at off + at, the sum left to the store (see lds_row()).
__device__ __forceinline__ void sts_row(uint32_t off, uint32_t at, float v)
{
    asm volatile("{\n .reg .u32 a;\n add.u32 a, %0, %1;\n st.shared.f32 [a], %2;\n}" ::"r"(off), "r"(at), "f"(v));
}
// Third part: what is above, and the stores.  Followed by a barrier.
__device__ __forceinline__ void flat_put(FlatBlock &v, const FlatCell &cell, const FlatSmem &s, const FlatShape &sh, int tile, int lane)
{
    f2_t up_a = pack2(0.f, 0.f), up_b = up_a;
    const uint32_t own = s.col + (tile * 32 + lane) * 16;
    if (sh.groups > kFlatTall) {
        const float4 u = lds128(own);
        up_a = pack2(u.x, u.y);
        up_b = pack2(u.z, u.w);
    } else {
        uint32_t above = own - cell.group * sh.strips * 16;
        for (int r = 0; r < cell.group; ++r, above += sh.strips * 16) {
            const float4 u = lds128(above);
            up_a = add2(up_a, pack2(u.x, u.y));
            up_b = add2(up_b, pack2(u.z, u.w));
        }
    }
    __syncwarp();
    // column c+1 of integral row p0+1: sub-row 1, cell strip + 2
    const uint32_t at = s.image + cell.plane * sh.plane + flat_row_at(cell.group * kFlatRows + 1, sh.row, sh.skew) + (cell.strip + 2) * 4;
#pragma unroll
    for (int i = 0; i < kFlatRows; ++i) {
        float x, y, z, u;
        unpack2(add2(v.a[i], up_a), x, y);
        unpack2(add2(v.b[i], up_b), z, u);
        const uint32_t to = i * sh.row + (i == kFlatRows - 1 ? sh.skew : 0);
        if (i < cell.rows) {
            sts_row(to + sh.sub, at, x);
            sts_row(to + 2 * sh.sub, at, y);
            sts_row(to + 3 * sh.sub, at, z);
            sts_row(to + 4, at, u);
        }
    }
    // What is past the plane repeats the value at w, seven words a row: four lanes a row for the last strip of a row group.
    const int k = lane & 3, i = lane >> 2;
    const int row = i * sh.row + (i == kFlatRows - 1 ? sh.skew : 0);
    const int one = row + (k ? 4 + k * sh.sub : 8), two = row + 8 + k * sh.sub;      // words 1 .. 3 of the cell behind, word 0 of the next; its words 1 .. 3
    __syncwarp();
    for (uint32_t ends = __ballot_sync(0xffffffffu, cell.rows > 0 && cell.strip == sh.strips - 1); ends; ends &= ends - 1u) {
        const int from = __ffs(ends) - 1;
        const uint32_t base = __shfl_sync(0xffffffffu, at, from);
        if (i < __shfl_sync(0xffffffffu, cell.rows, from)) {
            const float u = lds_row(base + 4, row);
            sts<0>(base + one, u);
            if (k) sts<0>(base + two, u);
        }
    }
}

// ---- gathering ----------------------------------------------------------------------------------------
// Shared addresses of a tap row's ten words: a lane's cell on either side, and sub-rows, which are the same for the whole warp.
struct FlatCols {
    uint32_t lo, hi, lo_sub[kStrip + 1], hi_sub[kStrip + 1];
};
// STEPS: tap after tap, as quad_window() has it (forward 0.985 of the time over 130 drawn planes; backward 1.012, whose registers are short).
template <bool STEPS>
__device__ __forceinline__ uint32_t flat_window(uint32_t (&sub)[kStrip + 1], int strip, int shift, const FlatShape &sh)
{
    const int r = shift & 3;
    uint32_t at = (uint32_t)(r * sh.sub);
    if (STEPS) sub[0] = at;
#pragma unroll
    for (int m = STEPS ? 1 : 0; m <= kStrip; ++m) {
        at = r + m == 4 ? 4u : at + (uint32_t)sh.sub;
        sub[m] = STEPS ? at : (uint32_t)(((r + m) & 3) * sh.sub + (r + m < 4 ? 0 : 4));
    }
    return (uint32_t)(min(max(strip + (shift >> 2), -2), sh.strips) + 2) * 4u;
}
template <bool STEPS>
__device__ __forceinline__ FlatCols flat_cols(const BoxTaps &t, const FlatCell &cell, uint32_t image, const FlatShape &sh)
{
    FlatCols c;
    image += cell.plane * sh.plane;
    c.lo = image + flat_window<STEPS>(c.lo_sub, cell.strip, t.lo_c - 1, sh);
    c.hi = image + flat_window<STEPS>(c.hi_sub, cell.strip, t.hi_c, sh);
    return c;
}
__device__ __forceinline__ void quad_taps(const FlatCols &c, uint32_t row0, uint32_t row1, f2_t (&l)[kStrip + 1], f2_t (&h)[kStrip + 1])
{
    const uint32_t l0 = c.lo + row0, l1 = c.lo + row1, h0 = c.hi + row0, h1 = c.hi + row1;
#pragma unroll
    for (int m = 0; m <= kStrip; ++m) {
        l[m] = pack2(lds_row(c.lo_sub[m], l0), lds_row(c.lo_sub[m], l1));
        h[m] = pack2(lds_row(c.hi_sub[m], h0), lds_row(c.hi_sub[m], h1));
    }
}

// Offsets of the tap rows p0+j+lo_r and p0+j+hi_r+1, j = -1 .. 7, clamped to the plane.  Rows of the lanes of a warp are a multiple of 8 apart, so all
// pass from one row group to the next at the same j, and offsets grow with the row: clamping the offset clamps the row.
// A strip that does not exist has only row 0, which is zero; LANES: so do strips of fewer than eight rows past their last tap row.
template <bool LANES>
struct FlatRows {
    const FlatShape &sh;
    int lo0, hi0, lo_at, hi_at, last, rows;
    __device__ __forceinline__ uint32_t row(int first, int at, int j) const
    {
        return (uint32_t)__viaddmin_s32_relu(first, sh.offset[at + j], LANES && j > rows ? 0 : last);
    }
    __device__ __forceinline__ uint32_t lo(int j) const { return row(lo0, lo_at, j); }
    __device__ __forceinline__ uint32_t hi(int j) const { return row(hi0, hi_at, j); }
};
template <bool LANES>
__device__ __forceinline__ FlatRows<LANES> flat_rows(const BoxTaps &t, const FlatCell &cell, int h, const FlatShape &sh)
{
    const int far = h + 2 * kFlatRows;      // a border that far outside reaches the same rows, and products stay small
    const int lo = min(max(t.lo_r, -far), far) - 1, hi = min(max(t.hi_r, -far), far);
    auto at = [&](int a) { return flat_row_at(cell.group * kFlatRows + (a & ~7), sh.row, sh.skew); };
    return FlatRows<LANES>{sh, at(lo), at(hi), lo & 7, hi & 7, cell.rows ? sh.last : 0, cell.rows};
}

// ---- how a backward pass is dealt out ------------------------------------------------------------------
constexpr int kFlatMaxTiles = 32;              // tensor memory: 64 columns a tile, four tiles side by side
constexpr size_t kFlatMaxSmem = 227 * 1024 - 64;      // (and a few words that the compiler places)

// Columns of tensor memory in which the warps of a CTA keep one set of their tiles' rows; an allocation is a power of two.
__host__ __device__ constexpr int flat_slot_columns(int tiles_a_warp, int warps) { return kTmemColumns * tiles_a_warp * ((warps + 3) / 4); }
inline int pow2_columns(int n)
{
    int columns = kTmemColumns;
    while (columns < n) columns *= 2;
    return columns;
}
// Samples that share a CTA, where a plane alone would not fill eight warps: no fewer CTAs than two an SM, and room for three on one (narrow
// planes are half padding).
inline int flat_samples(int N, int C, int h, int w)
{
    const int cells = flat_strips(w) * flat_groups(h), bytes = flat_shape(h, w, 1).plane;
    int64_t planes = cells >= 256 ? 1 : 256 / cells;
    const int64_t most[] = {(int64_t)N * C / 296, N, 255, 56 * 1024 / bytes};
    for (int64_t m : most) planes = planes > m ? m : planes;
    return planes > 1 ? (int)planes : 1;
}

// CTAs of a backward that an SM holds (80 registers a thread, with two tiles a warp 128), and clusters of them that a GPU runs at once: as many as the
// occupancy calculator has where each CTA needs an SM, because the GPU's parts have 14 to 20 SMs each and a cluster lies in one part.
constexpr int kFlatMaxCluster = 8, kFlatClusters[kFlatMaxCluster + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
inline int flat_ctas_an_sm(int tiles_a_warp, int warps, int columns, size_t smem)
{
    const int most[] = {512 / columns, (tiles_a_warp == 1 ? 25 : 16) / warps, (int)(228 * 1024 / (smem + 1024))};
    int n = 32;
    for (int m : most) n = n > m ? m : n;
    return n > 1 ? n : 1;
}
inline int64_t flat_clusters_at_once(int ctas, int an_sm) { return (int64_t)kFlatClusters[ctas] * an_sm; }

struct FlatPlan {
    FlatShape sh;
    int tiles_a_warp, warps;
    size_t smem;
    int each, rounds;      // filters of a CTA; how often the GPU fills with CTAs
    int full;              // percent of the room for CTAs that has filters to work on meanwhile
};
// How many samples share a CTA, tiles a warp, and how many CTAs share a plane's filters.
// One tile a warp where the CTA's registers allow it (80 a thread, 24 warps): with two, half as many warps cover latencies ((134,3,8,128,147),
// 19 tiles: 313 us against 226; (1335,1,3,232,104), 24 tiles: 429 against 351).  13 to 16 tiles: two, if there are planes for the second
// CTA that then fits an SM ((217,1,1,192,80): 24.0 us, 24.6; (103,1,4,168,88), fewer planes than SMs: 45 with two, 33 with one).
// Filters over several CTAs: 12 planes of 120 x 133, F = 8, 119 us -> 25; (5,1,8,280,34) 96 -> 18.  Over as many as make rounds of clusters
// times filters each (and one, for what a CTA does besides) least: 34 clusters of four, of which 33 run at once, took as long as 66 ((36,1,4,96,144) 32.0 us with
// four CTAs, 24.8 with two; (18,1,8,136,112) 35.8 with eight, 27.6 with four; (48,1,3,48,320) 31.9 with three, 24.3 with two; 24 such launches 0.79 of the time).
inline FlatPlan flat_backward_plan(int N, int C, int F, int h, int w, bool write_gin)
{
    const int planes = flat_samples(N, C, h, w);
    FlatPlan p;
    p.sh = flat_shape(h, w, planes);
    const int64_t ctas = (int64_t)((N + planes - 1) / planes) * C;
    p.tiles_a_warp = p.sh.tiles > 24 || (p.sh.tiles > 12 && p.sh.tiles <= 16 && ctas > 148) ? 2 : 1;
    p.warps = (p.sh.tiles + p.tiles_a_warp - 1) / p.tiles_a_warp;
    p.sh.tiles = p.warps * p.tiles_a_warp;      // (the last one may be empty)
    p.smem = flat_smem(p.sh, p.tiles_a_warp, F) + (size_t)F * p.warps * kNumSums * sizeof(float);
    const int slot = flat_slot_columns(p.tiles_a_warp, p.warps);
    const size_t rows = (size_t)p.sh.tiles * 32 * kFlatRows * 16;
    // A cluster's CTAs have to find room at once, with no more than eight warps and four CTAs on an SM (eight of one warp: (510,1,2,22,20) 27.2 us, 19.7 without
    // clusters; (141,1,8,39,19) 35.8, 29.7 in clusters of four) and the tensor memory that their filters take.
    const int64_t room = 148 * (p.warps >= 8 ? 1 : p.warps <= 2 ? 4 : 8 / p.warps);
    const size_t own = p.smem;
    int64_t least = 0;
    for (int k = 1; k <= F && k <= kFlatMaxCluster; ++k) {
        const int each = (F + k - 1) / k, columns = pow2_columns(k > 1 ? slot * each : slot);
        const size_t smem = k > 1 && write_gin && own < rows * each ? rows * each : own;
        if (k > 1 && (ctas * k > room || ctas * k > 148 * (512 / columns) || rows * each > kFlatMaxSmem)) continue;
        const int an_sm = flat_ctas_an_sm(p.tiles_a_warp, p.warps, columns, smem);
        const int64_t rounds = (ctas - 1) / flat_clusters_at_once(k, an_sm) + 1;
        if (k > 1 && rounds * (each + 1) >= least) continue;
        least = rounds * (each + 1);
        p.sh.split = k;
        p.sh.columns = columns;
        p.smem = smem;
        p.each = each;
        p.rounds = (int)rounds;
        p.full = (int)(ctas * F * 100 / (rounds * each * 148 * an_sm));
    }
    return p;
}

// ---- and a forward pass ------------------------------------------------------------------------------------
struct FlatForwardPlan {
    FlatShape sh;
    int warps, fsplit, tsplit;
    bool tight;      // no room for scan corners of their own (tall planes of up to 32 columns)
    size_t smem;
};
inline FlatForwardPlan flat_forward_plan(int N, int C, int F, int h, int w)
{
    FlatForwardPlan p;
    p.sh = flat_shape(h, w, flat_samples(N, C, h, w));
    const int64_t ctas = (int64_t)((N + p.sh.planes - 1) / p.sh.planes) * C;
    p.fsplit = F % 2 == 0 && ctas < 148 * 6 ? 2 : 1;
    const int64_t room = p.sh.tiles <= 16 ? 148 * 2 : 148;      // (of more than 16 warps an SM takes one CTA)
    for (int k = p.fsplit + 1; k <= F; ++k)
        if (F % k == 0 && ctas * k <= room) p.fsplit = k;
    p.tsplit = 1;
    while (p.sh.tiles > 8 && ctas * p.fsplit * p.tsplit * 2 <= 148 && p.tsplit < 4) p.tsplit *= 2;
    p.warps = p.sh.tiles;
    p.smem = flat_smem(p.sh, 1, F);
    p.tight = p.smem > kFlatMaxSmem && flat_image_bytes(p.sh) >= p.warps * kFlatScanBytes;
    if (p.tight) p.smem -= p.warps * kFlatScanBytes;
    return p;
}

}  // namespace

}  // namespace bc
