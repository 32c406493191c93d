// Quad layout of an integral image, and the gathers that read it.
//
// A row holds the integral columns -4 .. w+7 in P = w/4 + 3 cells of four columns, stored as four sub-rows:
// column c is word (c & 3) * P + (c >> 2) + 1 of the row.  The first cell (columns -4 .. -1) and column 0 are
// zero, columns past w repeat the value at w, so a tap's column is clamped to the plane by clamping its cell.
//
// Why: a lane gathers for four adjacent output columns and so reads five adjacent integral columns on
// either side of its box.  Lanes are four columns apart, which in a plain row is a 4-way bank conflict; here
// the same tap of the 32 lanes of a warp is 32 consecutive words of one sub-row, whatever the box's offset
// (its remainder modulo 4 selects the sub-row, the same for all lanes).  All lanes of a warp work on the same
// plane row, so the clamping of tap rows at the plane's border cannot make conflicts either.
#pragma once
#include "bc_smem_walk.cuh"

namespace bc {

__host__ __device__ inline int quad_cells(int w) { return (w >> 2) + 3; }
__host__ __device__ inline int quad_pitch(int w) { return 4 * quad_cells(w); }      // floats per row, multiple of 4

// Value of lane 0 in a form the compiler can keep in a uniform register.
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

// BoxTaps of the table with its integers in uniform registers.
__device__ __forceinline__ BoxTaps load_taps_uniform(const float *tab)
{
    BoxTaps t = load_taps(tab);
    t.lo_r = uniform(t.lo_r); t.hi_r = uniform(t.hi_r);
    t.lo_c = uniform(t.lo_c); t.hi_c = uniform(t.hi_c);
    return t;
}

// Inclusive sum over the warp, or over each group of LN lanes; the shuffle's own predicate tells which lanes have
// somebody to add.
template <int LN = 32>
__device__ __forceinline__ float warp_scan(float v)
{
#pragma unroll
    for (int d = 1; d < LN; d <<= 1)
        asm volatile("{\n .reg .f32 u;\n .reg .pred p;\n shfl.sync.up.b32 u|p, %0, %1, %2, 0xffffffff;\n @p add.f32 %0, %0, u;\n}"
                     : "+f"(v) : "r"(d), "n"((32 - LN) << 8));
    return v;
}

// The same, and in `before` the inclusive sum of the lane in front (zero for the first): taking a lane's own value off
// its inclusive sum again would leave its infinity or its rounding in the columns to its left.
template <int LN = 32>
__device__ __forceinline__ float warp_prefix(float v, float &before)
{
    const float incl = warp_scan<LN>(v);
    asm volatile("{\n .reg .f32 u;\n .reg .pred p;\n shfl.sync.up.b32 u|p, %1, 1, %2, 0xffffffff;\n selp.f32 %0, u, 0f00000000, p;\n}"
                 : "=f"(before) : "f"(incl), "n"((32 - LN) << 8));
    return incl;
}

// Byte offsets within a row of the five taps on either side of the box, for the strip of columns 4*j .. 4*j+3.
// `shift` (the tap's column less the strip's) is the same for the whole warp.
struct QuadCols {
    uint32_t lo[kStrip + 1], hi[kStrip + 1];
};
// `cells`: of the plane's own columns (quad_cells(w)); `stride`: of a sub-row, which may be longer.
__device__ __forceinline__ void quad_window(uint32_t (&off)[kStrip + 1], int j, int shift, int cells, int stride)
{
    const int r = shift & 3, j0 = j + (shift >> 2);
    const uint32_t a = (uint32_t)(min(max(j0, -1), cells - 2) + 1) * 4u, b = (uint32_t)(min(max(j0 + 1, -1), cells - 2) + 1) * 4u;
    // tap after tap one sub-row on, from the fourth to the first of the next cell: an addition and a selection each
    uint32_t at = (uint32_t)(r * stride * 4) + a;
    off[0] = at;
#pragma unroll
    for (int m = 1; m <= kStrip; ++m) off[m] = at = r + m == 4 ? b : at + (uint32_t)(stride * 4);
}
__device__ __forceinline__ QuadCols quad_cols(const BoxTaps &t, int j, int cells, int stride)
{
    QuadCols c;
    quad_window(c.lo, j, t.lo_c - 1, cells, stride);
    quad_window(c.hi, j, t.hi_c, cells, stride);
    return c;
}

// Load at row + off.  The addition is inside the statement so that it stays an addition of a warp-uniform row
// to a lane's offset, which the load instruction does by itself; spelled in C++ the compiler distributes it
// over the row's multiplication, one multiply-add per load.
__device__ __forceinline__ float lds_row(uint32_t row, uint32_t off)
{
    float v;
    asm volatile("{\n .reg .u32 a;\n add.u32 a, %1, %2;\n ld.shared.f32 %0, [a];\n}" : "=f"(v) : "r"(row), "r"(off));
    return v;
}

// Shared addresses of the tap rows of a strip of R rows: lo(j+1), hi(j+1) for the rows p0+j+lo_r and p0+j+hi_r+1,
// j = -1 .. R-1, clamped to the plane.  Lane k works out the k-th address and hands it to the warp, which
// costs one shuffle an address instead of the same clamps and multiplications in every lane.
template <int R>
struct QuadRows {
    uint32_t lo_at[R + 1], hi_at[R + 1];
    __device__ __forceinline__ uint32_t lo(int j) const { return lo_at[j]; }
    __device__ __forceinline__ uint32_t hi(int j) const { return hi_at[j]; }
};
// The same, handed out where they are used: 2 R + 1 registers fewer.
template <int R>
struct QuadRowsLater {
    uint32_t mine;
    __device__ __forceinline__ uint32_t lo(int j) const { return __shfl_sync(0xffffffffu, mine, j); }
    __device__ __forceinline__ uint32_t hi(int j) const { return __shfl_sync(0xffffffffu, mine, R + 1 + j); }
};
template <int R>
__device__ __forceinline__ QuadRowsLater<R> quad_rows_later(const BoxTaps &t, int p0, int h, uint32_t lo32, uint32_t hi32, int row_bytes, int lane)
{
    static_assert(2 * (R + 1) <= 32, "one lane per address");
    const bool hi = lane > R;
    const int a = p0 - 1 + (hi ? lane - R - 1 + t.hi_r + 1 : lane + t.lo_r);
    const uint32_t mine = (hi ? hi32 : lo32) + (uint32_t)(min(max(a, 0), h) * row_bytes);
    return QuadRowsLater<R>{mine};
}
template <int R>
__device__ __forceinline__ QuadRows<R> quad_rows(const BoxTaps &t, int p0, int h, uint32_t lo32, uint32_t hi32, int row_bytes, int lane)
{
    const QuadRowsLater<R> later = quad_rows_later<R>(t, p0, h, lo32, hi32, row_bytes, lane);
    QuadRows<R> q;
#pragma unroll
    for (int j = 0; j <= R; ++j) {
        q.lo_at[j] = later.lo(j);
        q.hi_at[j] = later.hi(j);
    }
    return q;
}

// The ten taps of the tap rows at shared addresses `row0` (low halves) and `row1` (high halves).
__device__ __forceinline__ void quad_taps(const QuadCols &c, uint32_t row0, uint32_t row1, f2_t (&l)[kStrip + 1], f2_t (&h)[kStrip + 1])
{
#pragma unroll
    for (int m = 0; m <= kStrip; ++m) {
        l[m] = pack2(lds_row(row0, c.lo[m]), lds_row(row1, c.lo[m]));
        h[m] = pack2(lds_row(row0, c.hi[m]), lds_row(row1, c.hi[m]));
    }
}

// Column-combined values of a tap-row pair: d = (1-f_hi) h[m] + f_hi h[m+1] - (1-f_lo) l[m+1] - f_lo l[m].
template <class Cols>
__device__ __forceinline__ void quad_pair(const Cols &c, uint32_t row0, uint32_t row1, const ColW2 &cw, f2_t (&d)[kStrip])
{
    f2_t l[kStrip + 1], h[kStrip + 1];
    quad_taps(c, row0, row1, l, h);
#pragma unroll
    for (int m = 0; m < kStrip; ++m)
        d[m] = fma2(cw.nfl, l[m], fma2(cw.nwl, l[m + 1], fma2(cw.fh, h[m + 1], mul2(cw.wh, h[m]))));
}
// The same plus the one-column strips outside the box: el = l[m+1] - l[m], eh = h[m+1] - h[m].
template <class Cols>
__device__ __forceinline__ void quad_pair_e(const Cols &c, uint32_t row0, uint32_t row1, const ColW2 &cw, f2_t (&d)[kStrip],
                                            f2_t (&el)[kStrip], f2_t (&eh)[kStrip])
{
    f2_t l[kStrip + 1], h[kStrip + 1];
    quad_taps(c, row0, row1, l, h);
#pragma unroll
    for (int m = 0; m < kStrip; ++m) {
        el[m] = sub2(l[m + 1], l[m]);
        eh[m] = sub2(h[m + 1], h[m]);
        d[m] = fma2(cw.fl, el[m], fma2(cw.fh, eh[m], sub2(h[m], l[m + 1])));
    }
}

// Sums the five values over the warp with 8 shuffles (each exchange halves what a lane still holds).  The
// lanes for which sum5_slot() is >= 0 return the sum of that value.
__device__ __forceinline__ int sum5_slot(int lane)
{
    const int k = lane >> 2;       // (bit 4, bit 3, bit 2)
    return (lane & 3) ? -1 : (k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 2 : k == 4 ? 3 : k == 5 ? 4 : -1);
}
__device__ __forceinline__ float warp_sum5(const float (&v)[kNumSums], int lane)
{
    const unsigned full = 0xffffffffu;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    const float k0 = (b4 ? v[3] : v[0]) + __shfl_xor_sync(full, b4 ? v[0] : v[3], 16);
    const float k1 = (b4 ? v[4] : v[1]) + __shfl_xor_sync(full, b4 ? v[1] : v[4], 16);
    const float k2 = (b4 ? 0.f : v[2]) + __shfl_xor_sync(full, b4 ? v[2] : 0.f, 16);
    const float m0 = (b3 ? k2 : k0) + __shfl_xor_sync(full, b3 ? k0 : k2, 8);
    const float m1 = (b3 ? 0.f : k1) + __shfl_xor_sync(full, b3 ? k1 : 0.f, 8);
    float s = (b2 ? m1 : m0) + __shfl_xor_sync(full, b2 ? m0 : m1, 4);
    s += __shfl_xor_sync(full, s, 2);
    s += __shfl_xor_sync(full, s, 1);
    return s;
}

// One filter's contribution of a strip of R rows to grad-input and to the five sums.  FULL: the strip has all its rows,
// else those at or past `rows` do not exist (their input values are zero there).
// at: the strip's input values and grad-input accumulators.  `first()` returns the input values of row 0, `fetch(i)`
// starts fetching row i's accumulators and the input values of row i + 1, which `next()` returns, `add(i, ...)` adds
// to the accumulators.
// The column strips enter the sums weighted by u(j), what the rows of the box make of the input values next to
// tap row j: sum_i x_i (row combination of e) = sum_j e(j) (w_a x_(j+1) + w_b x_j).
// PACKED: an input value is held twice, as the factor of a pair of tap rows.  That saves operations, which pays where registers
// leave three or two CTAs an SM and the tiles are full, of one column ((256,32,4,64,128): 504 us, scalar 522; (32,32,4,64,128) in
// bfloat16 71 and 74; with two columns it costs 0.5 to 1 %).  Where rows are cut or unaligned, scalars ((60,16,4,40,250): 140 us in pairs, 131).
// The same values either way.
template <int R, bool NEED_PARAMS, bool FULL, bool PACKED = false, bool LANES = false, class Cols, class Rows, class Cells>
__device__ __forceinline__ void quad_backward_strip(const BoxTaps &t, const Cols &cols, const Rows &q, const ColW2 &cw,
                                                    Cells &&at, float (&sums)[kNumSums], int rows)
{
    f2_t pd[kStrip];
    const f2_t scale = pack2(t.scale, t.scale);
    // gather value of one column from its two tap-row pairs and their difference
    auto gather = [&](f2_t cur, f2_t prev, f2_t diff) {
        float lo_new, hi_new, lo_old, hi_old, top, bot;
        unpack2(cur, lo_new, hi_new);
        unpack2(prev, lo_old, hi_old);
        unpack2(diff, top, bot);
        (void)hi_new; (void)lo_old;
        return (hi_old - lo_new) + t.f_hi_r * bot + t.f_lo_r * top;
    };
    if (NEED_PARAMS) {
        f2_t left = pack2(0.f, 0.f), right = left, out2 = left, topbot = left;
        float s_top = 0.f, s_bot = 0.f;
        f2_t el[kStrip], eh[kStrip], xx[kStrip];      // (topbot, xx: PACKED)
        quad_pair_e(cols, q.lo(0), q.hi(0), cw, pd, el, eh);
        float4 e = at.first();
        // What the rows of the box make of the input values next to a pair of tap rows.  (Two products: the values' difference,
        // an operation less, is infinite for large ones of opposite sign.)
        const float wb_top = t.f_lo_r - 1.0f, wa_bot = 1.0f - t.f_hi_r;
        const f2_t wa = pack2(-t.f_lo_r, wa_bot), wb = pack2(wb_top, t.f_hi_r);
        auto weigh = [&](float x, float next) { return pack2(fmaf(-t.f_lo_r, next, wb_top * x), fmaf(wa_bot, next, t.f_hi_r * x)); };
        {
            const float x0[kStrip] = {e.x, e.y, e.z, e.w};
#pragma unroll
            for (int m = 0; m < kStrip; ++m) {
                f2_t u;
                if constexpr (PACKED) {
                    xx[m] = pack2(x0[m], x0[m]);
                    u = mul2(wa, xx[m]);
                } else {
                    u = weigh(0.f, x0[m]);
                }
                left = fma2(u, el[m], left);
                right = fma2(u, eh[m], right);
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (FULL || i < rows) {
                f2_t cd[kStrip], dd[kStrip];
                at.fetch(i);
                quad_pair_e(cols, q.lo(i + 1), q.hi(i + 1), cw, cd, el, eh);
                const float4 below = at.next();
                const float x0[kStrip] = {e.x, e.y, e.z, e.w};
                const float x1[kStrip] = {i + 1 < R ? below.x : 0.f, i + 1 < R ? below.y : 0.f, i + 1 < R ? below.z : 0.f, i + 1 < R ? below.w : 0.f};
#pragma unroll
                for (int m = 0; m < kStrip; ++m) {
                    f2_t u;
                    dd[m] = sub2(cd[m], pd[m]);
                    if constexpr (PACKED) {
                        u = mul2(wb, xx[m]);
                        topbot = fma2(xx[m], dd[m], topbot);
                        if (i + 1 < R) {
                            xx[m] = pack2(x1[m], x1[m]);
                            u = fma2(wa, xx[m], u);
                        }
                    } else {
                        u = weigh(x0[m], x1[m]);
                        float top, bot;
                        unpack2(dd[m], top, bot);
                        s_top = fmaf(x0[m], top, s_top);
                        s_bot = fmaf(x0[m], bot, s_bot);
                    }
                    left = fma2(u, el[m], left);
                    right = fma2(u, eh[m], right);
                }
                const f2_t g01 = pack2(gather(cd[0], pd[0], dd[0]), gather(cd[1], pd[1], dd[1]));
                const f2_t g23 = pack2(gather(cd[2], pd[2], dd[2]), gather(cd[3], pd[3], dd[3]));
                out2 = fma2(pack2(e.x, e.y), g01, fma2(pack2(e.z, e.w), g23, out2));
                at.add(i, g01, g23, scale);
#pragma unroll
                for (int m = 0; m < kStrip; ++m) pd[m] = !LANES || i + 1 < rows ? cd[m] : pack2(0.f, 0.f);
                if (i + 1 < R) e = below;
            }
        }
        if constexpr (PACKED) unpack2(topbot, s_top, s_bot);
        float a, b;
        unpack2(out2, a, b); sums[0] = a + b;
        sums[1] = s_top; sums[2] = s_bot;
        unpack2(left, a, b); sums[3] = a + b;
        unpack2(right, a, b); sums[4] = a + b;
    } else {
        quad_pair(cols, q.lo(0), q.hi(0), cw, pd);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (FULL || i < rows) {
                f2_t cd[kStrip];
                float g[kStrip];
                at.fetch(i);
                quad_pair(cols, q.lo(i + 1), q.hi(i + 1), cw, cd);
                at.next();
#pragma unroll
                for (int m = 0; m < kStrip; ++m) {
                    g[m] = gather(cd[m], pd[m], sub2(cd[m], pd[m]));
                    pd[m] = cd[m];
                }
                at.add(i, pack2(g[0], g[1]), pack2(g[2], g[3]), scale);
            }
        }
    }
}

// The four outputs of row p from the tap-row pairs of rows p-1 and p, times scale (sfl, sfh: scale times the
// fractions of the row borders).
__device__ __forceinline__ void quad_forward_row(const f2_t (&prev)[kStrip], const f2_t (&cur)[kStrip], float scale, float sfl,
                                                 float sfh, float (&v)[kStrip])
{
#pragma unroll
    for (int m = 0; m < kStrip; ++m) {
        float b, dd, a, cc, top, bot;
        unpack2(cur[m], b, dd);
        unpack2(prev[m], a, cc);
        unpack2(sub2(cur[m], prev[m]), top, bot);
        (void)a; (void)dd;
        v[m] = (cc - b) * scale + sfh * bot + sfl * top;
    }
}

}  // namespace bc
