// Shared-memory-resident kernels in tiles of 32 x 32, for planes small enough to keep on chip that waste less in these than in
// tiles of 8 x 128 (quad_prefers_forward() in box_quad_plane.cuh), or by strips dealt out to lanes (bc_flat.cuh).  HBM traffic is
// the compulsory minimum: the forward reads the input once and writes the output once; the backward reads the input and grad_output
// once and writes grad_input once.  No integral image ever goes to global memory.
//
// Forward : one CTA per (plane, group of filters).  The plane's integral image is built in shared
//           memory, then every thread walks its 4-column x 8-row strip (bc_walk.cuh scheme) for
//           each filter of the group and writes 128-bit rows of the output.
// Backward: one CTA per plane.  For each filter the grad_output plane is integrated in shared memory and
//           gathered with the mirrored box.  The input plane waits in shared memory, grad-input accumulates over the filters in
//           registers.  The five sums that finish the parameter gradients are reduced per CTA and left for
//           finish_param_grads_kernel or the channel's last CTA (bc_finish.cuh).
//
// Thread layout (same for building the integral image and for gathering): a warp owns a tile of
// 32 x 32 pixels; lane = 8 column groups (cg, 4 columns each) x 4 row groups (rg, 8 rows each).
//
// Shared-memory layout of the integral image: row a (0..h) starts at a*pitch + a/8 floats and
// holds [4 zeros | I[a][0..w] | 4 copies of I[a][w]].
//   * the padding turns the clamping of the five adjacent column taps of a strip into a clamp of
//     the window start, so a tap row is read with two base addresses and immediate offsets;
//   * the a/8 skew puts the four row groups of a warp (tap rows 8 apart) into the four bank
//     residues modulo 4 while the eight column groups are 4 floats apart: 32 lanes, 32 banks.
//
// Integral image construction: each thread loads its 8 x 4 block (128-bit loads), scans it in
// registers, the 8 column-group lanes scan row totals with shuffles, warps of the same tile row
// exchange row totals through shared memory; the same again down the columns.  The block is then
// stored with the layout above (conflict-free).
//
// The forward is instantiated twice: FAST for planes whose height is a multiple of 8 and width
// a multiple of 4 with aligned tensors (no per-row guards, one vector access per strip row), and
// a guarded version for everything else.  The backward serves the former only.
//
// This file holds the kernels and their launchers as templates over the storage type of the big
// tensors (Io<> below); box_plane_smem.cu instantiates them for float, box_plane_half.cu for
// __half and __nv_bfloat16.  What limits these kernels is the shared-memory data pipe: every
// output value takes about five 4-byte words from the integral image in shared memory, against
// four bytes of HBM traffic.
#pragma once
#include "bc_common.cuh"
#include "bc_finish.cuh"
#include "bc_flat.cuh"
#include "bc_smem_walk.cuh"
#include "bc_tile_io.cuh"
#include "bc_tmem.cuh"
#include "box_quad_plane.cuh"
#include "box_tmem_plane.cuh"

namespace bc {

namespace {

constexpr int kR = 8;            // rows per strip
constexpr int kTile = 32;        // a warp covers kTile x kTile pixels
constexpr int kPad = 4;          // padding columns on either side of an integral-image row
constexpr int kMaxTiles = 32;
constexpr int kMaxSmem = 200 * 1024;

__host__ __device__ inline int layout_pitch(int w) { return w + 1 + 2 * kPad; }
__host__ __device__ inline int layout_floats(int h, int w) { return (((h + 1) * layout_pitch(w) + (h >> 3) + 4) + 3) & ~3; }

inline int warp_tiles(int h, int w) { return ((w + kTile - 1) / kTile) * ((h + kTile - 1) / kTile); }

struct Geometry {
    int h, w, col_tiles, row_tiles, ntiles, pitch4;
};

__device__ __forceinline__ Geometry geometry(int h, int w)
{
    Geometry g;
    g.h = h; g.w = w;
    g.col_tiles = (w + kTile - 1) / kTile;
    g.row_tiles = (h + kTile - 1) / kTile;
    g.ntiles = g.col_tiles * g.row_tiles;
    g.pitch4 = layout_pitch(w) * 4;
    return g;
}

// Everything a thread needs to know about one of its strips; computed once per kernel.
struct Strip {
    int p0, q0, rt, ct;
    int pix;              // p0*w + q0: offset of the strip's first pixel in a plane
    uint32_t store;       // shared address of column q0 of integral row p0+1
    bool tile;            // the warp tile exists
    bool active;          // ... and this strip has pixels inside the plane
};

__device__ __forceinline__ Strip make_strip(const Geometry &g, uint32_t sI32, int wt, int cg, int rg)
{
    Strip t;
    t.rt = wt / g.col_tiles;
    t.ct = wt - t.rt * g.col_tiles;
    t.p0 = t.rt * kTile + rg * kR;
    t.q0 = t.ct * kTile + cg * kStrip;
    t.pix = t.p0 * g.w + t.q0;
    t.tile = wt < g.ntiles;
    t.active = t.tile && t.p0 < g.h && t.q0 < g.w;
    const int a = t.p0 + 1;
    t.store = sI32 + (kPad + t.q0) * 4 + a * g.pitch4 + ((a >> 3) << 2);
    return t;
}

// Zeroes what never changes in the integral image: row 0 and the left-hand padding (and column
// 0) of every row.  Followed by the barriers inside the build.
__device__ __forceinline__ void init_integral_padding(float *sI, const Geometry &g)
{
    const int pitch = g.pitch4 >> 2;
    for (int c = threadIdx.x; c < pitch; c += blockDim.x) sI[c] = 0.0f;
    for (int i = threadIdx.x; i < g.h * (kPad + 1); i += blockDim.x) {
        const int a = 1 + i / (kPad + 1), c = i - (a - 1) * (kPad + 1);
        sI[a * pitch + (a >> 3) + c] = 0.0f;
    }
}

// Register block of a strip while the integral image is being built.
template <int T>
struct Blocks {
    float v[T][kR][kStrip];
    float carry[T][kR];
};

// Build, part 1: fetch every strip's 8 x 4 block (from the staged copy of the plane in shared
// memory when STAGED, else from global memory), prefix it along rows inside the thread and across
// the 8 column-group lanes, publish the tile's row totals.  Ends with a barrier, after which the
// staged plane is no longer needed.
template <typename IO, int T, bool FAST, bool STAGED, bool MAYBE_RELU = false>
__device__ __forceinline__ void build_rows(Blocks<T> &b, const Strip (&st)[T], const IO *__restrict__ src,
                                           uint32_t sG32, float *sRow, const Geometry &g, int cg, int rg,
                                           bool relu = false)
{
#pragma unroll
    for (int k = 0; k < T; ++k) {
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            if (STAGED) {
                const float4 t = st[k].active ? Io<IO>::lds4(sG32 + (st[k].pix + i * g.w) * (uint32_t)sizeof(IO))
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
                b.v[k][i][0] = t.x; b.v[k][i][1] = t.y; b.v[k][i][2] = t.z; b.v[k][i][3] = t.w;
            } else if (FAST) {
                const float4 t = st[k].active ? Io<IO>::load4(src + st[k].pix + i * g.w) : make_float4(0.f, 0.f, 0.f, 0.f);
                b.v[k][i][0] = t.x; b.v[k][i][1] = t.y; b.v[k][i][2] = t.z; b.v[k][i][3] = t.w;
            } else {
                const bool in = st[k].active && st[k].p0 + i < g.h;
#pragma unroll
                for (int m = 0; m < kStrip; ++m)
                    b.v[k][i][m] = (in && st[k].q0 + m < g.w) ? Io<IO>::load1(src + st[k].pix + i * g.w + m) : 0.0f;
            }
        }
    }
    if (MAYBE_RELU && relu) {
#pragma unroll
        for (int k = 0; k < T; ++k)
#pragma unroll
            for (int i = 0; i < kR; ++i)
#pragma unroll
                for (int m = 0; m < kStrip; ++m) b.v[k][i][m] = fmaxf(b.v[k][i][m], 0.0f);
    }
#pragma unroll
    for (int k = 0; k < T; ++k) {
        float tot[kR];
#pragma unroll
        for (int i = 0; i < kR; ++i) {
            b.v[k][i][1] += b.v[k][i][0]; b.v[k][i][2] += b.v[k][i][1]; b.v[k][i][3] += b.v[k][i][2];
            const float own = b.v[k][i][3];
            float incl = own;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {
                const float u = __shfl_up_sync(0xffffffffu, incl, d, 8);
                incl += cg >= d ? u : 0.0f;
            }
            b.carry[k][i] = incl - own;
            tot[i] = incl;
        }
        if (cg == 7 && st[k].tile) {
            float4 *dst = reinterpret_cast<float4 *>(sRow + (st[k].ct * g.row_tiles + st[k].rt) * kTile + rg * kR);
            dst[0] = make_float4(tot[0], tot[1], tot[2], tot[3]);
            dst[1] = make_float4(tot[4], tot[5], tot[6], tot[7]);
        }
    }
    __syncthreads();
}

// Build, part 2: row totals of the tiles to the left, prefix down the columns (thread, the 4
// row-group lanes, tiles above), store rows p0+1 .. p0+8 with the right-hand padding.  Ends with
// a barrier: the integral image is complete.
template <int T, bool FAST>
__device__ __forceinline__ void build_columns(Blocks<T> &b, const Strip (&st)[T], float *sRow, float *sCol,
                                              const Geometry &g, int cg, int rg)
{
    float ccarry[T][kStrip];
#pragma unroll
    for (int k = 0; k < T; ++k) {
        if (st[k].tile) {
            for (int c2 = 0; c2 < st[k].ct; ++c2) {
                const float4 *s = reinterpret_cast<const float4 *>(sRow + (c2 * g.row_tiles + st[k].rt) * kTile + rg * kR);
                const float4 x = s[0], y = s[1];
                b.carry[k][0] += x.x; b.carry[k][1] += x.y; b.carry[k][2] += x.z; b.carry[k][3] += x.w;
                b.carry[k][4] += y.x; b.carry[k][5] += y.y; b.carry[k][6] += y.z; b.carry[k][7] += y.w;
            }
        }
        // apply the row carry and run the in-thread column prefix in the same sweep
#pragma unroll
        for (int m = 0; m < kStrip; ++m) b.v[k][0][m] += b.carry[k][0];
#pragma unroll
        for (int i = 1; i < kR; ++i)
#pragma unroll
            for (int m = 0; m < kStrip; ++m) b.v[k][i][m] += b.carry[k][i] + b.v[k][i - 1][m];

        float tot[kStrip];
#pragma unroll
        for (int m = 0; m < kStrip; ++m) {
            const float own = b.v[k][kR - 1][m];
            float incl = own;
            float u = __shfl_up_sync(0xffffffffu, incl, 8);
            incl += rg >= 1 ? u : 0.0f;
            u = __shfl_up_sync(0xffffffffu, incl, 16);
            incl += rg >= 2 ? u : 0.0f;
            ccarry[k][m] = incl - own;
            tot[m] = incl;
        }
        if (rg == 3 && st[k].tile)
            *reinterpret_cast<float4 *>(sCol + (st[k].rt * g.col_tiles + st[k].ct) * kTile + cg * kStrip) =
                make_float4(tot[0], tot[1], tot[2], tot[3]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < T; ++k) {
        if (st[k].tile) {
            for (int r2 = 0; r2 < st[k].rt; ++r2) {
                const float4 x = *reinterpret_cast<const float4 *>(sCol + (r2 * g.col_tiles + st[k].ct) * kTile + cg * kStrip);
                ccarry[k][0] += x.x; ccarry[k][1] += x.y; ccarry[k][2] += x.z; ccarry[k][3] += x.w;
            }
        }
        if (st[k].active) {
            const bool last = st[k].q0 + kStrip >= g.w;
            const int npad = g.w - st[k].q0;      // padding columns still to fill (1..4) when `last`
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                if (FAST || st[k].p0 + i < g.h) {
                    // p0 is a multiple of 8, so only the last of the 8 rows moves to the next skew
                    const uint32_t ra = st[k].store + i * g.pitch4 + (i == kR - 1 ? 4 : 0);
                    const float x0 = b.v[k][i][0] + ccarry[k][0], x1 = b.v[k][i][1] + ccarry[k][1];
                    const float x2 = b.v[k][i][2] + ccarry[k][2], x3 = b.v[k][i][3] + ccarry[k][3];
                    // past the plane's last column the running value is I[a][w], which is exactly
                    // what the right-hand padding has to hold
                    sts<4>(ra, x0); sts<8>(ra, x1); sts<12>(ra, x2); sts<16>(ra, x3);
                    if (last) {
                        sts<20>(ra, x3);
                        if (npad > 1) sts<24>(ra, x3);
                        if (npad > 2) sts<28>(ra, x3);
                        if (npad > 3) sts<32>(ra, x3);
                    }
                }
            }
        }
    }
    __syncthreads();
}

__device__ __forceinline__ Walk make_walk(uint32_t sI32, const BoxTaps &t, int q0, const Geometry &g)
{
    const int bl = min(max(q0 + t.lo_c - 1, -kPad), g.w);
    const int bh = min(max(q0 + t.hi_c, -kPad), g.w);
    Walk o;
    o.lo = sI32 + (kPad + bl) * 4;
    o.dhi = (uint32_t)((bh - bl) * 4);
    o.pitch4 = g.pitch4;
    o.h = g.h;
    return o;
}

// FUSED: the inference steps of `Fusion` around the gather (the output may then alias the residual,
// so it is not declared restrict).
// INTEG: `integ` holds the plane's integral image, plain rows of w + 1 floats, which is only copied (instantiations of
// their own: as a run-time branch it cost the others 3 to 5 %).
template <typename IO, int T, bool FAST, bool FUSED = false, bool INTEG = false>
__global__ void __launch_bounds__(T == 1 ? 256 : 512, T == 1 ? (FUSED ? 2 : 4) : 1)
forward_plane_kernel(const IO *__restrict__ x, const float *__restrict__ integ, BoxParams bp, IO *out, int C, int F,
                     int h, int w, int fsplit, bool normalize, bool exact, Fusion fu)
{
    extern __shared__ float4 smem4[];
    float *sI = reinterpret_cast<float *>(smem4);
    const Geometry g = geometry(h, w);
    float *sRow = sI + layout_floats(h, w);
    float *sCol = sRow + g.ntiles * kTile;
    __shared__ __align__(16) float sTaps[kMaxFilters * kTapWords];
    grid_dependency_release();

    const int64_t nc = blockIdx.x / fsplit;
    const int part = blockIdx.x % fsplit;
    const int c = (int)(nc % C);
    const int f_begin = (F * part) / fsplit, f_end = (F * (part + 1)) / fsplit;
    const uint32_t sI32 = smem_u32(sI);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int cg = lane & 7, rg = lane >> 3;

    // a hint only: the plane on its way to L2 while this CTA still waits for the kernel in front
    if (FUSED && fu.residual) prefetch_l2(fu.residual + (nc * F + f_begin) * (int64_t)h * w, (size_t)(f_end - f_begin) * h * w * sizeof(float));
    if (FAST && !INTEG && IsFloat<IO>::value && threadIdx.x == 0 && part == 0)
        bulk_prefetch_l2(x + nc * (int64_t)h * w, (uint32_t)(h * w) * 4u);
    Strip st[T];
#pragma unroll
    for (int k = 0; k < T; ++k) st[k] = make_strip(g, sI32, warp + k * nwarps, cg, rg);
    init_integral_padding(sI, g);

    // everything above touches registers and shared memory only (and hints); from here on the parameters and
    // the input are read, which the kernel in front of this one in the stream may have written
    grid_dependency_wait();
    if ((int)threadIdx.x < f_end - f_begin) {
        const Box box = load_box(bp, c * F + f_begin + threadIdx.x);
        store_taps(sTaps + threadIdx.x * kTapWords,
                   taps_forward(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    if (INTEG) {
        const float *I = integ + nc * (int64_t)(h + 1) * (w + 1);
        const int pitch = g.pitch4 >> 2;
        __syncthreads();      // (the zero padding has been written)
        copy_integral_rows(I, h, w, w + 1 + kPad, warp, nwarps, lane,
                           [&](int a, int col, float e) { sI[a * pitch + (a >> 3) + kPad + col] = e; });
        __syncthreads();
    } else {
        Blocks<T> blk;
        build_rows<IO, T, FAST, false, FUSED>(blk, st, x + nc * (int64_t)h * w, 0u, sRow, g, cg, rg, FUSED && fu.input_relu);
        build_columns<T, FAST>(blk, st, sRow, sCol, g, cg, rg);
    }

    for (int f = f_begin; f < f_end; ++f) {
        const BoxTaps t = load_taps(sTaps + (f - f_begin) * kTapWords);
        const ColW2 cw = col_weights(t);
        const float sfl = t.scale * t.f_lo_r, sfh = t.scale * t.f_hi_r;
        IO *o = out + (nc * F + f) * (int64_t)h * w;
        float mul = 1.0f, add = 0.0f;
        if (FUSED) {
            if (fu.scale) mul = __ldg(fu.scale + c * F + f);
            if (fu.shift) add = __ldg(fu.shift + c * F + f);
        }
#pragma unroll
        for (int k = 0; k < T; ++k) {
            if (!st[k].active) continue;
            const Walk wk = make_walk(sI32, t, st[k].q0, g);
            f2_t prev[kStrip];                 // (d of row lo-1, d of row hi) of the current pixel row
            load_pair(wk, st[k].p0 + t.lo_r - 1, st[k].p0 + t.hi_r, cw, prev);
            IO *dst = o + st[k].pix;
            const float *res = (FUSED && fu.residual) ? fu.residual + (nc * F + f) * (int64_t)h * w + st[k].pix : nullptr;
            float4 skip[FUSED ? kR : 1];       // all residual rows in flight before the gather
            if (FUSED && res) {
#pragma unroll
                for (int i = 0; i < kR; ++i, res += w) {
                    if (FAST) {
                        skip[FUSED ? i : 0] = *reinterpret_cast<const float4 *>(res);
                    } else {
                        const bool in = st[k].p0 + i < h;
                        const int q = st[k].q0;
                        skip[FUSED ? i : 0] = make_float4(in ? res[0] : 0.f, in && q + 1 < w ? res[1] : 0.f, in && q + 2 < w ? res[2] : 0.f,
                                                          in && q + 3 < w ? res[3] : 0.f);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kR; ++i) {
                const int p = st[k].p0 + i;
                if (FAST || p < h) {
                    f2_t cur[kStrip];          // (d of row lo, d of row hi+1)
                    load_pair(wk, p + t.lo_r, p + t.hi_r + 1, cw, cur);
                    float v[kStrip];
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) {
                        // (C - B) + f_hi (D - C) + f_lo (B - A), times scale
                        float b, dd, a, cc, top, bot;
                        unpack2(cur[m], b, dd);
                        unpack2(prev[m], a, cc);
                        unpack2(sub2(cur[m], prev[m]), top, bot);
                        v[m] = (cc - b) * t.scale + sfh * bot + sfl * top;
                        (void)a; (void)dd;
                        prev[m] = cur[m];
                    }
                    if (FUSED) {
#pragma unroll
                        for (int m = 0; m < kStrip; ++m) v[m] = v[m] * mul + add;
                        if (res) {
                            const float4 r = skip[FUSED ? i : 0];
                            v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
                        }
                        if (fu.output_relu) {
#pragma unroll
                            for (int m = 0; m < kStrip; ++m) v[m] = fmaxf(v[m], 0.0f);
                        }
                    }
                    if (FAST) {
                        Io<IO>::store4(dst, v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int m = 0; m < kStrip; ++m)
                            if (st[k].q0 + m < w) Io<IO>::store1(dst + m, v[m]);
                    }
                    dst += w;
                }
            }
        }
    }
}

// Backward of aligned planes of up to eight tiles, one a warp (flat_beats_square() says which).
// The input plane waits in shared memory, float whatever IO is: float planes arrive by a bulk copy when STAGED, narrow ones are
// converted by the threads as they are copied in.
// STAGED: the input plane and each grad_output plane arrive in shared memory by asynchronous bulk
// copies (one instruction per plane, issued by one thread); the copy of the next grad_output
// plane runs while the current one is gathered.
// INTEG: the input is given as its integral image (instantiations of their own: as a run-time branch it cost the others 5 %).
template <typename IO, bool STAGED, bool NEED_PARAMS, bool COUNTED = false, bool INTEG = false>
__global__ void __launch_bounds__(512)
backward_square_kernel(const IO *__restrict__ x, const float *__restrict__ x_integ, const IO *__restrict__ grad_output, BoxParams bp,
                      IO *__restrict__ grad_input, float *__restrict__ partials, int N, int C, int F,
                      int h, int w, bool normalize, bool exact, bool write_gin, Finish fin)
{
    extern __shared__ float4 smem4[];
    const Geometry g = geometry(h, w);
    const int npix = h * w;
    float *sI = reinterpret_cast<float *>(smem4);          // integral(grad_output plane)
    float *sRow = sI + layout_floats(h, w);
    float *sCol = sRow + g.ntiles * kTile;
    float *sX = sCol + g.ntiles * kTile;                   // the input plane, pitch w (NEED_PARAMS)
    constexpr bool X_BY_COPY = STAGED && IsFloat<IO>::value;
    float *sG = sX + (NEED_PARAMS ? npix : 0);             // staged grad_output plane, as stored (STAGED)
    __shared__ __align__(16) float sTaps[kMaxFilters * kTapWords];
    __shared__ float red[16][kNumSums];
    __shared__ __align__(8) unsigned long long mbar[2];
    grid_dependency_release();

    const int64_t nc = blockIdx.x;
    const int c = (int)(nc % C), n = (int)(nc / C);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int cg = lane & 7, rg = lane >> 3;
    const uint32_t sI32 = smem_u32(sI), sX32 = smem_u32(sX), sG32 = smem_u32(sG);
    const uint32_t mbarX = smem_u32(&mbar[0]), mbarG = smem_u32(&mbar[1]);
    const IO *gbase = grad_output + nc * F * (int64_t)npix;
    const uint32_t plane_bytes = (uint32_t)npix * (uint32_t)sizeof(IO);
    bool timed_out = false;

    Strip st[1] = {make_strip(g, sI32, warp, cg, rg)};

    // The first copies are started as early as possible, by a thread of the second warp (when there is
    // one) so that they do not queue behind the box arithmetic of the first warp's threads.  That thread
    // initialises the barriers itself and so needs no CTA barrier before it uses them; the other
    // threads first wait on them after the __syncthreads() below.
    const int starter = blockDim.x > 32 ? 32 : 0;
    if (STAGED && tid == starter) {
        mbar_init(mbarX, 1);
        mbar_init(mbarG, 1);
        fence_mbar_init();
        // While this CTA waits for the kernel in front of it, its first planes can already travel to L2
        // (a hint: if that kernel is still writing them, L2 receives its writes as well).
        bulk_prefetch_l2(gbase, plane_bytes);
        if (NEED_PARAMS && X_BY_COPY && !INTEG) bulk_prefetch_l2(x + nc * (int64_t)npix, plane_bytes);
        grid_dependency_wait();      // grad_output and the input may come from the kernel in front
        bulk_load(sG32, gbase, plane_bytes, mbarG);
        if (NEED_PARAMS && X_BY_COPY && !INTEG) bulk_load(sX32, x + nc * (int64_t)npix, plane_bytes, mbarX);
        if (F > 1) bulk_prefetch_l2(gbase + (int64_t)npix, plane_bytes);
    }
    init_integral_padding(sI, g);

    // registers and shared memory only up to here; now global memory that the kernel in front of
    // this one in the stream may still be using
    grid_dependency_wait();
    if (tid < F) {
        const Box box = load_box(bp, c * F + tid);
        store_taps(sTaps + tid * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
    }
    if (STAGED) __syncthreads();                           // barriers initialised before anyone waits
    if (NEED_PARAMS && INTEG) {
        // (read by the first gather, which follows the barriers of the first build)
        const float *I = x_integ + nc * (int64_t)(h + 1) * (w + 1);
        for (int p = warp; p < h; p += nwarps)
            for (int q = lane; q < w; q += 32) sX[p * w + q] = pixel_of_integral(I + p * (w + 1) + q, w + 1);
    } else if (!X_BY_COPY && NEED_PARAMS) {
        // (read by the first gather, which follows the barriers of the first build)
        const IO *xp = x + nc * (int64_t)npix;
        for (int i = tid; i < (npix >> 2); i += blockDim.x) reinterpret_cast<float4 *>(sX)[i] = Io<IO>::load4(xp + 4 * i);
    }

    float gin[kR][kStrip];
#pragma unroll
    for (int i = 0; i < kR; ++i)
#pragma unroll
        for (int m = 0; m < kStrip; ++m) gin[i][m] = 0.0f;

    for (int f = 0; f < F; ++f) {
        // (the barrier that ends the previous iteration protects sI, sRow, sCol)
        {
            Blocks<1> blk;
            if (STAGED) timed_out |= !mbar_wait(mbarG, f & 1);
            build_rows<IO, 1, true, STAGED>(blk, st, gbase + f * (int64_t)npix, sG32, sRow, g, cg, rg);
            if (STAGED && tid == 0 && f + 1 < F) {
                // every thread has taken its block out of the staging buffer (barrier above)
                fence_proxy_async();
                bulk_load(sG32, gbase + (f + 1) * (int64_t)npix, plane_bytes, mbarG);
                // the plane after that one on its way to L2 already (about 1 % on 256-sample batches)
                if (f + 2 < F) bulk_prefetch_l2(gbase + (f + 2) * (int64_t)npix, plane_bytes);
            }
            build_columns<1, true>(blk, st, sRow, sCol, g, cg, rg);
        }
        if (!STAGED && f + 1 < F && cg == 0) {
            // pull the next grad_output plane towards L2 while this one is gathered
#pragma unroll
            for (int i = 0; i < kR; ++i)
                if (st[0].active) asm volatile("prefetch.global.L2 [%0];" ::"l"(gbase + (f + 1) * (int64_t)npix + st[0].pix + i * w));
        }
        if (X_BY_COPY && NEED_PARAMS && !INTEG && f == 0) timed_out |= !mbar_wait(mbarX, 0);

        const BoxTaps t = load_taps(sTaps + f * kTapWords);
        const ColW2 cw = col_weights(t);
        // accumulators of this filter: see ParamSums.  The strip sums are kept per tap-row pair and
        // combined after the walk: sum x*(C-B) in *1, (sum x*(B-A), sum x*(D-C)) in *2.
        // sums over the strip of x times the column-strip values of the four tap rows, kept per
        // tap-row pair: *P = (row lo-1, row hi), *Q = (row lo, row hi+1); combined after the walk
        float s_out = 0.f;
        f2_t topbot2 = pack2(0.f, 0.f);
        f2_t leftP = pack2(0.f, 0.f), leftQ = pack2(0.f, 0.f), rightP = pack2(0.f, 0.f), rightQ = pack2(0.f, 0.f);
        if (st[0].active) {
            const int p0 = st[0].p0;
            const Walk wk = make_walk(sI32, t, st[0].q0, g);
            if (NEED_PARAMS) {
                f2_t pd[kStrip], pel[kStrip], peh[kStrip];
                load_pair_e(wk, p0 + t.lo_r - 1, p0 + t.hi_r, cw, pd, pel, peh);
                uint32_t xa = sX32 + st[0].pix * 4;
#pragma unroll
                for (int i = 0; i < kR; ++i) {
                    f2_t cd[kStrip], cel[kStrip], ceh[kStrip];
                    load_pair_e(wk, p0 + i + t.lo_r, p0 + i + t.hi_r + 1, cw, cd, cel, ceh);
                    const float4 x4 = lds128(xa);
                    const float xv[kStrip] = {x4.x, x4.y, x4.z, x4.w};
                    xa += w * 4;
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) {
                        const f2_t xx = pack2(xv[m], xv[m]);
                        float lo_new, hi_new, lo_old, hi_old, top, bot;
                        // d: gather value and the two row strips
                        const f2_t dd = sub2(cd[m], pd[m]);
                        unpack2(cd[m], lo_new, hi_new);
                        unpack2(pd[m], lo_old, hi_old);
                        unpack2(dd, top, bot);
                        const float gg = (hi_old - lo_new) + t.f_hi_r * bot + t.f_lo_r * top;
                        topbot2 = fma2(xx, dd, topbot2);
                        s_out += xv[m] * gg;
                        gin[i][m] += gg * t.scale;
                        // e_lo / e_hi: the two column strips
                        leftP = fma2(xx, pel[m], leftP);
                        leftQ = fma2(xx, cel[m], leftQ);
                        rightP = fma2(xx, peh[m], rightP);
                        rightQ = fma2(xx, ceh[m], rightQ);
                        pd[m] = cd[m]; pel[m] = cel[m]; peh[m] = ceh[m];
                    }
                }
            } else {
                f2_t prev[kStrip];
                load_pair(wk, p0 + t.lo_r - 1, p0 + t.hi_r, cw, prev);
#pragma unroll
                for (int i = 0; i < kR; ++i) {
                    f2_t cur[kStrip];
                    load_pair(wk, p0 + i + t.lo_r, p0 + i + t.hi_r + 1, cw, cur);
#pragma unroll
                    for (int m = 0; m < kStrip; ++m) {
                        float b, dd, a, cc, top, bot;
                        unpack2(cur[m], b, dd);
                        unpack2(prev[m], a, cc);
                        unpack2(sub2(cur[m], prev[m]), top, bot);
                        gin[i][m] += ((cc - b) + t.f_hi_r * bot + t.f_lo_r * top) * t.scale;
                        (void)a; (void)dd;
                        prev[m] = cur[m];
                    }
                }
            }
        }
        if (NEED_PARAMS) {
            float tb_top, tb_bot, la, lc, lb, ld, ra, rc, rb, rd;
            unpack2(topbot2, tb_top, tb_bot);
            unpack2(leftP, la, lc);
            unpack2(leftQ, lb, ld);
            unpack2(rightP, ra, rc);
            unpack2(rightQ, rb, rd);
            float v[kNumSums] = {s_out, tb_top, tb_bot,
                                 combine_rows(la, lb, lc, ld, t.f_lo_r, t.f_hi_r),
                                 combine_rows(ra, rb, rc, rd, t.f_lo_r, t.f_hi_r)};
#pragma unroll
            for (int j = 0; j < kNumSums; ++j) v[j] = warp_sum(v[j]);
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < kNumSums; ++j) red[warp][j] = v[j];
            }
        }
        __syncthreads();      // gathers of this filter are done: sI may be rebuilt; red[] is complete
        if (NEED_PARAMS && tid < kNumSums) {
            float s = 0.0f;
            for (int j = 0; j < nwarps; ++j) s += red[j][tid];
            partials[((int64_t)(c * F + f) * N + n) * kNumSums + tid] = s;
        }
        // red[] is next written after the barriers inside the next build
    }
    if (STAGED && timed_out && lane == 0) atomicAdd(&g_wait_timeouts, 1);

    if (write_gin && st[0].active) {
        IO *dst = grad_input + nc * (int64_t)npix + st[0].pix;
#pragma unroll
        for (int i = 0; i < kR; ++i, dst += w) Io<IO>::store4(dst, gin[i][0], gin[i][1], gin[i][2], gin[i][3]);
    }
    if (COUNTED) finish_if_last(fin, partials, bp, c, C, F, normalize, exact);
}

// The limit is raised to its maximum once per kernel and device (it is a ceiling, not a reservation: what a
// launch occupies is what it asks for), so that threads launching different sizes do not lower it for
// one another and a launch does not pay for the call.
template <class K>
int opt_in_smem(K kernel, size_t bytes)
{
    if (bytes <= 34 * 1024) return BC_OK;     // static scratch included, this stays under the 48 KB default
    return raise_smem_limit(reinterpret_cast<const void *>(kernel), kMaxSmem);
}

inline size_t plane_forward_smem_bytes(int h, int w)
{
    return ((size_t)layout_floats(h, w) + 2 * (size_t)warp_tiles(h, w) * kTile) * sizeof(float);
}

// io_bytes: element size of the staged grad_output plane
inline size_t plane_backward_smem_bytes(int h, int w, bool need_params, bool staged, size_t io_bytes)
{
    return plane_forward_smem_bytes(h, w) + (need_params ? (size_t)h * w * sizeof(float) : 0) +
           (staged ? (size_t)h * w * io_bytes : 0);
}

// (A rule on numbers of planes and alignments chooses between the kernel in 32 x 32 tiles and strips, so the plane has to fit both.)
inline bool plane_fits_forward(int F, int h, int w)
{
    return F <= kMaxFilters && warp_tiles(h, w) <= kMaxTiles && plane_forward_smem_bytes(h, w) <= kMaxSmem && flat_fits_forward(F, h, w);
}

// Forward from the input's integral image: copying it to shared memory pays where several filters, or several CTAs an
// SM, share the copy's latency ((4,16,4,96,160): 13 us, straight from global memory 23; 3060 planes of 120 x 56, F = 3: 96, 316).
// Not for one or two filters of large planes, which have an SM to themselves ((83,20,1,97,199): 180 against 115;
// (65,11,2,224,120): 163 against 106), nor where few such planes leave most SMs idle, which the tiles of the global kernel do
// not ((1,11,6,166,135): 23 against 15; (2,5,6,176,40): 12 against 8.5).
inline bool plane_prefers_global_forward_integ(int64_t planes, int F, int h, int w)
{
    const int tiles = warp_tiles(h, w);
    return (F <= 2 && tiles >= 16) || (planes * 8 <= 148 && tiles >= 12);
}

// (Planes of more than 32 tiles of 32 x 32 would fit the kernel that deals out strips in part; with 25 to 32 tiles of its own it is no better than slabs.)
inline bool plane_fits_backward(int F, int h, int w) { return warp_tiles(h, w) <= kMaxTiles && flat_fits_backward(F, h, w); }

// From the input's integral image, large planes are better off as slabs where they are wide enough or leave half of
// the SMs idle ((8,1,1,43,326): 13.2 us against 16.8; (43,1,6,176,108), 19 tiles of strips: 38, 62), unless 12 tiles of strips hold them and few samples
// spread their filters over CTAs or many fill the GPU ((573,1,6,29,336): 174, 132; (17,1,6,24,338): 24, 18; but (45,1,8,20,396): 32, 50).
// 13 to 16 tiles of strips with four filters or more (few rows: six) take a CTA an SM, or two of two tiles a warp, and win where the GPU is full of them.
// Filters over CTAs, all at once: with one each ((1,1,8,40,328) 26.4 us as slabs, 19.7; (2,1,4,86,175) 20.0, 20.8), eight filters or more ((20,1,8,80,188)
// 34, 29; (10,1,16,203,64) 53, 31; in two rounds (37,1,8,75,194) 40, 59), or half of the SMs at work ((4,16,4,96,160) 31.8, 27.3; (34,1,4,190,78), 46 %,
// 27, 30).  Not shared: 60 % at work ((8,16,4,96,160) 53, 35; (16,16,4,96,160) 91, 68; (64,16,4,96,160) 309, 220; (16,16,6,104,144) 146, 96;
// (180,5,6,88,144) 379, 291; but (25,2,32,95,134), 34 %, 163, 246; (37,2,6,72,208), half, 41, 49; (80,2,8,88,144), 54 %, 108, 112), with fewer rows, which
// slabs cut less, 88 % ((74,2,6,48,340) 71, 51; (45,2,8,25,446), 61 %, 52, 67; (125,2,32,26,395), 84 %, 434, 551).  Of 216 drawn launches: always
// slabs 1, always strips 0.99 of that time, by this rule 0.90.
inline bool plane_prefers_slabs_backward(int64_t planes, int F, int h, int w)
{
    const int strips = ((w + 3) / 4) * ((h + 7) / 8);
    if ((w <= 96 && planes > 74) || warp_tiles(h, w) <= 8 || quad_fits_backward(F, h, w)) return false;
    if (strips <= 12 * 32) return planes > 20 && planes <= 148;
    if (strips > 16 * 32 || F < (h >= 64 ? 4 : 6)) return true;
    const FlatPlan p = flat_backward_plan((int)(planes < 0x7fffffff ? planes : 0x7fffffff), 1, F, h, w, true);
    if (p.sh.split > 1) return p.rounds > 1 || (p.each > 1 && F < 8 && p.full < 50);
    return p.full < (h >= 64 ? 60 : 88);
}

// On which planes the kernel that deals out strips (box_flat.cu) is faster than those with fixed tiles: it has fewer lanes without a
// pixel, and a fifth more instructions a strip.  `strips`: a 32nd of its tiles.  Samples, channels, filters, rows, columns:
// against 8 x 128 tiles (795,2,4,40,150) 201 us -> 130; (2611,1,4,120,72) 438 -> 308; (202,3,4,48,144) 83 -> 64; but (1265,1,2,56,96), 7 tiles
// for 5.25, 53.6 -> 56.8; (2104,1,4,80,120), 10 for 9.4, 213 -> 260; (111,8,6,86,126) 179 -> 209;
// against pairs of them, or few planes of which one tile a warp: (575,1,4,128,72) 88 -> 76; (593,1,4,72,168) 166 -> 103; (653,1,8,80,240), 20 for 18.8, 318 ->
// 404; 14 and 16 tiles for two thirds of them to nine tenths (1500,1,8,112,92) 391 -> 424, (148,1,6,56,176) 34.8 -> 39.8, (149,1,8,64,200) 80 -> 102, though with
// few planes, whose filters strips spread over a cluster, (37,1,6,64,200) 35.7 -> 26.0; with one or two filters up to 148 planes
// (148,1,2,128,76) 16.3 -> 18.6, (37,1,2,64,140) 15.8 -> 15.0, above a wash but for the emptiest (700,1,2,56,136) 58 -> 45;
// against 32 x 32 tiles, more than eight: always (below); fewer, aligned: (1042,1,8,72,40) 144 -> 83; (64,40), 4 for 2.5, 61 -> 62, with fewer
// planes 1.1 to 1.4 times as long; unaligned (2857,1,6,47,36) 233 -> 106, (2858,1,4,110,36) in bfloat16 424 -> 149.
// The rules ask for sides and filters only: kernels of different tiles add up in different orders, and a part of a batch is to
// get the grad-input of the whole to the last bit.
inline bool flat_beats_quad(int F, int h, int w)
{
    const int tiles = quad_row_tiles(h) * quad_col_tiles(w), strips = ((w + 3) / 4) * ((h + 7) / 8);
    if (tiles <= 8) return F > 1 && tiles * 32 * 10 > strips * 16;
    if (strips > 12 * 32) return tiles * 32 * 10 > strips * 12;
    return tiles * 32 * 10 > strips * (w % 4 || h % 8 ? 13 : 15);
}
inline bool flat_beats_pair(int F, int h, int w)
{
    const int tiles = quad_row_tiles(h) * quad_col_tiles(w), strips = ((w + 3) / 4) * ((h + 7) / 8);
    if (F <= 2) return false;
    if (tiles <= kQuadMaxWarps) return tiles * 32 * 10 > strips * 15;
    return strips <= 24 * 32 && tiles * 32 * 20 > strips * 25;
}
inline bool flat_beats_square(int F, int h, int w)
{
    const int tiles = warp_tiles(h, w), strips = ((w + 3) / 4) * ((h + 7) / 8);
    return F > 1 && tiles > 4 && tiles * 32 * 10 > strips * 17;
}

// The backward kernel of a plane.  `pair_rows`: the input itself is given and all addresses fit the pair kernel's accesses; `fast`: rows and addresses
// fit vector accesses.  The number of planes decides between the two kernels of 8 x 128 tiles, which add up alike, and, with one or two filters, between
// pairs of them and strips for planes of 72 to 96 rows and 132 to 160 columns: only there does a part of a batch get another order of additions.
enum PlaneBackward { BACKWARD_PAIR, BACKWARD_QUAD, BACKWARD_SQUARE, BACKWARD_STRIPS };
inline PlaneBackward plane_backward_choice(int64_t planes, int F, int h, int w, bool wide, bool pair_rows, bool fast)
{
    const bool pairs = pair_rows && quad_pair_fits_backward(F, h, w, wide);
    if (!(pairs ? flat_beats_pair(F, h, w) : flat_beats_quad(F, h, w))) {
        if (pairs && quad_pair_suits_backward(planes, F, h, w, wide)) return BACKWARD_PAIR;
        if (quad_fits_backward(F, h, w)) return BACKWARD_QUAD;
    }
    return !fast || w >= kQuadMinWidth || warp_tiles(h, w) > 8 || flat_beats_square(F, h, w) ? BACKWARD_STRIPS : BACKWARD_SQUARE;
}

// The same in the forward, by the fixed tiles that it has or else would have (`quad`: of 8 x 128).
// More than eight of 32 x 32: where rows are cut or unaligned ((1050,1,8,134,33), 10 tiles for 4.8, 122 us against 85; 139 drawn planes 0.77 of the time), where
// they waste more than a quarter ((693,1,1,48,280) 37.7 and 27.5; (419,1,3,272,40) 40.9 and 27.0; 40 planes 0.8; below that 1.03 to 1.15: (1239,1,1,128,96) 36 and
// 41, (1221,1,4,88,144) 91 and 104), and of few samples ((3,1,4,280,96) 9.5 and 7.9; 25 planes 0.85).  Up to eight, with filters' CTAs to hand and several on
// an SM, they are as fast or faster.
// Against more than eight of 8 x 128: where rows are cut or unaligned, or two fifths of the lanes idle ((6,3,4,184,77) 8.9 and 6.9, (14,8,4,35,224) 16.8 and 10.1;
// 41 such planes 0.81).
// Not against 8 x 128 of a few planes so large that these are split by rows ((5,1,4,112,246) fused 10.6 us, 13.5; (3,1,4,214,115) 8.9, 10.4), nor with one or
// two filters of some ((64,1,1,91,159) 9.0, 10.9; (15,1,1,168,90) 7.6, 8.6; fused ones gain).
// Unlike the backward's, these rules ask for the number of planes: outputs of a part of a batch that crosses a line agree with the whole's to rounding.
inline bool flat_suits_forward(int64_t planes, int F, int h, int w, bool quad, bool aligned, bool fused)
{
    const int tiles = quad ? quad_row_tiles(h) * quad_col_tiles(w) : warp_tiles(h, w), strips = ((w + 3) / 4) * ((h + 7) / 8);
    if (tiles <= 8 || (quad && planes <= 6 && strips > 20 * 32)) return false;
    if (quad && !fused && F <= 2 && planes < 100 && strips > 8 * 32) return false;
    return !aligned || (!quad && planes < 40) || tiles * 32 * 100 > strips * (quad ? 160 : 128);
}
// From the input's integral image: of few samples also smaller planes (51 aligned ones 0.87, 59 unaligned ones 0.96 of the time), but not of one
// to four square tiles ((12,16,4,20,58) 8.0 us, 9.3; (1,90,8,38,41) 10.5, 13.6), nor with many filters ((1,93,8,30,75) 12.3, 14.2).
inline bool flat_suits_forward_integ(int64_t planes, int F, int h, int w, bool quad)
{
    const int tiles = quad ? quad_row_tiles(h) * quad_col_tiles(w) : warp_tiles(h, w);
    return tiles > 8 || (planes < 600 && (quad ? planes * F < 400 : tiles > 4));
}

// `fu` (inference steps around the gather) exists for float tensors only.
template <typename IO>
int launch_forward_plane_t(const IO *x, const float *integ, const BoxParams &bp, const Fusion *fu, IO *out, int N, int C, int F, int h,
                           int w, bool normalize, bool exact, cudaStream_t s)
{
    if (x && !fu && tmem_suits_forward((int64_t)N * C, F, h, w) && aligned_to(x, Io<IO>::kVecBytes) && aligned_to(out, Io<IO>::kVecBytes))
        return launch_forward_tmem_t<IO>(x, bp, out, N, C, F, h, w, normalize, exact, s);
    const int64_t planes = (int64_t)N * C;
    const int vec = Io<IO>::kVecBytes;
    const bool fast = (h % kR == 0) && (w % kStrip == 0) && aligned_to(x, vec) && aligned_to(out, vec) &&
                      (!fu || !fu->residual || aligned_to(fu->residual, 16));
    const bool quad = quad_fits_forward(F, h, w) && (x ? quad_prefers_forward(planes, F, h, w) : quad_prefers_forward_integ(planes, F, h, w));
    if (x ? flat_suits_forward(planes, F, h, w, quad, fast, fu != nullptr) : flat_suits_forward_integ(planes, F, h, w, quad))
        return launch_forward_flat(x, integ, Io<IO>::kKind, bp, fu, out, N, C, F, h, w, normalize, exact, s);
    if (quad) return launch_forward_quad_t<IO>(x, integ, bp, fu, out, N, C, F, h, w, normalize, exact, s);
    // Split the filters of a plane over two CTAs when there are too few planes to balance 148 SMs
    // (each part rebuilds the integral image; the second read of the plane comes from L2).
    int fsplit = 1;
    if (F % 2 == 0 && planes < 148 * 6) fsplit = 2;
    while (fsplit < F && F % (fsplit * 2) == 0 && planes * fsplit * 2 <= 148 * 2) fsplit *= 2;   // tiny batches: fill the SMs
    if (planes * fsplit > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const size_t smem = plane_forward_smem_bytes(h, w);
    const int tiles = warp_tiles(h, w);
    // one tile per warp up to 8 tiles, two beyond (up to 16 warps: a CTA of a large plane has the SM to itself)
    const int T = tiles > 8 ? 2 : 1;
    if (T == 2 && !(fast && x)) return BC_ERR_UNSUPPORTED;      // (flat_suits_forward() has taken those)
    const int warps = (tiles + T - 1) / T;
    void (*kern)(const IO *, const float *, BoxParams, IO *, int, int, int, int, int, bool, bool, Fusion);
    constexpr bool FL = IsFloat<IO>::value;      // (integral images are float)
    if (fu && !FL) return BC_ERR_UNSUPPORTED;
    if (T == 2) kern = fu ? forward_plane_kernel<IO, 2, true, FL> : forward_plane_kernel<IO, 2, true>;
    else if (!x) kern = fast ? forward_plane_kernel<IO, 1, true, false, FL> : forward_plane_kernel<IO, 1, false, false, FL>;
    else if (fu) kern = fast ? forward_plane_kernel<IO, 1, true, FL> : forward_plane_kernel<IO, 1, false, FL>;
    else kern = fast ? forward_plane_kernel<IO, 1, true> : forward_plane_kernel<IO, 1, false>;
    int st = opt_in_smem(kern, smem);
    if (st != BC_OK) return st;
    const Fusion none{0, nullptr, nullptr, nullptr, 0};
    {
        LaunchScope scope(KID_FORWARD_PLANE, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)(planes * fsplit), warps * 32, smem, s, x, integ, bp, out, C, F, h, w,
                                              fsplit, normalize, exact, fu ? *fu : none))
            return cuda_failed(e, "forward_plane");
    }
    return check_launch("forward_plane");
}

template <typename IO>
int launch_backward_plane_t(const IO *x, const float *x_integ, const IO *grad_output, const BoxParams &bp, float rep_h, float rep_w, int N,
                            int C, int F, int h, int w, bool normalize, bool exact, int need_mask, IO *grad_input,
                            void *grad_params, int grad_params_kind, float *partials, cudaStream_t s)
{
    const int64_t planes = (int64_t)N * C;
    if (planes > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    const bool need_params = (need_mask & (BC_NEED_ALL & ~BC_NEED_INPUT)) != 0;
    const bool write_gin = (need_mask & BC_NEED_INPUT) != 0;
    const int vec = Io<IO>::kVecBytes;
    const bool fits = aligned_to(x, vec) && (!write_gin || aligned_to(grad_input, vec));
    const PlaneBackward choice = plane_backward_choice(planes, F, h, w, IsFloat<IO>::value, x && fits && aligned_to(grad_output, 16),
                                                       h % kR == 0 && w % kStrip == 0 && fits && aligned_to(grad_output, vec));
    if (choice == BACKWARD_PAIR)
        return launch_backward_quad_pair_t<IO>(x, grad_output, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact, need_mask, grad_input, grad_params,
                                               grad_params_kind, partials, s);
    if (choice == BACKWARD_QUAD)
        return launch_backward_quad_t<IO>(x, x_integ, grad_output, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact, need_mask, grad_input,
                                          grad_params, grad_params_kind, partials, s);
    if (choice == BACKWARD_STRIPS)
        return launch_backward_flat(x, x_integ, Io<IO>::kKind, grad_output, bp, rep_h, rep_w, N, C, F, h, w, normalize, exact, need_mask, grad_input,
                                    grad_params, grad_params_kind, partials, s);
    const int tiles = warp_tiles(h, w);
    const size_t io = sizeof(IO);
    // bulk copies need 16-byte aligned planes of a multiple of 16 bytes and room for the staging buffer;
    // staging must not cost a resident CTA (two fit below ~112 KB each)
    const size_t two_ctas = 112 * 1024;
    const size_t with_staging = plane_backward_smem_bytes(h, w, need_params, true, io);
    const bool staged = with_staging <= kMaxSmem && aligned_to(grad_output, 16) && aligned_to(x, 16) && ((size_t)h * w * io) % 16 == 0 &&
                        (with_staging <= two_ctas || plane_backward_smem_bytes(h, w, need_params, false, io) > two_ctas);
    const size_t smem = plane_backward_smem_bytes(h, w, need_params, staged, io);
    void (*kern)(const IO *, const float *, const IO *, BoxParams, IO *, float *, int, int, int, int, int, bool, bool, bool, Finish);
    // With the input plane in shared memory, finishing here costs more than the launch it saves, from all but the
    // smallest problems on ((18,14,8,40,56): 41 us against 32 with the launch; (9,12,4,248,48): 67 against 53; (1,8,4,32,32): 17 against 14.5
    // and 3 us of the host).
    const int64_t outputs = planes * F * h * w;
    const bool may_finish = need_params && planes <= 148 && outputs <= 256 * 1024;
    const Finish fin = finish_here(bp, may_finish, planes, outputs, C, grad_params, grad_params_kind, need_mask, N, rep_h, rep_w, s);
    auto pick = [&](auto copied) {
        constexpr bool S = decltype(copied)::value;
        if (!need_params) kern = backward_square_kernel<IO, S, false>;
        else if (x_integ) kern = backward_square_kernel<IO, S, true, false, IsFloat<IO>::value>;      // (the four functions have no counters)
        else kern = fin.total ? backward_square_kernel<IO, S, true, true> : backward_square_kernel<IO, S, true>;
    };
    if (staged) pick(Flag<true>{});
    else pick(Flag<false>{});
    int st = opt_in_smem(kern, smem);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_SQUARE, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)planes, tiles * 32, smem, s, x, x_integ, grad_output, bp, grad_input,
                                              partials, N, C, F, h, w, normalize, exact, write_gin, fin))
            return cuda_failed(e, "backward_square");
    }
    st = check_launch("backward_square");
    if (st != BC_OK || !need_params || fin.total) return st;
    return launch_finish_param_grads<float>(partials, bp, C * F, N, normalize, exact, rep_h, rep_w, need_mask,
                                            grad_params, s, grad_params_kind);
}

}  // namespace

}  // namespace bc
