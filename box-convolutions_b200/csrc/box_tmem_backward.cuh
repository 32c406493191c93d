// Whole-plane backward, one axis after the other, for planes of one column tile whose combined rows fit tensor memory.
//
// With G a grad_output plane, grad-input adds up a box of G around every pixel, and the parameter gradients need that box and its
// four one-pixel border strips, each summed up against the input X.  The other backward kernels take both from the
// corners of a 2-D integral image, 20 words of shared memory and about 180 instructions a row of 128 pixels and warp.  Here
// a row of G is first combined along the row, from its own prefix sums, into R (the box's width), e_lo and e_hi (the pixels
// beside the box); nothing but the warp that holds the row takes part.  Then
//   * running sums of R down the columns, D, go to tensor memory, from where two rows of D give a row of grad-input;
//   * the five sums are turned round: with XV the box of X, taken down the columns around the row of G,
//     sum_p X(p) (sum of e over the box's rows at p) = sum_g e(g) XV(g), and likewise for R; the strips above and
//     below the box need single rows of X.  XV and those rows are differences of rows of X's running sums down the columns,
//     which lie in shared memory once a plane.
// About 100 instructions and two thirds of the shared-memory words.  Sums along a row or down a column are of h or w values where
// those of an integral image are of h w, so less is lost when they are subtracted.
//
// A plane belongs to four warps of the same number modulo 4, which reach the same lanes of tensor memory: 4 h columns for D, as many for
// the grad-input accumulators.  A CTA has four such groups, each with planes of its own and barriers of its own, and an SM one CTA.
#pragma once
#include "box_tmem_plane.cuh"

namespace bc {

namespace {

constexpr int kFlowRows = 64;                   // rows of a plane: D and the accumulators share 512 columns
constexpr int kFlowCells = 35;                  // of a sub-row of a pair of prefix rows: 128 columns, quad layout, 8 bytes a cell
constexpr int kFlowPair = 4 * kFlowCells * 8;   // bytes of a pair
constexpr int kFlowWarp = 2 * kFlowPair + kScanBytes;      // a warp's two pairs and scan corner

// Shared memory of a group: X's running sums (h + 1 rows of 128), the warps' scratch, last rows and sums, the boxes.
__host__ __device__ inline int flow_group_bytes(int F, int h) { return (h + 1) * 512 + 4 * (kFlowWarp + 512 + 32) + F * kTapWords * 4; }

template <int OFF>
__device__ __forceinline__ f2_t lds2(uint32_t a)
{
    f2_t v;
    asm volatile("ld.shared.b64 %0, [%1+%2];" : "=l"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF>
__device__ __forceinline__ void sts2(uint32_t a, f2_t v)
{
    asm volatile("st.shared.b64 [%0+%1], %2;" ::"r"(a), "n"(OFF), "l"(v) : "memory");
}

// Rows of four columns a lane, fetched a batch ahead and converted where they are used.
template <typename IO>
struct RawRow { uint2 v; };
template <>
struct RawRow<float> { float4 v; };
template <typename IO>
__device__ __forceinline__ void raw_load(RawRow<IO> &r, const IO *p, bool there)
{
    if constexpr (IsFloat<IO>::value) {
        if (there) asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r.v.x), "=f"(r.v.y), "=f"(r.v.z), "=f"(r.v.w) : "l"(p));
        else r.v = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        if (there) asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(r.v.x), "=r"(r.v.y) : "l"(p));
        else r.v = make_uint2(0u, 0u);
    }
}
template <typename IO>
__device__ __forceinline__ float4 raw_get(const RawRow<IO> &r)
{
    if constexpr (IsFloat<IO>::value) return r.v;
    else return Io<IO>::widen(r.v);
}

template <typename IO>
__global__ void __launch_bounds__(512, 1)
backward_tmem_kernel(const IO *__restrict__ x, const IO *__restrict__ grad_output, BoxParams bp, IO *__restrict__ grad_input,
                     float *__restrict__ partials, int planes, int N, int C, int F, int h, int w, bool normalize, bool exact)
{
    extern __shared__ float4 smem4[];
    __shared__ uint32_t tmem_base;
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), group = warp & 3, part = warp >> 2;
    const int npix = h * w, cells = quad_cells(w), group_bytes = flow_group_bytes(F, h);
    const uint32_t vx = smem_u32(smem4) + group * group_bytes;                 // X's running sums: row k (0 .. h) at 512 k
    const uint32_t pairs = vx + (h + 1) * 512 + part * kFlowWarp, scan = pairs + 2 * kFlowPair;
    const uint32_t last32 = vx + (h + 1) * 512 + 4 * kFlowWarp;
    float *sTaps = reinterpret_cast<float *>(reinterpret_cast<char *>(smem4) + group * group_bytes + (h + 1) * 512 + 4 * (kFlowWarp + 512 + 32));
    float *red = sTaps - 4 * 8;
    const int q0 = lane * kStrip;
    const bool inside = q0 < w;

    // what never changes: row 0 of X's sums; the first cells and column 0 of the prefix rows
    if (part == 0) sts128(vx + lane * 16, make_float4(0.f, 0.f, 0.f, 0.f));
    if (lane < 10) {
        const int b = lane / 5, k = lane - 5 * b;
        sts2<0>(pairs + b * kFlowPair + (k < 4 ? k * kFlowCells * 8 : 8), 0ull);
    }
    __syncwarp();
    grid_dependency_wait();
    if (warp == 0) tmem_alloc(&tmem_base, 512);
    __syncthreads();
    tmem_acquire();
    const uint32_t rows32 = tmem_base + ((uint32_t)group << 21), gin32 = rows32 + 4 * kFlowRows;

    const int row_tiles = h / kTileRows, part_rows = (row_tiles + 3) / 4 * kTileRows;
    const int r_begin = part * part_rows, r_end = min(r_begin + part_rows, h);
    const int batches = max(r_end - r_begin, 0) / kTileRows;
    const int stride = 4 * gridDim.x;
    auto meet = [&] {
        tmem_release();
        unit_barrier(1 + group, 128);
        tmem_acquire();
    };

    RawRow<IO> v[kTileRows];
    int plane = blockIdx.x + group * gridDim.x;
    if (plane < planes && batches) {
        const IO *p = grad_output + (int64_t)plane * F * npix + r_begin * w + q0;
#pragma unroll
        for (int i = 0; i < kTileRows; ++i) raw_load(v[i], p + i * w, inside);
    }
    for (; plane < planes; plane += stride) {
        const int c = plane % C, n = plane / C;
        const bool more = plane + stride < planes;
        if (!more) grid_dependency_release();      // (any earlier, and the next kernel's CTAs would wait on SMs that are still at work)
        else if (part == 0 && lane == 0) bulk_prefetch_l2(x + (int64_t)(plane + stride) * npix, npix * (uint32_t)sizeof(IO));
        // X's running sums down the columns: the warp's rows, then what the parts above have
        if (part == 0 && lane < F) {
            const Box box = load_box(bp, c * F + lane);
            store_taps(sTaps + lane * kTapWords, taps_mirrored(box.xmin, box.xmax, box.ymin, box.ymax, normalize, exact));
        }
        {
            float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
            const IO *p = x + (int64_t)plane * npix + r_begin * w + q0;
            for (int b = 0; b < batches; ++b, p += kTileRows * w) {
                RawRow<IO> e[kTileRows];
#pragma unroll
                for (int i = 0; i < kTileRows; ++i) raw_load(e[i], p + i * w, inside);
#pragma unroll
                for (int i = 0; i < kTileRows; ++i) {
                    const float4 a = raw_get<IO>(e[i]);
                    run.x += a.x; run.y += a.y; run.z += a.z; run.w += a.w;
                    sts128(vx + (r_begin + b * kTileRows + i + 1) * 512 + lane * 16, run);
                }
            }
            sts128(last32 + part * 512 + lane * 16, run);
            unit_barrier(1 + group, 128);
            float4 up = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int k = 0; k < part; ++k) {
                const float4 a = lds128(last32 + k * 512 + lane * 16);
                up.x += a.x; up.y += a.y; up.z += a.z; up.w += a.w;
            }
            if (part) {
                for (int r = r_begin + 1; r <= r_end; ++r) {
                    const uint32_t at = vx + r * 512 + lane * 16;
                    float4 a = lds128(at);
                    a.x += up.x; a.y += up.y; a.z += up.z; a.w += up.w;
                    sts128(at, a);
                }
            }
            unit_barrier(1 + group, 128);
        }
        for (int f = 0; f < F; ++f) {
            const BoxTaps t = load_taps_uniform(sTaps + f * kTapWords);
            if (part == 0 && lane == 0 && (f + 1 < F || more))      // the plane after this one on its way to L2
                bulk_prefetch_l2(grad_output + (f + 1 < F ? (int64_t)plane * F + f + 1 : (int64_t)(plane + stride) * F) * npix, npix * (uint32_t)sizeof(IO));
            float s_out = 0.f, s_top = 0.f, s_bot = 0.f, s_left = 0.f, s_right = 0.f;
            float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
            if (batches) {
                uint32_t lo[kStrip + 1], hi[kStrip + 1];
                {
                    const QuadCols cols = quad_cols(t, lane, cells, kFlowCells);
#pragma unroll
                    for (int m = 0; m <= kStrip; ++m) {
                        lo[m] = pairs + 2 * cols.lo[m];      // (8 bytes a cell)
                        hi[m] = pairs + 2 * cols.hi[m];
                    }
                }
                const f2_t fl = pack2(t.f_lo_c, t.f_lo_c), fh = pack2(t.f_hi_c, t.f_hi_c);
                const f2_t gl = pack2(t.f_lo_r, t.f_lo_r), gh = pack2(t.f_hi_r, t.f_hi_r);
                auto vx_row = [&](int k) { return lds128(vx + min(max(k, 0), h) * 512 + lane * 16); };
                // X's sums up to the rows that enter and leave the box around row g
                float4 xu = vx_row(r_begin - t.lo_r + 1), xv = vx_row(r_begin - t.hi_r);
                for (int b = 0; b < batches; ++b) {
                    const int g0 = r_begin + b * kTileRows;
                    // where the batch after this one begins (the last one is fetched again)
                    const IO *next = grad_output + ((int64_t)plane * F + f) * npix + (g0 + kTileRows) * w + q0;
                    if (b + 1 == batches) {
                        if (f + 1 < F) next = grad_output + ((int64_t)plane * F + f + 1) * npix + r_begin * w + q0;
                        else next = grad_output + (int64_t)(more ? plane + stride : plane) * F * npix + r_begin * w + q0;
                    }
                    float4 e[kTileRows];
                    float carry[kTileRows];
#pragma unroll
                    for (int i = 0; i < kTileRows; ++i) {
                        e[i] = raw_get<IO>(v[i]);
                        e[i].y += e[i].x; e[i].z += e[i].y; e[i].w += e[i].z;
                        carry[i] = e[i].w;
                    }
                    rows8_before(scan, carry, lane);
                    auto two_rows = [&](auto I) {
                        constexpr int i = decltype(I)::value, kAt = (i >> 1 & 1) * kFlowPair;
                        float4 a = e[i], d = e[i + 1];
                        a.x += carry[i]; a.y += carry[i]; a.z += carry[i]; a.w += carry[i];
                        d.x += carry[i + 1]; d.y += carry[i + 1]; d.z += carry[i + 1]; d.w += carry[i + 1];
                        // columns past w hold exactly what column w holds
                        const float la = __shfl_sync(0xffffffffu, a.w, (w - 1) >> 2), ld = __shfl_sync(0xffffffffu, d.w, (w - 1) >> 2);
                        if (w < 128 && !inside) {
                            a = make_float4(la, la, la, la);
                            d = make_float4(ld, ld, ld, ld);
                        }
                        const uint32_t at = pairs + (lane + 1) * 8;
                        sts2<kAt + kFlowCells * 8>(at, pack2(a.x, d.x));
                        sts2<kAt + 2 * kFlowCells * 8>(at, pack2(a.y, d.y));
                        sts2<kAt + 3 * kFlowCells * 8>(at, pack2(a.z, d.z));
                        sts2<kAt + 8>(at, pack2(a.w, d.w));
                        if ((w >> 2) + 2 > 32 && lane < 7)
                            sts2<kAt>(pairs + (lane < 3 ? lane + 1 : lane - 3) * (kFlowCells * 8) + (lane < 3 ? 33 : 34) * 8, pack2(la, ld));
                        raw_load(v[i], next + i * w, inside);
                        raw_load(v[i + 1], next + (i + 1) * w, inside);
                        // X around rows g and g + 1
                        const float4 u0 = vx_row(g0 + i - t.lo_r + 2), w0 = vx_row(g0 + i - t.hi_r + 1);
                        const float4 u1 = vx_row(g0 + i - t.lo_r + 3), w1 = vx_row(g0 + i - t.hi_r + 2);
                        __syncwarp();
                        f2_t l[kStrip + 1], r[kStrip + 1];
#pragma unroll
                        for (int m = 0; m <= kStrip; ++m) {
                            l[m] = lds2<kAt>(lo[m]);
                            r[m] = lds2<kAt>(hi[m]);
                        }
                        float xt[2][4], xb[2][4], xx[2][4];
                        auto around = [&](const float4 &u, const float4 &z, float (&top)[4], float (&bot)[4], float (&box)[4]) {
                            auto half = [&](f2_t u_, f2_t z_, f2_t pu, f2_t pz, int m) {
                                const f2_t tt = sub2(u_, pu), bb = sub2(z_, pz);
                                unpack2(tt, top[m], top[m + 1]);
                                unpack2(bb, bot[m], bot[m + 1]);
                                unpack2(fma2(gh, bb, fma2(gl, tt, sub2(pu, z_))), box[m], box[m + 1]);
                            };
                            half(pack2(u.x, u.y), pack2(z.x, z.y), pack2(xu.x, xu.y), pack2(xv.x, xv.y), 0);
                            half(pack2(u.z, u.w), pack2(z.z, z.w), pack2(xu.z, xu.w), pack2(xv.z, xv.w), 2);
                            xu = u;
                            xv = z;
                        };
                        around(u0, w0, xt[0], xb[0], xx[0]);
                        around(u1, w1, xt[1], xb[1], xx[1]);
                        float sum[2][4];
#pragma unroll
                        for (int m = 0; m < kStrip; ++m) {
                            const f2_t el = sub2(l[m + 1], l[m]), eh = sub2(r[m + 1], r[m]);
                            const f2_t box = fma2(fl, el, fma2(fh, eh, sub2(r[m], l[m + 1])));
                            float p0, p1;
                            unpack2(box, sum[0][m], sum[1][m]);
                            s_out = fmaf(sum[0][m], xx[0][m], s_out); s_out = fmaf(sum[1][m], xx[1][m], s_out);
                            s_top = fmaf(sum[0][m], xt[0][m], s_top); s_top = fmaf(sum[1][m], xt[1][m], s_top);
                            s_bot = fmaf(sum[0][m], xb[0][m], s_bot); s_bot = fmaf(sum[1][m], xb[1][m], s_bot);
                            unpack2(el, p0, p1);
                            s_left = fmaf(p0, xx[0][m], s_left); s_left = fmaf(p1, xx[1][m], s_left);
                            unpack2(eh, p0, p1);
                            s_right = fmaf(p0, xx[0][m], s_right); s_right = fmaf(p1, xx[1][m], s_right);
                        }
                        float4 d0, d1;
                        d0.x = run.x + sum[0][0]; d0.y = run.y + sum[0][1]; d0.z = run.z + sum[0][2]; d0.w = run.w + sum[0][3];
                        d1.x = d0.x + sum[1][0]; d1.y = d0.y + sum[1][1]; d1.z = d0.z + sum[1][2]; d1.w = d0.w + sum[1][3];
                        run = d1;
                        __syncwarp();
                        tmem_store8(rows32 + 4 * (g0 + i), d0, d1);
                    };
                    two_rows(Index<0>{}); two_rows(Index<2>{}); two_rows(Index<4>{}); two_rows(Index<6>{});
                }
                tmem_wait_store();
            }
            sts128(last32 + part * 512 + lane * 16, run);
            {
                const float sums[kNumSums] = {s_out, s_top, s_bot, s_left, s_right};
                const float s = warp_sum5(sums, lane);
                const int slot = sum5_slot(lane);
                if (slot >= 0) red[part * 8 + slot] = s;
            }
            meet();
            if (part == 0 && lane < kNumSums)
                partials[((int64_t)(c * F + f) * N + n) * kNumSums + lane] = red[lane] + red[8 + lane] + red[16 + lane] + red[24 + lane];
            if (part && batches) {
                float4 up = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int k = 0; k < part; ++k) {
                    const float4 a = lds128(last32 + k * 512 + lane * 16);
                    up.x += a.x; up.y += a.y; up.z += a.z; up.w += a.w;
                }
                for (int r = r_begin; r < r_end; r += 4) {
                    float4 a[4];
                    __syncwarp();
                    tmem_load16(rows32 + 4 * r, a);
                    tmem_wait_load(a);
#pragma unroll
                    for (int i = 0; i < 4; ++i) { a[i].x += up.x; a[i].y += up.y; a[i].z += up.z; a[i].w += up.w; }
                    tmem_store16(rows32 + 4 * r, a);
                }
                tmem_wait_store();
            }
            meet();
            if (batches) {
                const TmemUnit unit{rows32, r_begin, r_end, h};
                IO *row = grad_input + (int64_t)plane * npix + r_begin * w + q0;
                tmem_box_rows<true>(unit, t, [&](int p, f2_t (&g)[4][2]) {
                    const f2_t scale = pack2(t.scale, t.scale);
                    float4 acc[4];
                    if (f) {
                        __syncwarp();
                        tmem_load16(gin32 + 4 * p, acc);
                        tmem_wait_load(acc);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const f2_t zero = 0ull;
                        unpack2(fma2(g[i][0], scale, f ? pack2(acc[i].x, acc[i].y) : zero), acc[i].x, acc[i].y);
                        unpack2(fma2(g[i][1], scale, f ? pack2(acc[i].z, acc[i].w) : zero), acc[i].z, acc[i].w);
                    }
                    if (f + 1 < F) {
                        __syncwarp();
                        tmem_store16(gin32 + 4 * p, acc);
                    } else if (inside) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) Io<IO>::store4(row + (p - r_begin + i) * w, acc[i].x, acc[i].y, acc[i].z, acc[i].w);
                    }
                });
                tmem_wait_store();
            }
            meet();      // the rows of D have been read
        }
    }
    tmem_release();
    __syncthreads();
    if (warp == 0) tmem_free(tmem_base, 512);
}

inline bool tmem_suits_backward(int64_t planes, int F, int h, int w)
{
    return w % 4 == 0 && h % kTileRows == 0 && w >= kQuadMinWidth && w <= 128 && h <= kFlowRows && F <= kMaxFilters &&
           4 * (size_t)flow_group_bytes(F, h) <= 220 * 1024 && planes >= 148;
}

template <typename IO>
int launch_backward_tmem_t(const IO *x, const IO *grad_output, const BoxParams &bp, int N, int C, int F, int h, int w, bool normalize, bool exact,
                           IO *grad_input, float *partials, cudaStream_t s)
{
    const int64_t planes = (int64_t)N * C;
    if (planes > 0x7fffffffLL - 4 * 148) return BC_ERR_BAD_SHAPE;
    void (*kern)(const IO *, const IO *, BoxParams, IO *, float *, int, int, int, int, int, int, bool, bool) = backward_tmem_kernel<IO>;
    int st = raise_smem_limit(reinterpret_cast<const void *>(kern), 220 * 1024);
    if (st != BC_OK) return st;
    {
        LaunchScope scope(KID_BACKWARD_QUAD, s);
        if (cudaError_t e = launch_overlapped(kern, (unsigned)std::min<int64_t>(planes, 148), 512, 4 * flow_group_bytes(F, h), s, x, grad_output, bp, grad_input,
                                              partials, (int)planes, N, C, F, h, w, normalize, exact))
            return cuda_failed(e, "backward_tmem");
    }
    return check_launch("backward_tmem");
}

}  // namespace

}  // namespace bc
