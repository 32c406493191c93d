// Integral images, one pass over HBM: of the public entry point (plain rows of w + 1 floats) and in the quad layout
// of the slab kernels (bc_quad.cuh).
//
// A warp works on 8 rows x 128 columns in registers, a lane on four columns: column sums down the lane's rows, the
// rows' prefixes in the lane, across the warp by shuffles and across the warps of a row through shared memory; the
// results go straight from registers to global memory.  Rows of any length and alignment are read and written
// with vector accesses (bc_tile_io.cuh).
//
// Up to 16 such tiles are a CTA.  With few planes, up to 8 CTAs share one as a cluster, so that every element of it
// is in flight at once; with many, a CTA walks down its plane.  What the tiles above add to a tile's columns comes
// through shared memory and, across CTAs, through distributed shared memory.
#include "bc_cluster.cuh"
#include "scan_shape.cuh"
#include "bc_common.cuh"
#include "bc_quad.cuh"
#include "bc_tile_io.cuh"

namespace bc {

namespace {

constexpr int kScanRows = 8;               // rows a warp works on at a time

__device__ __forceinline__ float4 relu4(float4 v)
{
    return make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
}

__device__ __forceinline__ float4 add4(const float4 &a, const float4 &b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Where a lane's four columns go, row after row.  QUAD: rows in the quad layout, with the constant zeros at their
// left and the copies of the last value behind column w, which some lanes of the first and the last warp write.
template <bool QUAD, int LN = 32>
struct RowSink {
    float *row, *d0, *d1, *d2, *d3, *extra;
    int pitch, w, c, lane, extra_at, from;
    bool in123, in0, zero, first, last_warp, edge_warp;

    // first_row: the row's first float; warp / nwarps: of the row's warps
    __device__ __forceinline__ RowSink(float *first_row, int w_, int warp, int nwarps, int lane_) : row(first_row), w(w_), lane(lane_)
    {
        const int L = warp * LN + lane;
        c = L * 4;
        first = L == 0;
        if (!QUAD) {
            pitch = w + 1;
            return;
        }
        const int cells = quad_cells(w), cell = L + 1;
        pitch = 4 * cells;
        in123 = cell < cells;
        in0 = cell + 1 < cells;
        d1 = row + cells + cell;
        d2 = d1 + cells;
        d3 = d2 + cells;
        d0 = row + cell + 1;
        extra_at = -1;
        if (warp == 0 && lane < 5) extra_at = lane < 4 ? lane * cells : 1;
        zero = extra_at >= 0;
        last_warp = warp == nwarps - 1;
        edge_warp = warp == 0 || last_warp;
        from = ((w - 1) >> 2) & 31;
        if (last_warp && lane >= 8 && lane < 20) {
            const int at = 32 * nwarps + 1 + ((lane - 8) >> 2), sub = lane & 3;
            if (at < cells && (sub || at > 32 * nwarps + 1)) extra_at = sub * cells + at;
        }
        extra = row + extra_at;
    }

    // (a full tile of rows has been put)
    __device__ __forceinline__ void skip(int rows)
    {
        const int64_t by = (int64_t)rows * pitch;
        row += by;
        if (QUAD) { d0 += by; d1 += by; d2 += by; d3 += by; extra += by; }
    }

    // v: prefixes of the lane's own columns; carry: what the row has to their left
    __device__ __forceinline__ void put(const float4 &v, float carry, bool ok = true)
    {
        if (!QUAD) {
            const float o[4] = {v.x + carry, v.y + carry, v.z + carry, v.w + carry};
            store_row4_wide<float, false, LN>(row + 1, c, w, o, lane, ok);
            if (ok && first) *row = 0.0f;
            row += pitch;
            return;
        }
        float x4 = v.w + carry, last = 0.0f;
        const float add = carry;
        if (last_warp) {
            // columns past w: exactly the value at w (a box border out there contributes nothing), which a lane's own
            // scan adds up in another order
            last = __shfl_sync(0xffffffffu, x4, from);
        }
        const bool past = last_warp && c >= w;
        if (past) x4 = last;
        if (in123) {
            *d1 = past ? last : v.x + add;
            *d2 = past ? last : v.y + add;
            *d3 = past ? last : v.z + add;
        }
        if (in0) *d0 = x4;
        if (edge_warp && extra_at >= 0) *extra = zero ? 0.0f : last;
        extra += pitch;
        d0 += pitch; d1 += pitch; d2 += pitch; d3 += pitch;
    }
};

// W warps a row, G warps on top of one another a CTA; `cluster` CTAs share a plane, each with `steps` sets of G warps'
// tiles, which it walks down.
// LN: lanes that a tile's row takes.  Narrow planes (W = 1) take 8 or 16, and a warp works on four or two tiles.
// QUAD: rows in the quad layout; else plain rows of w + 1 floats, the public integral image.
template <typename IO, bool VEC, bool QUAD, int LN, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 4 : 2)
integral_tile_kernel(const IO *__restrict__ in, float *__restrict__ out, int h, int w, int W, int G, int cluster, int steps, bool relu)
{
    constexpr int kGroups = 32 / LN;           // tiles a warp
    extern __shared__ float4 sCol[];           // [G + 1][LN W]: column sums of the warps' rows; last: of all rows above the CTA's
    __shared__ __align__(16) float sTot[kScanWarps][kScanRows];
    grid_dependency_release();
    const int lane = threadIdx.x & (LN - 1), group = (threadIdx.x & 31) / LN, warp = uniform(threadIdx.x >> 5);
    const int g = warp / W, cw = warp - g * W, L = cw * LN + lane, c = L * 4, row_lanes = LN * W;
    const int64_t plane = blockIdx.x / cluster;
    const int rank = blockIdx.x % cluster;
    const int pitch = QUAD ? quad_pitch(w) : w + 1;
    const int stride = G * kGroups * kScanRows;
    int r0 = rank * steps * stride + (g * kGroups + group) * kScanRows;       // first row of this tile
    float *dst = out + plane * (int64_t)(h + 1) * pitch;
    const IO *from = in + plane * (int64_t)h * w + (int64_t)r0 * w;
    float4 *above = sCol + G * row_lanes + L;
    const bool writer = g == 0 && (LN == 32 || group == 0);

    grid_dependency_wait();
    if (rank == 0)
        for (int i = threadIdx.x; i < pitch; i += blockDim.x) dst[i] = 0.0f;      // the zero row on top
    if (writer) *above = make_float4(0.f, 0.f, 0.f, 0.f);
    RowSink<QUAD, LN> sink(dst + (int64_t)(r0 + 1) * pitch, w, cw, W, lane);

    // Column sums of the CTA's rows, one row of sCol per warp, handed to the CTAs below; `above` receives what the CTAs
    // above have.
    auto exchange = [&] {
        __syncthreads();
        float4 up = make_float4(0.f, 0.f, 0.f, 0.f);
        if (writer) {
            float4 s = sCol[L];
            for (int k = 1; k < G; ++k) s = add4(s, sCol[k * row_lanes + L]);
            *above = s;
        }
        cluster_sync();
        if (writer) {
            const uint32_t at = smem_u32(above);
            for (int k = 0; k < rank; ++k) up = add4(up, cluster_load4(cluster_map(at, k)));
        }
        cluster_sync();      // everybody has read: the slots may be used again, and CTAs may leave
        if (writer) *above = up;
        __syncthreads();
    };
    // what the groups above this one in the warp have (v: the group's own sums); returns the warp's sums in `total`
    auto over_groups = [&](const float4 &v, float4 &total) {
        float4 incl = v;
        if (kGroups > 1) {
#pragma unroll
            for (int d = LN; d < 32; d <<= 1) {
                float4 u;
                u.x = __shfl_up_sync(0xffffffffu, incl.x, d); u.y = __shfl_up_sync(0xffffffffu, incl.y, d);
                u.z = __shfl_up_sync(0xffffffffu, incl.z, d); u.w = __shfl_up_sync(0xffffffffu, incl.w, d);
                if (group * LN >= d) incl = add4(incl, u);
            }
        }
        total = incl;
        float4 excl = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kGroups > 1) {
            excl.x = __shfl_up_sync(0xffffffffu, incl.x, LN & 31); excl.y = __shfl_up_sync(0xffffffffu, incl.y, LN & 31);
            excl.z = __shfl_up_sync(0xffffffffu, incl.z, LN & 31); excl.w = __shfl_up_sync(0xffffffffu, incl.w, LN & 31);
            if (group == 0) excl = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        return excl;
    };

    if (cluster > 1 && steps > 1) {      // first all sums, then the walk: the rows are read a second time, from L2
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        const IO *at = from;
        for (int k = 0, r = r0; k < steps; ++k, r += stride, at += (int64_t)stride * w) {
            Rows8 t;
            rows8_load<IO, VEC, false, LN>(t, at, w, c, h - r, lane);
            float4 pair[kScanRows / 2];      // (added up in a tree: one rounding in three of a row after the other's)
#pragma unroll
            for (int i = 0; i < kScanRows; i += 2) {
                float4 u = rows8_get<IO, VEC, LN>(t, at, w, c, lane, i), v = rows8_get<IO, VEC, LN>(t, at, w, c, lane, i + 1);
                if (relu) u = relu4(u), v = relu4(v);
                pair[i / 2] = add4(u, v);
            }
            sum = add4(sum, add4(add4(pair[0], pair[1]), add4(pair[2], pair[3])));
        }
        float4 total;
        over_groups(sum, total);
        if (kGroups == 1 || group == kGroups - 1) sCol[g * row_lanes + L] = total;
        exchange();
    }
    for (int step = 0; step < steps; ++step) {
        const int rows = h - r0;               // rows of this tile: at most 8 (may be none)
        float4 v[kScanRows];
        {
            Rows8 t;
            rows8_load<IO, VEC, false, LN>(t, from, w, c, rows, lane);
#pragma unroll
            for (int i = 0; i < kScanRows; ++i) {
                v[i] = rows8_get<IO, VEC, LN>(t, from, w, c, lane, i);
                if (relu) v[i] = relu4(v[i]);
            }
        }
#pragma unroll
        for (int i = 1; i < kScanRows; ++i) v[i] = add4(v[i], v[i - 1]);
        float4 total, up = over_groups(v[kScanRows - 1], total);
        if (kGroups == 1 || group == kGroups - 1) sCol[g * row_lanes + L] = total;
        if (cluster > 1 && steps == 1) exchange();
        else __syncthreads();
        if (kGroups == 1) up = *above;
        else up = add4(up, *above);
        for (int k = 0; k < g; ++k) up = add4(up, sCol[k * row_lanes + L]);
        const float4 next = add4(v[kScanRows - 1], up);      // what the plane has above the CTA's next tiles (the last tile knows)
        float carry[kScanRows];
#pragma unroll
        for (int i = 0; i < kScanRows; ++i) {
            v[i].x += up.x;
            v[i].y += up.y + v[i].x;
            v[i].z += up.z + v[i].y;
            v[i].w += up.w + v[i].z;
            const float incl = warp_prefix<LN>(v[i].w, carry[i]);
            if (LN == 32 && W > 1 && lane == 31) sTot[warp][i] = incl;
        }
        __syncthreads();
        if (g == G - 1 && (kGroups == 1 || group == kGroups - 1)) *above = next;
        if (LN == 32) {
            for (int k = warp - cw; k < warp; ++k) {
#pragma unroll
                for (int i = 0; i < kScanRows; i += 4) {
                    const float4 a = *reinterpret_cast<const float4 *>(&sTot[k][i]);
                    carry[i] += a.x; carry[i + 1] += a.y; carry[i + 2] += a.z; carry[i + 3] += a.w;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kScanRows; ++i) {
            if (kGroups > 1) sink.put(v[i], carry[i], i < rows);
            else if (i < rows) sink.put(v[i], carry[i]);
        }
        sink.skip(stride - kScanRows);
        r0 += stride;
        from += (int64_t)stride * w;
    }
}

// A row's prefixes, columns last: the lane's four, then the warp's lanes, then the warps to the left one after the
// other.  Leaves the lane's prefixes in v and returns what the row has to the left of them within the warp; `total`:
// the warp's sum (lane 31).
__device__ __forceinline__ float row_prefix(float4 &v, float &total)
{
    v.y += v.x; v.z += v.y; v.w += v.z;
    total = warp_scan(v.w);
    return total - v.w;
}

// The same, in a fixed order of additions: along the rows first, then down the columns one row after the other from
// the top of the plane, or of the plane's band when there are `bands` of `band_tiles` tiles each (what the bands
// above add up to is added last).  This is the order in which integral_image_kernel adds up planes whose rows a vector
// access fits, and in which integral images of grad_output have been added up since before this kernel; it includes
// that kernel's way of taking a lane's own sum off the warp's.  Parameter gradients of large planes hang on its
// rounding (differences of sums of 1e5 values: relative errors of 1e-5), so a change of order shows in the fifth digit of
// results that users compare between versions.  Not every plane has it: rows of other lengths, tensors that begin
// off a vector's alignment and some tall planes go to the other kernel (integral_ordered_t), which rounds otherwise, so
// that the same values at another address can give gradients that differ in that digit.
// What is serial are only the additions: tile after tile through shared memory, about 130 cycles each, CTA after
// CTA through distributed shared memory.
// T: 8-row tiles a thread holds (2 where one would need more than 8 CTAs a plane).
template <typename IO, int T>
__global__ void __launch_bounds__(32 * kScanWarps, T == 1 ? 2 : 1)
integral_ordered_kernel(const IO *__restrict__ in, float *__restrict__ out, int h, int w, int W, int G, int cluster, int bands,
                        int band_tiles)
{
    extern __shared__ float4 sLast[];          // [tiles of the CTA][32 W]: the tiles' last rows
    __shared__ __align__(16) float sTot[kScanWarps][T * kScanRows];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5);
    const int g = warp / W, cw = warp - g * W, L = cw * 32 + lane, c = L * 4, row_lanes = 32 * W;
    const int64_t plane = blockIdx.x / cluster;
    const int rank = blockIdx.x % cluster;
    const int pitch = quad_pitch(w);
    int tile0 = (rank * G + g) * T;
    const int stride = G * T * kScanRows;
    float *dst = out + plane * (int64_t)(h + 1) * pitch;
    const IO *from = in + plane * (int64_t)h * w + (int64_t)tile0 * kScanRows * w;

    grid_dependency_wait();
    if (rank == 0)
        for (int i = threadIdx.x; i < pitch; i += blockDim.x) dst[i] = 0.0f;      // the zero row on top
    RowSink<true> sink(dst + (int64_t)(tile0 * kScanRows + 1) * pitch, w, cw, W, lane);
    for (int left = cluster > 1 ? 1 : h; left > 0; left -= stride) {
        const int rows = h - tile0 * kScanRows;
        float4 v[T][kScanRows];
        {
            Rows8 t[T];
#pragma unroll
            for (int k = 0; k < T; ++k) rows8_load<IO, true>(t[k], from + (int64_t)k * kScanRows * w, w, c, rows - k * kScanRows, lane);
#pragma unroll
            for (int k = 0; k < T; ++k)
#pragma unroll
                for (int i = 0; i < kScanRows; ++i) v[k][i] = t[k].a[i];
        }
        float before[T][kScanRows];
#pragma unroll
        for (int k = 0; k < T; ++k)
#pragma unroll
            for (int i = 0; i < kScanRows; ++i) {
                float total;
                before[k][i] = row_prefix(v[k][i], total);
                if (W > 1 && lane == 31) sTot[warp][k * kScanRows + i] = total;
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < T; ++k) {
            float running[kScanRows] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int j = warp - cw; j < warp; ++j) {
#pragma unroll
                for (int i = 0; i < kScanRows; i += 4) {
                    const float4 a = *reinterpret_cast<const float4 *>(&sTot[j][k * kScanRows + i]);
                    running[i] += a.x; running[i + 1] += a.y; running[i + 2] += a.z; running[i + 3] += a.w;
                }
            }
#pragma unroll
            for (int i = 0; i < kScanRows; ++i) {
                const float add = running[i] + before[k][i];
                v[k][i].x += add; v[k][i].y += add; v[k][i].z += add; v[k][i].w += add;
            }
        }
        // down the columns
        // (bands that begin and end with CTAs need not wait for one another)
        const int turns = band_tiles > 0 && (G * T) % band_tiles == 0 ? 1 : cluster;
        for (int turn = 0; turn < turns; ++turn) {
            if (turns == 1 || turn == rank) {
                for (int step = 0; step < G; ++step) {
                    if (step == g) {
                        float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (tile0 % band_tiles) {
                            if (g) run = sLast[(g * T - 1) * row_lanes + L];
                            else if (cluster > 1) run = cluster_load4(cluster_map(smem_u32(sLast + (G * T - 1) * row_lanes + L), rank - 1));
                            else run = sLast[(G * T - 1) * row_lanes + L];
                        }
#pragma unroll
                        for (int k = 0; k < T; ++k) {
                            if (k && (tile0 + k) % band_tiles == 0) run = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int i = 0; i < kScanRows; ++i) {
                                run.x += v[k][i].x; run.y += v[k][i].y; run.z += v[k][i].z; run.w += v[k][i].w;
                                v[k][i] = run;
                            }
                            sLast[(g * T + k) * row_lanes + L] = run;
                        }
                    }
                    __syncthreads();
                }
            }
            if (cluster > 1) cluster_sync();
        }
        // what the bands above add up to (bands come with clusters only)
        if (bands > 1) {
            const int per_cta = G * T;
#pragma unroll
            for (int k = 0; k < T; ++k) {
                float4 above = make_float4(0.f, 0.f, 0.f, 0.f);
                const int band = (tile0 + k) / band_tiles;
                for (int b = 1; b <= band; ++b) {
                    const int last = b * band_tiles - 1, owner = last / per_cta;
                    const float4 *at = sLast + (last - owner * per_cta) * row_lanes + L;
                    const float4 u = owner == rank ? *at : cluster_load4(cluster_map(smem_u32(at), owner));
                    above.x += u.x; above.y += u.y; above.z += u.z; above.w += u.w;
                }
                if (band > 0) {
#pragma unroll
                    for (int i = 0; i < kScanRows; ++i) { v[k][i].x += above.x; v[k][i].y += above.y; v[k][i].z += above.z; v[k][i].w += above.w; }
                }
            }
            if (cluster > 1) cluster_sync();      // no CTA leaves while another still reads its last rows
        }
#pragma unroll
        for (int k = 0; k < T; ++k)
#pragma unroll
            for (int i = 0; i < kScanRows; ++i)
                if (k * kScanRows + i < rows) sink.put(v[k][i], 0.0f);
        sink.skip(stride - T * kScanRows);
        tile0 += G * T;
        from += (int64_t)stride * w;
    }
}

template <typename IO, bool QUAD, int LN>
int integral_tile_t(const IO *in, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    const int warps = LN < 32 ? 1 : (w + 127) / 128, warp_rows = kScanRows * (32 / LN);
    const bool vec = w % 4 == 0 && aligned_to(in, Io<IO>::kVecBytes);
    // two CTAs of 16 warps an SM: up to one and a half rounds of them ((256,280,560): 80 us, 149 with 8 warps; (404,60,341):
    // 21, 33; (424,568,105): 67, 77); not in the quad layout (368 planes of 110 x 450: 6 us more)
    const int tiles = (h + warp_rows - 1) / warp_rows;
    const ScanShape sh = scan_clusters_that_fit(scan_shape(planes, tiles, warps, QUAD ? 148 : 3 * 148), planes, tiles, warps, QUAD);
    if (planes * sh.ctas > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    void (*kern)(const IO *, float *, int, int, int, int, int, int, bool);
    if (sh.G * warps <= 8) kern = vec ? integral_tile_kernel<IO, true, QUAD, LN, 256> : integral_tile_kernel<IO, false, QUAD, LN, 256>;
    else kern = vec ? integral_tile_kernel<IO, true, QUAD, LN, 512> : integral_tile_kernel<IO, false, QUAD, LN, 512>;
    {
        LaunchScope scope(KID_INTEGRAL, s);
        if (cudaError_t e = launch_overlapped_cluster(kern, (unsigned)(planes * sh.ctas), sh.G * warps * 32,
                                                      (sh.G + 1) * warps * LN * sizeof(float4), sh.ctas, s, in, out, h, w, warps, sh.G,
                                                      sh.ctas, sh.steps, relu))
            return cuda_failed(e, "integral_tile");
    }
    return check_launch("integral_tile");
}

template <typename IO, bool QUAD>
int integral_scan_t(const IO *in, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    if constexpr (!QUAD) {      // (the slab path, which reads the quad layout, has no planes this narrow worth a kernel)
        if (w <= 32) return integral_tile_t<IO, QUAD, 8>(in, out, planes, h, w, relu, s);
        if (w <= 64) return integral_tile_t<IO, QUAD, 16>(in, out, planes, h, w, relu, s);
    }
    return integral_tile_t<IO, QUAD, 32>(in, out, planes, h, w, relu, s);
}

// Quad layout, additions in the order that integral_ordered_kernel describes.  Planes whose rows are no multiple of
// four floats, and a few of more rows than a cluster holds, are added up in the other kernel's order.
template <typename IO>
int integral_ordered_t(const IO *in, float *out, int64_t planes, int h, int w, cudaStream_t s)
{
    const bool vec = w % 4 == 0 && aligned_to(in, Io<IO>::kVecBytes);
    if (!vec || planes > 0x7fffffffLL / 8) return integral_scan_t<IO, true>(in, out, planes, h, w, false, s);
    const int warps = (w + 127) / 128, tiles = (h + kScanRows - 1) / kScanRows;
    int band_rows = h, bands = 1;
    if (planes <= 64 && h >= 64) {
        const int want = (int)((2 * 148 + planes - 1) / planes);
        int rows = (h + want - 1) / want;
        rows = ((rows < 16 ? 16 : rows) + 7) & ~7;
        if (rows < h) {
            band_rows = rows;
            bands = (h + rows - 1) / rows;
        }
    }
    const int band_tiles = (band_rows + kScanRows - 1) / kScanRows;
    int T = 1;
    ScanShape sh = scan_shape(planes, tiles, warps);
    if (sh.ctas > 1 && sh.steps > 1) {      // too many rows for a cluster: twice the rows a thread, or a walk
        sh = scan_shape(planes, (tiles + 1) / 2, warps);
        T = 2;
        if (sh.steps > 1 && bands > 1) return integral_scan_t<IO, true>(in, out, planes, h, w, false, s);
        if (sh.steps > 1) {
            sh = scan_shape(148, tiles, warps);
            T = 1;
        }
    }
    void (*kern)(const IO *, float *, int, int, int, int, int, int, int) = T == 1 ? integral_ordered_kernel<IO, 1> : integral_ordered_kernel<IO, 2>;
    {
        LaunchScope scope(KID_INTEGRAL, s);
        if (cudaError_t e = launch_overlapped_cluster(kern, (unsigned)(planes * sh.ctas), sh.G * warps * 32,
                                                      sh.G * T * warps * 32 * sizeof(float4), sh.ctas, s, in, out, h, w, warps, sh.G,
                                                      sh.ctas, bands, band_tiles))
            return cuda_failed(e, "integral_ordered");
    }
    return check_launch("integral_ordered");
}

}  // namespace

int launch_integral_quad(const void *in, int io_kind, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    if (planes == 0) return BC_OK;
    if (io_kind == BC_IO_F16) return integral_scan_t<__half, true>(static_cast<const __half *>(in), out, planes, h, w, relu, s);
    if (io_kind == BC_IO_BF16) return integral_scan_t<__nv_bfloat16, true>(static_cast<const __nv_bfloat16 *>(in), out, planes, h, w, relu, s);
    return integral_scan_t<float, true>(static_cast<const float *>(in), out, planes, h, w, relu, s);
}

int launch_integral_quad_ordered(const void *in, int io_kind, float *out, int64_t planes, int h, int w, cudaStream_t s)
{
    if (planes == 0) return BC_OK;
    if (io_kind == BC_IO_F16) return integral_ordered_t(static_cast<const __half *>(in), out, planes, h, w, s);
    if (io_kind == BC_IO_BF16) return integral_ordered_t(static_cast<const __nv_bfloat16 *>(in), out, planes, h, w, s);
    return integral_ordered_t(static_cast<const float *>(in), out, planes, h, w, s);
}

static int scan_steps(int64_t planes, int h, int w, int lanes)
{
    const int rows = kScanRows * (32 / lanes);
    return scan_shape(planes, (h + rows - 1) / rows, lanes < 32 ? 1 : (w + 127) / 128).steps;      // (of up to 147 planes)
}

// A plane or two, down which a cluster would walk many steps while the rest of the GPU has nothing to do: the kernels of
// integral_image.cu cut them into bands that all SMs share (forward of (1,1,1,4000,900): 68 us against 125,
// (1,1,4,2048,2048): 121 against 164, (1,2,2,20000,1): 62 against 129; of (1,2,2,2000,600), eleven steps: 50 against 52).
bool integral_scan_starves(int64_t planes, int h, int w)
{
    return w <= 128 * kScanWarps && planes <= 2 && scan_steps(planes, h, w, 32) > 12;
}

// Plain rows.  The older kernel is faster on few planes of many steps as long as what its bands read again is in L2
// ((1,2048,2048): 51 us against 128, (15,583,1121): 69 against 79; (11,2190,879): 328 against 166), and on nearly as many planes as
// there are SMs, which clusters read twice, if their rows fit vector accesses ((128,280,560): 60 us against 69,
// (108,260,860): 72 against 81; with other row lengths it is two to four times slower).
bool integral_scan_suits(const float *in, int64_t planes, int h, int w)
{
    if (w > 128 * kScanWarps) return false;
    const int steps = scan_steps(planes, h, w, w <= 32 ? 8 : w <= 64 ? 16 : 32);
    if (planes <= 64 && steps > 8 && planes * h * w * 8 <= 96 << 20) return false;
    return !(w % 4 == 0 && aligned_to(in, 16) && planes >= 100 && planes < 148 && steps > 1);
}

int launch_integral_scan(const float *in, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    return integral_scan_t<float, false>(in, out, planes, h, w, relu, s);
}

}  // namespace bc
