// Integral images, one pass over HBM: of the public entry point (plain rows of w + 1 floats) and in the quad layout
// of the slab kernels (bc_quad.cuh).
//
// A warp works on 8 rows x 128 columns in registers, a lane on four columns: column sums down the lane's rows, the
// rows' prefixes in the lane, across the warp by shuffles and across the warps of a row through shared memory; the
// results go straight from registers to global memory.  Rows of any length and alignment are read and written
// with vector accesses (bc_tile_io.cuh).
//
// integral_tile_kernel: up to 16 such tiles a CTA and up to 8 CTAs a plane, one cluster, so that every element of
//   a plane is in flight at once; what the tiles above add to a tile's columns comes through shared memory and,
//   across CTAs, through distributed shared memory.
// integral_scan_kernel: planes too large for that.  A CTA walks down its plane, or with few planes its part of it,
//   eight rows at a time, the next eight being loaded meanwhile.
#include "bc_common.cuh"
#include "bc_quad.cuh"
#include "bc_tile_io.cuh"

namespace bc {

namespace {

constexpr int kScanWarps = 16;             // warps a CTA
constexpr int kScanRows = 8;               // rows a warp works on at a time

__device__ __forceinline__ float4 relu4(float4 v)
{
    return make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
}

__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float4 cluster_load4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Where a lane's four columns go, row after row.  QUAD: rows in the quad layout, with the constant zeros at their
// left and the copies of the last value behind column w, which some lanes of the first and the last warp write.
template <bool QUAD>
struct RowSink {
    float *row, *d0, *d1, *d2, *d3, *extra;
    int pitch, w, c, lane, extra_at, from;
    bool in123, in0, zero, first, last_warp, edge_warp;

    // first_row: the row's first float; warp / nwarps: of the row's warps
    __device__ __forceinline__ RowSink(float *first_row, int w_, int warp, int nwarps, int lane_) : row(first_row), w(w_), lane(lane_)
    {
        const int L = warp * 32 + lane;
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

    // v: prefixes of the lane's own columns (zero past the plane); carry: what the row has to their left
    __device__ __forceinline__ void put(const float4 &v, float carry)
    {
        if (!QUAD) {
            const float o[4] = {v.x + carry, v.y + carry, v.z + carry, v.w + carry};
            store_row4<float, false>(row + 1, c, w, o, lane);
            if (first) *row = 0.0f;
            row += pitch;
            return;
        }
        float x4 = v.w + carry, add = carry, last = 0.0f;
        if (last_warp) {
            // columns past w: exactly the value at w (a box border out there contributes nothing), which a lane's own
            // scan adds up in another order
            last = __shfl_sync(0xffffffffu, x4, from);
            if (c >= w) x4 = add = last;
        }
        if (in123) {
            *d1 = v.x + add;
            *d2 = v.y + add;
            *d3 = v.z + add;
        }
        if (in0) *d0 = x4;
        if (edge_warp) {
            if (extra_at >= 0) *extra = zero ? 0.0f : last;
            extra += pitch;
        }
        d0 += pitch; d1 += pitch; d2 += pitch; d3 += pitch;
    }
};

// W warps a row, G tiles on top of one another a CTA, `cluster` CTAs a plane.
template <typename IO, bool VEC, bool QUAD, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 256 ? 4 : 2)
integral_tile_kernel(const IO *__restrict__ in, float *__restrict__ out, int h, int w, int W, int G, int cluster, bool relu)
{
    extern __shared__ float4 sCol[];           // [G + 1][32 W]: column sums of the tiles; last: of the whole CTA, later of the CTAs above
    __shared__ __align__(16) float sTot[kScanWarps][kScanRows];
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5);
    const int g = warp / W, cw = warp - g * W, L = cw * 32 + lane, c = L * 4, row_lanes = 32 * W;
    const int64_t plane = blockIdx.x / cluster;
    const int rank = blockIdx.x % cluster;
    const int pitch = QUAD ? quad_pitch(w) : w + 1;
    const int r0 = (rank * G + g) * kScanRows, rows = h - r0;      // rows of this tile: at most 8 (may be none)
    float *dst = out + plane * (int64_t)(h + 1) * pitch;
    const IO *from = in + plane * (int64_t)h * w + (int64_t)r0 * w;

    grid_dependency_wait();
    float4 v[kScanRows];
    {
        Rows8 t;
        rows8_load<IO, VEC>(t, from, w, c, rows, lane);
        if (rank == 0)
            for (int i = threadIdx.x; i < pitch; i += blockDim.x) dst[i] = 0.0f;      // the zero row on top
#pragma unroll
        for (int i = 0; i < kScanRows; ++i) {
            v[i] = rows8_get<IO, VEC>(t, from, w, c, lane, i);
            if (relu) v[i] = relu4(v[i]);
        }
    }
#pragma unroll
    for (int i = 1; i < kScanRows; ++i) { v[i].x += v[i - 1].x; v[i].y += v[i - 1].y; v[i].z += v[i - 1].z; v[i].w += v[i - 1].w; }
    sCol[g * row_lanes + L] = v[kScanRows - 1];
    __syncthreads();
    float4 up = make_float4(0.f, 0.f, 0.f, 0.f);
    if (cluster > 1) {
        float4 *own = sCol + G * row_lanes + L;
        if (g == 0) {
            float4 s = sCol[L];
            for (int k = 1; k < G; ++k) {
                const float4 u = sCol[k * row_lanes + L];
                s.x += u.x; s.y += u.y; s.z += u.z; s.w += u.w;
            }
            *own = s;
        }
        cluster_sync();
        if (g == 0) {
            const uint32_t at = smem_u32(own);
            for (int k = 0; k < rank; ++k) {
                const float4 u = cluster_load4(cluster_map(at, k));
                up.x += u.x; up.y += u.y; up.z += u.z; up.w += u.w;
            }
        }
        cluster_sync();      // everybody has read: the slots may be used again, and CTAs may leave
        if (g == 0) *own = up;
        __syncthreads();
        up = *own;
    }
    for (int k = 0; k < g; ++k) {
        const float4 u = sCol[k * row_lanes + L];
        up.x += u.x; up.y += u.y; up.z += u.z; up.w += u.w;
    }
    float carry[kScanRows];
#pragma unroll
    for (int i = 0; i < kScanRows; ++i) {
        v[i].x += up.x;
        v[i].y += up.y + v[i].x;
        v[i].z += up.z + v[i].y;
        v[i].w += up.w + v[i].z;
        const float incl = warp_scan(v[i].w);
        carry[i] = incl - v[i].w;
        if (W > 1 && lane == 31) sTot[warp][i] = incl;
    }
    if (W > 1) {
        __syncthreads();
        for (int k = warp - cw; k < warp; ++k) {
#pragma unroll
            for (int i = 0; i < kScanRows; i += 4) {
                const float4 a = *reinterpret_cast<const float4 *>(&sTot[k][i]);
                carry[i] += a.x; carry[i + 1] += a.y; carry[i + 2] += a.z; carry[i + 3] += a.w;
            }
        }
    }
    RowSink<QUAD> sink(dst + (int64_t)(r0 + 1) * pitch, w, cw, W, lane);
#pragma unroll
    for (int i = 0; i < kScanRows; ++i)
        if (i < rows) sink.put(v[i], carry[i]);
}

// QUAD: rows in the quad layout; else plain rows of w + 1 floats, the public integral image.
template <typename IO, bool VEC, bool RELU, bool QUAD, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT <= 128 ? (VEC ? 5 : 4) : 1)
integral_scan_kernel(const IO *__restrict__ in, float *__restrict__ out, int h, int w, int rows_per_cta, int cluster)
{
    __shared__ __align__(16) float sTot[2][kScanWarps][kScanRows];
    extern __shared__ float4 sCol[];           // column sums of this CTA's rows (clusters only)
    grid_dependency_release();
    const int lane = threadIdx.x & 31, warp = uniform(threadIdx.x >> 5), nwarps = blockDim.x >> 5;
    const int64_t plane = blockIdx.x / cluster;
    const int rank = blockIdx.x % cluster;
    const int L = threadIdx.x, c = L * 4;
    const int cells = quad_cells(w), pitch = QUAD ? 4 * cells : w + 1;
    const int r0 = min(rank * rows_per_cta, h), r1 = min(r0 + rows_per_cta, h);
    const IO *src = in + plane * (int64_t)h * w;
    float *dst = out + plane * (int64_t)(h + 1) * pitch;

    grid_dependency_wait();
    Rows8 nxt;
    const IO *from = src + (int64_t)r0 * w;
    rows8_load<IO, VEC>(nxt, from, w, c, r1 - r0, lane);

    float run[4] = {0.f, 0.f, 0.f, 0.f};
    if (cluster > 1) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        Rows8 g = nxt;
        const IO *at = from;
        for (int r = r0; r < r1; r += kScanRows) {
            Rows8 ahead;
            rows8_load<IO, VEC>(ahead, at + (int64_t)kScanRows * w, w, c, r1 - r - kScanRows, lane);
#pragma unroll
            for (int i = 0; i < kScanRows; ++i) {
                float4 v = rows8_get<IO, VEC>(g, at, w, c, lane, i);
                if (RELU) v = relu4(v);
                sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            }
            g = ahead;
            at += (int64_t)kScanRows * w;
        }
        sCol[L] = sum;
        cluster_sync();
        const uint32_t own = smem_u32(sCol) + L * 16;
        for (int k = 0; k < rank; ++k) {
            const float4 u = cluster_load4(cluster_map(own, k));
            run[0] += u.x; run[1] += u.y; run[2] += u.z; run[3] += u.w;
        }
        cluster_sync();      // no CTA leaves while another still reads its sums
    }

    if (rank == 0)
        for (int i = threadIdx.x; i < pitch; i += blockDim.x) dst[i] = 0.0f;      // the zero row on top
    RowSink<QUAD> sink(dst + (int64_t)(r0 + 1) * pitch, w, warp, nwarps, lane);
    int buf = 0;
    for (int r = r0; r < r1; r += kScanRows) {
        float4 v[kScanRows];
        float carry[kScanRows];
#pragma unroll
        for (int i = 0; i < kScanRows; ++i) {
            v[i] = rows8_get<IO, VEC>(nxt, from, w, c, lane, i);
            if (RELU) v[i] = relu4(v[i]);
        }
        from += (int64_t)kScanRows * w;
        rows8_load<IO, VEC>(nxt, from, w, c, r1 - r - kScanRows, lane);
#pragma unroll
        for (int i = 0; i < kScanRows; ++i) {
            run[0] += v[i].x; run[1] += v[i].y; run[2] += v[i].z; run[3] += v[i].w;
            v[i].x = run[0];
            v[i].y = run[1] + v[i].x;
            v[i].z = run[2] + v[i].y;
            v[i].w = run[3] + v[i].z;
            const float incl = warp_scan(v[i].w);
            carry[i] = incl - v[i].w;
            if (lane == 31) sTot[buf][warp][i] = incl;
        }
        if (nwarps > 1) {
            __syncthreads();
            for (int k = 0; k < warp; ++k) {
#pragma unroll
                for (int i = 0; i < kScanRows; i += 4) {
                    const float4 a = *reinterpret_cast<const float4 *>(&sTot[buf][k][i]);
                    carry[i] += a.x; carry[i + 1] += a.y; carry[i + 2] += a.z; carry[i + 3] += a.w;
                }
            }
            buf ^= 1;
        }
#pragma unroll
        for (int i = 0; i < kScanRows; ++i)
            if (r + i < r1) sink.put(v[i], carry[i]);
    }
}

template <typename IO, bool QUAD>
int integral_scan_t(const IO *in, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    const int warps = (w + 127) / 128;
    const bool vec = w % 4 == 0 && aligned_to(in, Io<IO>::kVecBytes);
    const int tiles = (h + kScanRows - 1) / kScanRows, most = kScanWarps / warps;
    const int ctas = (tiles + most - 1) / most;
    // The tile kernel where a cluster holds the plane; but many planes that take several CTAs each are faster walked
    // down ((512,256,512): 111 us against 156; (2500,136,80): 73 against 88), as long as rows are aligned.
    if (ctas <= 8 && !(ctas > 1 && vec && planes >= 2 * 148)) {
        const int G = (tiles + ctas - 1) / ctas;
        if (planes * ctas > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
        void (*kern)(const IO *, float *, int, int, int, int, int, bool);
        if (G * warps <= 8) kern = vec ? integral_tile_kernel<IO, true, QUAD, 256> : integral_tile_kernel<IO, false, QUAD, 256>;
        else kern = vec ? integral_tile_kernel<IO, true, QUAD, 512> : integral_tile_kernel<IO, false, QUAD, 512>;
        {
            LaunchScope scope(KID_INTEGRAL, s);
            if (cudaError_t e = launch_overlapped_cluster(kern, (unsigned)(planes * ctas), G * warps * 32,
                                                          (G + 1) * warps * 32 * sizeof(float4), ctas, s, in, out, h, w, warps, G, ctas,
                                                          relu))
                return cuda_failed(e, "integral_tile");
        }
        return check_launch("integral_tile");
    }
    // few planes: clusters of up to 8 CTAs share one, as long as each keeps 16 rows
    int cluster = 1;
    while (cluster < 8 && planes * cluster < 2 * 148 && h >= 32 * cluster) cluster *= 2;
    const int rows = ((h + cluster - 1) / cluster + kScanRows - 1) / kScanRows * kScanRows;
    if (planes * cluster > 0x7fffffffLL) return BC_ERR_BAD_SHAPE;
    void (*kern)(const IO *, float *, int, int, int, int);
    constexpr int S = 128, L = 32 * kScanWarps;
    if (warps * 32 <= S) {
        if (relu) kern = vec ? integral_scan_kernel<IO, true, true, QUAD, S> : integral_scan_kernel<IO, false, true, QUAD, S>;
        else kern = vec ? integral_scan_kernel<IO, true, false, QUAD, S> : integral_scan_kernel<IO, false, false, QUAD, S>;
    } else {
        if (relu) kern = vec ? integral_scan_kernel<IO, true, true, QUAD, L> : integral_scan_kernel<IO, false, true, QUAD, L>;
        else kern = vec ? integral_scan_kernel<IO, true, false, QUAD, L> : integral_scan_kernel<IO, false, false, QUAD, L>;
    }
    {
        LaunchScope scope(KID_INTEGRAL, s);
        if (cudaError_t e = launch_overlapped_cluster(kern, (unsigned)(planes * cluster), warps * 32,
                                                      cluster > 1 ? warps * 32 * sizeof(float4) : 0, cluster, s, in, out, h, w, rows,
                                                      cluster))
            return cuda_failed(e, "integral_scan");
    }
    return check_launch("integral_scan");
}

}  // namespace

int launch_integral_quad(const void *in, int io_kind, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    if (planes == 0) return BC_OK;
    if (io_kind == BC_IO_F16) return integral_scan_t<__half, true>(static_cast<const __half *>(in), out, planes, h, w, relu, s);
    if (io_kind == BC_IO_BF16) return integral_scan_t<__nv_bfloat16, true>(static_cast<const __nv_bfloat16 *>(in), out, planes, h, w, relu, s);
    return integral_scan_t<float, true>(static_cast<const float *>(in), out, planes, h, w, relu, s);
}

int launch_integral_scan(const float *in, float *out, int64_t planes, int h, int w, bool relu, cudaStream_t s)
{
    return integral_scan_t<float, false>(in, out, planes, h, w, relu, s);
}

}  // namespace bc
