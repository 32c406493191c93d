// Device helpers of the kernels that stage tiles in shared memory: bulk asynchronous copies with bounded
// waits, and loads / stores of the big tensors in their storage type.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "bc_common.cuh"
#include "bc_smem_walk.cuh"

namespace bc {

namespace {

// ---- asynchronous bulk copies (TMA, no tensor map) global -> shared, completion on an mbarrier.
// Every wait is bounded: when the limit expires the kernel counts the event in g_wait_timeouts
// and carries on, so a lost copy shows up as a reported error instead of a hung GPU.
static __device__ int g_wait_timeouts = 0;      // one counter per translation unit that includes this file
constexpr long long kWaitLimitCycles = 2000000000LL;      // about a second

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t mbar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}
// Hint that `bytes` (a multiple of 16) at `src` (16-byte aligned) will be copied soon: brings them into L2.
__device__ __forceinline__ void bulk_prefetch_l2(const void *src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// The same hint for memory of any alignment, spread over the CTA's threads.
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes)
{
    const char *c = static_cast<const char *>(p);
    for (size_t at = (size_t)threadIdx.x * 128; at < bytes; at += (size_t)blockDim.x * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(c + at));
}
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity)
{
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
                     " selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(mbar), "r"(parity), "r"(2000u) : "memory");
        if (done) return true;
        if (clock64() - t0 > kWaitLimitCycles) return false;
    }
}

// ---- storage types of the big tensors --------------------------------------------------------
// The kernels are instantiated for float, __half and __nv_bfloat16 input / grad_output / output /
// grad_input tensors.  Narrow types are converted as they are loaded and rounded to nearest as they
// are stored; the integral images, every accumulator and the parameter gradients stay float.
// load4 / store4 move the 4 values of one strip row with one instruction (16 or 8 bytes).
template <typename IO>
struct Io;

template <>
struct Io<float> {
    static constexpr int kKind = BC_IO_F32;
    static constexpr int kVecBytes = 16;
    static __device__ __forceinline__ float4 load4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
    static __device__ __forceinline__ float load1(const float *p) { return __ldg(p); }
    // for memory that this kernel may also write
    static __device__ __forceinline__ float4 load4_plain(const float *p) { return *reinterpret_cast<const float4 *>(p); }
    static __device__ __forceinline__ void store4(float *p, float a, float b, float c, float d)
    {
        *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
    }
    static __device__ __forceinline__ void store2(float *p, float a, float b) { *reinterpret_cast<float2 *>(p) = make_float2(a, b); }
    static __device__ __forceinline__ void store1(float *p, float v) { *p = v; }
    static __device__ __forceinline__ float4 lds4(uint32_t a) { return lds128(a); }
};

__device__ __forceinline__ uint2 lds64(uint32_t a)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}

template <>
struct Io<__half> {
    static constexpr int kKind = BC_IO_F16;
    static constexpr int kVecBytes = 8;
    static __device__ __forceinline__ float4 widen(uint2 r)
    {
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&r.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&r.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ float4 load4(const __half *p) { return widen(__ldg(reinterpret_cast<const uint2 *>(p))); }
    static __device__ __forceinline__ float load1(const __half *p) { return __half2float(__ldg(p)); }
    static __device__ __forceinline__ void store4(__half *p, float a, float b, float c, float d)
    {
        const __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
        uint2 r;
        r.x = *reinterpret_cast<const uint32_t *>(&lo);
        r.y = *reinterpret_cast<const uint32_t *>(&hi);
        *reinterpret_cast<uint2 *>(p) = r;
    }
    static __device__ __forceinline__ void store2(__half *p, float a, float b) { *reinterpret_cast<__half2 *>(p) = __floats2half2_rn(a, b); }
    static __device__ __forceinline__ void store1(__half *p, float v) { *p = __float2half_rn(v); }
    static __device__ __forceinline__ float4 lds4(uint32_t a) { return widen(lds64(a)); }
};

template <>
struct Io<__nv_bfloat16> {
    static constexpr int kKind = BC_IO_BF16;
    static constexpr int kVecBytes = 8;
    static __device__ __forceinline__ float4 widen(uint2 r)
    {
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&r.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&r.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ float4 load4(const __nv_bfloat16 *p) { return widen(__ldg(reinterpret_cast<const uint2 *>(p))); }
    static __device__ __forceinline__ float load1(const __nv_bfloat16 *p) { return __bfloat162float(__ldg(p)); }
    static __device__ __forceinline__ void store4(__nv_bfloat16 *p, float a, float b, float c, float d)
    {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
        uint2 r;
        r.x = *reinterpret_cast<const uint32_t *>(&lo);
        r.y = *reinterpret_cast<const uint32_t *>(&hi);
        *reinterpret_cast<uint2 *>(p) = r;
    }
    static __device__ __forceinline__ void store2(__nv_bfloat16 *p, float a, float b) { *reinterpret_cast<__nv_bfloat162 *>(p) = __floats2bfloat162_rn(a, b); }
    static __device__ __forceinline__ void store1(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }
    static __device__ __forceinline__ float4 lds4(uint32_t a) { return widen(lds64(a)); }
};

template <typename IO>
struct IsFloat { static constexpr bool value = false; };
template <>
struct IsFloat<float> { static constexpr bool value = true; };

// Pixel at the upper left of the four integral-image values around `I` (rows of `pitch`).
__device__ __forceinline__ float pixel_of_integral(const float *I, int pitch)
{
    return __ldg(I + pitch + 1) - __ldg(I + 1) - __ldg(I + pitch) + __ldg(I);
}

// The same for eight rows of columns c .. c+3 from the integral row `I` above them on (rows of w + 1): every value is loaded once, not by all
// four pixels around it, and all of them are in flight together.  Zero at or past `rows` and column w.
template <class Emit>
__device__ __forceinline__ void pixels_of_integral(const float *I, int w, int c, int rows, Emit &&emit)
{
    float prev[5];
    int at[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        at[m] = min(c + m, w);
        prev[m] = rows > 0 ? __ldg(I + at[m]) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float cur[5], e[4];
        I += w + 1;
#pragma unroll
        for (int m = 0; m < 5; ++m) cur[m] = i < rows ? __ldg(I + at[m]) : 0.0f;
#pragma unroll
        for (int m = 0; m < 4; ++m) e[m] = i < rows && c + m < w ? cur[m + 1] - prev[m + 1] - cur[m] + prev[m] : 0.0f;
        emit(i, make_float4(e[0], e[1], e[2], e[3]));
#pragma unroll
        for (int m = 0; m < 5; ++m) prev[m] = cur[m];
    }
}

// ---- rows of four columns a lane, whatever their alignment -------------------------------------
// A warp works on 128 adjacent columns, lane L on columns c .. c+3 with c = c0 + 4 L.  Rows whose length is no
// multiple of four start anywhere relative to a 4-element boundary; k, the same for the whole warp, is by how
// many elements.  The memory access is then done on the aligned group that begins k elements earlier, one
// vector access a lane, and the elements move k places between neighbouring lanes by shuffles.
// All 32 lanes take part.  LN < 32: the warp is cut into groups of LN lanes, each on rows of its own (8 rows, or a
// multiple, apart), and c0 is 0; `lane` is then the lane within its group.  ALIGNED: k is zero for every row and w a multiple of four.
template <typename IO>
__device__ __forceinline__ int row_shift(const IO *row)
{
    return (int)(reinterpret_cast<uintptr_t>(row) / sizeof(IO)) & 3;
}

// Eight rows are loaded at a time: first all loads (rows8_load), then, where the values are used, the moves
// between lanes (rows8_get), so that the loads of all rows are in flight together.  The group that follows
// lane 31's is loaded for row i by lane i.
struct Rows8 {
    float4 a[8], next;
};
// Rows row0, row0 + w, ...; those at or past `rows` do not exist and read as zero.  PLAIN: the kernel may
// write the rows later.
template <typename IO, bool ALIGNED, bool PLAIN = false, int LN = 32>
__device__ __forceinline__ void rows8_load(Rows8 &g, const IO *row0, int w, int c, int rows, int lane)
{
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load = [](const IO *at) {
        if constexpr (PLAIN) return Io<IO>::load4_plain(at);
        else return Io<IO>::load4(at);
    };
    if (ALIGNED) {
        const IO *p = row0 + c;
#pragma unroll
        for (int i = 0; i < 8; ++i, p += w) g.a[i] = i < rows && c < w ? load(p) : zero;
        return;
    }
    const int k0 = row_shift(row0);
    const IO *p = row0 + c;
#pragma unroll
    for (int i = 0; i < 8; ++i, p += w) {
        const int k = (k0 + i * w) & 3;
        g.a[i] = i < rows && c - k < w ? load(p - k) : zero;
    }
    const int k = (k0 + lane * w) & 3, at = c - lane * 4 + 4 * LN - k;
    g.next = lane < rows && lane < 8 && k && at < w ? load(row0 + lane * w + at) : zero;
}
// Columns c .. c+3 of row i; zero from column w on.  The shift by k is done in two steps, by one and by two places,
// each with or without effect: four ways through the code would cost more instruction fetches than that saves.
template <typename IO, bool ALIGNED, int LN = 32>
__device__ __forceinline__ float4 rows8_get(const Rows8 &g, const IO *row0, int w, int c, int lane, int i)
{
    float4 a = g.a[i];
    if (ALIGNED) return a;
    const int k = (row_shift(row0) + i * w) & 3;
    const bool one = k & 1, two = k & 2, end = lane == LN - 1;
    const unsigned full = 0xffffffffu;
    const float e0 = __shfl_sync(full, g.next.x, i, LN), e1 = __shfl_sync(full, g.next.y, i, LN), e2 = __shfl_sync(full, g.next.z, i, LN);
    float n0 = __shfl_down_sync(full, a.x, 1, LN);
    if (end) n0 = e0;
    if (one) a = make_float4(a.y, a.z, a.w, n0);
    float m0 = __shfl_down_sync(full, a.x, 1, LN), m1 = __shfl_down_sync(full, a.y, 1, LN);
    if (end) {
        m0 = one ? e1 : e0;
        m1 = one ? e2 : e1;
    }
    if (two) a = make_float4(a.z, a.w, m0, m1);
    if (c >= w) a.x = 0.f;
    if (c + 1 >= w) a.y = 0.f;
    if (c + 2 >= w) a.z = 0.f;
    if (c + 3 >= w) a.w = 0.f;
    return a;
}

// Columns c .. c+3 of a row, as far as they are in the plane.  Rows of any alignment: one, two or three accesses, whatever the row's first
// element is aligned to.  Moving elements between lanes until groups are aligned costs kernels that gather more than the accesses it saves
// (1000 unaligned planes of up to 8 tiles, forward 1.19 of the time of single elements with, 1.05 without).
template <typename IO, bool ALIGNED>
__device__ __forceinline__ void store_row4(IO *row, int c, int w, const float (&v)[4])
{
    IO *p = row + c;
    if (c + 4 <= w) {
        const int k = ALIGNED ? 0 : row_shift(row);
        if (k == 0) {
            Io<IO>::store4(p, v[0], v[1], v[2], v[3]);
        } else if (k == 2) {
            Io<IO>::store2(p, v[0], v[1]);
            Io<IO>::store2(p + 2, v[2], v[3]);
        } else {
            Io<IO>::store1(p, v[0]);
            Io<IO>::store2(p + 1, v[1], v[2]);
            Io<IO>::store1(p + 3, v[3]);
        }
    } else if (!ALIGNED) {
#pragma unroll
        for (int m = 0; m < 3; ++m)
            if (c + m < w) Io<IO>::store1(p + m, v[m]);
    }
}

// `ok`: the row exists.  Unaligned rows: one vector store a lane for the aligned groups that lie inside the row and
// belong to this warp whole, and single elements for the rest: the 4 - k elements in front of the first group (the
// first lane's), the k behind the last one (the last lane's), and what the row's end cuts off a group.  For kernels that are bound by their stores:
// branches on the shift k, twice the code and fewer instructions (integral images of 512 planes of 256 x 512: 105 us against 115).
template <typename IO, bool ALIGNED, int LN = 32>
__device__ __forceinline__ void store_row4_wide(IO *row, int c, int w, const float (&v)[4], int lane, bool ok = true)
{
    if (ALIGNED) {
        if (ok && c < w) Io<IO>::store4(row + c, v[0], v[1], v[2], v[3]);
        return;
    }
    const int k = row_shift(row);
    float o[4] = {v[0], v[1], v[2], v[3]};
    if (k) {
        const float p3 = __shfl_up_sync(0xffffffffu, v[3], 1, LN);
        const float p2 = k > 1 ? __shfl_up_sync(0xffffffffu, v[2], 1, LN) : 0.f;
        const float p1 = k > 2 ? __shfl_up_sync(0xffffffffu, v[1], 1, LN) : 0.f;
        if (k == 1) { o[3] = v[2]; o[2] = v[1]; o[1] = v[0]; o[0] = p3; }
        else if (k == 2) { o[3] = v[1]; o[2] = v[0]; o[1] = p3; o[0] = p2; }
        else { o[3] = v[0]; o[2] = p3; o[1] = p2; o[0] = p1; }
        if (ok && lane == LN - 1) {      // its last k columns have no lane after them
#pragma unroll
            for (int m = 1; m < 4; ++m)
                if (m >= 4 - k && c + m < w) Io<IO>::store1(row + c + m, v[m]);
        }
    }
    if (!ok) return;
    const int first = lane == 0 ? c : c - k;      // lane 0 has no lane before it
    if (first == c - k && c - k + 4 <= w) {
        Io<IO>::store4(row + (c - k), o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int at = c - k + m;
            if (at >= first && at < w) Io<IO>::store1(row + at, o[m]);
        }
    }
}

// Rows 0 .. h of an integral image (plain rows of w + 1 floats) into shared memory by a CTA's warps: `put(a, col, value)`
// for the columns 0 .. cols-1, of which those past w repeat the value at w.  A warp has nine rows in flight; with one,
// whose load the store waits for, a CTA spent most of its time here ((1,8,4,32,32): 18 us, now 6.5).
template <class Put>
__device__ __forceinline__ void copy_integral_rows(const float *I, int h, int w, int cols, int warp, int nwarps, int lane, Put &&put)
{
    constexpr int kRowsInFlight = 9;      // (eight, and row 0, where a warp's share is a tile of eight rows)
    const int stride = nwarps * (w + 1);
    for (int a0 = warp; a0 <= h; a0 += kRowsInFlight * nwarps) {
        for (int col = lane; col < cols; col += 32) {
            const float *at = I + a0 * (w + 1) + min(col, w);
            float e[kRowsInFlight];
#pragma unroll
            for (int i = 0; i < kRowsInFlight; ++i) e[i] = a0 + i * nwarps <= h ? __ldg(at + i * stride) : 0.0f;
#pragma unroll
            for (int i = 0; i < kRowsInFlight; ++i)
                if (a0 + i * nwarps <= h) put(a0 + i * nwarps, col, e[i]);
        }
    }
}

inline bool aligned_to(const void *p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (uintptr_t)(bytes - 1)) == 0; }

inline bool ranges_overlap(const void *a, size_t a_bytes, const void *b, size_t b_bytes)
{
    const uintptr_t p = reinterpret_cast<uintptr_t>(a), q = reinterpret_cast<uintptr_t>(b);
    return p < q + b_bytes && q < p + a_bytes;
}

// Bounded waits that expired in the kernels of this translation unit (synchronises).
inline int read_wait_timeouts_here(int *count)
{
    if (cudaError_t e = cudaMemcpyFromSymbol(count, g_wait_timeouts, sizeof(int))) return cuda_failed(e, "read_wait_timeouts");
    return BC_OK;
}

}  // namespace

}  // namespace bc
