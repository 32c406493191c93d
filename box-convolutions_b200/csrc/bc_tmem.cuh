// Tensor memory as a warp's private store: what the backward kernels keep of their pixels from filter to filter.
//
// A lane of those kernels owns 8 rows x 4 columns: 32 grad-input accumulators and 32 input values, used once a
// filter, row by row.  In registers the accumulators alone are a quarter of what two CTAs an SM leave a thread, and
// the input values cost the shared-memory pipe, the busiest one, a word per output.  Tensor memory (512 columns of
// 128 lanes an SM, a warp sees the 32 lanes of its number modulo 4) is private to warps by nature, needs no barriers
// between filters and is otherwise idle: 64 columns hold both.  Registers fall from 128 to 80 a thread, and an SM
// takes three CTAs of eight warps instead of two (five of four instead of four for slabs).
#pragma once
#include "bc_quad.cuh"

namespace bc {

constexpr int kTmemColumns = 64;      // per warp

// Columns of a CTA of at most 16 warps with T tiles each: warps w and w + 4 share lanes.  A power of two.
template <int T = 1>
__host__ __device__ __forceinline__ uint32_t tmem_columns(int nwarps) { return (nwarps > 8 ? 256u : nwarps > 4 ? 128u : 64u) * T; }

// One whole warp allocates and frees.  An allocation waits for columns that other CTAs of the SM hold, so a CTA
// allocates only behind grid_dependency_wait(): one that still waits for the kernel in front must not hold what
// that kernel's CTAs may ask for.
__device__ __forceinline__ void tmem_alloc(uint32_t *where, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(where)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
// Between the allocation and the first access by another warp, behind a barrier.
__device__ __forceinline__ void tmem_acquire() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Every warp's last access, in front of a barrier; then one warp frees.
__device__ __forceinline__ void tmem_release() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t columns)
{
    tmem_acquire();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
}

__device__ __forceinline__ void tmem_store8(uint32_t at, const float4 &a, const float4 &b)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(at), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w) : "memory");
}
__device__ __forceinline__ void tmem_store4(uint32_t at, const float4 &a)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w) : "memory");
}
__device__ __forceinline__ void tmem_load8(uint32_t at, float4 &a, float4 &b)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w),
                 "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "r"(at) : "memory");
}
__device__ __forceinline__ void tmem_load4(uint32_t at, float4 &a)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w) : "r"(at) : "memory");
}
// Four rows of four columns.
__device__ __forceinline__ void tmem_load16(uint32_t at, float4 (&v)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[0].z), "=f"(v[0].w), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[1].z), "=f"(v[1].w),
                   "=f"(v[2].x), "=f"(v[2].y), "=f"(v[2].z), "=f"(v[2].w), "=f"(v[3].x), "=f"(v[3].y), "=f"(v[3].z), "=f"(v[3].w)
                 : "r"(at) : "memory");
}
// (the loaded registers are operands, so that nothing uses them before)
__device__ __forceinline__ void tmem_wait_load(float4 &a, float4 &b)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(a.w), "+f"(b.x), "+f"(b.y), "+f"(b.z), "+f"(b.w)::"memory");
}
__device__ __forceinline__ void tmem_wait_load(float4 &a)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(a.x), "+f"(a.y), "+f"(a.z), "+f"(a.w)::"memory");
}
__device__ __forceinline__ void tmem_wait_load(float4 (&v)[4])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[0].z), "+f"(v[0].w), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[1].z), "+f"(v[1].w),
                   "+f"(v[2].x), "+f"(v[2].y), "+f"(v[2].z), "+f"(v[2].w), "+f"(v[3].x), "+f"(v[3].y), "+f"(v[3].z), "+f"(v[3].w)::"memory");
}
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// A lane's 8 rows of tile k of its warp's T.  Row i's eight words: its grad-input accumulators, then the input values
// of row i + AHEAD (modulo 8) that the gather of row i needs too, so that it fetches both at once.  All accesses are
// the whole warp's, in converged code.
template <int AHEAD, int T = 1>
struct TmemRows {
    uint32_t base;
    float4 g, e;
    __device__ __forceinline__ TmemRows(uint32_t cta_base, int warp, int k = 0)
        : base(cta_base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * T + k) * kTmemColumns)
    {
    }
    // before the first filter: row i's input values; accumulators that are zero
    __device__ __forceinline__ void init(int i, const float4 &x)
    {
        __syncwarp();
        tmem_store8(base + 8 * ((i + 8 - AHEAD) & 7), make_float4(0.f, 0.f, 0.f, 0.f), x);
    }
    __device__ __forceinline__ void sync() { tmem_wait_store(); }      // between filters, and behind init()
    __device__ __forceinline__ float4 first()      // AHEAD 1: row 0's input values
    {
        float4 v;
        __syncwarp();
        tmem_load4(base + 60, v);
        tmem_wait_load(v);
        return v;
    }
    __device__ __forceinline__ void fetch(int i) { tmem_load8(base + 8 * i, g, e); }
    __device__ __forceinline__ float4 next()
    {
        tmem_wait_load(g, e);
        return e;
    }
    __device__ __forceinline__ void add(int i, f2_t g01, f2_t g23, f2_t scale)
    {
        float4 v;
        unpack2(fma2(g01, scale, pack2(g.x, g.y)), v.x, v.y);
        unpack2(fma2(g23, scale, pack2(g.z, g.w)), v.z, v.w);
        tmem_store4(base + 8 * i, v);
    }
    __device__ __forceinline__ float4 grad_input(int i)
    {
        float4 v;
        __syncwarp();
        tmem_load4(base + 8 * i, v);
        tmem_wait_load(v);
        return v;
    }
};

}  // namespace bc
