// One warp's scans of the strips kernels (csrc/bc_flat.cuh) on the host, its lanes one after the other as far as the code's own warp
// barriers let them: what a lane writes before it is known that the others have read it shows as a wrong sum.  Host code only, compiled by
// tests/test_flat_host.py beside a copy of bc_flat.cuh and empty files in the place of what that includes; the few
// device functions that the scans use stand here.
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline

using std::max;
using std::min;

struct float4 { float x, y, z, w; };
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
struct Dim { unsigned x; };

namespace {

constexpr int kLanes = 32;
ucontext_t g_main, g_lane_at[kLanes];
int g_lane;
bool g_done[kLanes];
float g_value[kLanes];
std::vector<char> g_shared, g_stacks(kLanes * 65536);
const Dim threadIdx{0}, blockDim{kLanes};

void __syncwarp() { swapcontext(&g_lane_at[g_lane], &g_main); }
float __shfl_sync(unsigned, float v, int from)
{
    g_value[g_lane] = v;
    __syncwarp();
    const float r = g_value[from & 31];
    __syncwarp();
    return r;
}
float __shfl_down_sync(unsigned mask, float v, int d) { return __shfl_sync(mask, v, g_lane + d < kLanes ? g_lane + d : g_lane); }
unsigned __ballot_sync(unsigned mask, bool p)
{
    unsigned r = 0;
    for (int i = 0; i < kLanes; ++i) r |= (unsigned)(__shfl_sync(mask, (float)p, i) != 0.f) << i;
    return r;
}
int __ffs(unsigned v) { return __builtin_ffs((int)v); }
int __viaddmin_s32_relu(int a, int b, int c) { return max(min(a + b, c), 0); }

}  // namespace

namespace bc {

constexpr int kStrip = 4, kTapWords = 12, kNumSums = 5, kTmemColumns = 64;
struct f2_t { float x, y; };
struct BoxTaps { int lo_r, hi_r, lo_c, hi_c; };
template <typename IO>
struct Io;

inline f2_t pack2(float x, float y) { return {x, y}; }
inline void unpack2(f2_t v, float &x, float &y) { x = v.x; y = v.y; }
inline f2_t add2(f2_t a, f2_t b) { return {a.x + b.x, a.y + b.y}; }
inline uint32_t smem_u32(const void *) { return 0; }
template <int OFF>
void sts(uint32_t at, float v) { std::memcpy(&g_shared[at + OFF], &v, 4); }
template <int OFF>
float lds(uint32_t at) { float v; std::memcpy(&v, &g_shared[at + OFF], 4); return v; }
inline void sts128(uint32_t at, float4 v) { std::memcpy(&g_shared[at], &v, 16); }
inline float4 lds128(uint32_t at) { float4 v; std::memcpy(&v, &g_shared[at], 16); return v; }
inline float lds_row(uint32_t row, uint32_t off) { return lds<0>(row + off); }

}  // namespace bc

#include "bc_flat.cuh"

namespace bc {

namespace {

struct Work {
    const float *in;
    float *out;
    int h, w;
    FlatShape sh;
    FlatSmem s;
} g_work;

// What a warp that has all of a plane's tiles does up to its strips' stores.
template <int T>
void lane_main()
{
    const Work &k = g_work;
    const int lane = g_lane;
    FlatBlock v[T];
    float carry[T][kFlatRows];
    uint32_t starts[T];
    for (int t = 0; t < T; ++t) {
        const FlatCell cell = flat_cell(k.sh, t * 32 + lane, 1, k.h);
        starts[t] = __ballot_sync(0xffffffffu, cell.strip == 0);
        for (int i = 0; i < kFlatRows; ++i) {
            float e[4];
            for (int m = 0; m < 4; ++m) {
                const int c = cell.strip * 4 + m;
                e[m] = i < cell.rows && c < k.w ? k.in[(cell.group * kFlatRows + i) * k.w + c] : 0.f;
            }
            v[t].a[i] = pack2(e[0], e[1]);
            v[t].b[i] = pack2(e[2], e[3]);
        }
    }
    for (int t = 0; t < T; ++t) flat_scan<T>(v[t], carry[t], k.s, t, starts[t], k.sh.spans, 0, 1, lane);
    if (k.sh.spans) __syncwarp();
    for (int t = 0; t < T; ++t) flat_publish(v[t], carry[t], k.s, t * 32 / k.sh.strips * k.sh.strips / 32, t, starts[t], lane);
    for (int t = 0; t < T; ++t)
        for (int i = 0; i < kFlatRows; ++i) {
            float *to = k.out + ((t * 32 + lane) * kFlatRows + i) * 4;
            unpack2(v[t].a[i], to[0], to[1]);
            unpack2(v[t].b[i], to[2], to[3]);
        }
    g_done[lane] = true;
}

template <int T>
void run(bool backwards)
{
    for (int i = 0; i < kLanes; ++i) {
        g_done[i] = false;
        getcontext(&g_lane_at[i]);
        g_lane_at[i].uc_stack.ss_sp = &g_stacks[(size_t)i * 65536];
        g_lane_at[i].uc_stack.ss_size = 65536;
        g_lane_at[i].uc_link = &g_main;
        makecontext(&g_lane_at[i], lane_main<T>, 0);
    }
    for (int live = kLanes; live;) {
        live = 0;
        for (int i = 0; i < kLanes; ++i) {
            g_lane = backwards ? kLanes - 1 - i : i;
            if (g_done[g_lane]) continue;
            swapcontext(&g_main, &g_lane_at[g_lane]);
            live += !g_done[g_lane];
        }
    }
}

}  // namespace

// out: 32 T strips x 8 rows x 4 columns of sums over the row group's rows and the row's columns so far; published: their last rows.
extern "C" void flat_warp(int T, int backwards, int h, int w, const float *in, float *out, float *published)
{
    FlatShape sh = flat_shape(h, w, 1);
    sh.tiles = T;
    FlatSmem s{0, 0, (uint32_t)T * 512, (uint32_t)T * 544, 0};
    g_shared.assign((size_t)T * 544 + kFlatScanBytes, 0);
    g_work = Work{in, out, h, w, sh, s};
    T == 1 ? run<1>(backwards != 0) : run<2>(backwards != 0);
    std::memcpy(published, &g_shared[0], (size_t)T * 512);
}

}  // namespace bc
