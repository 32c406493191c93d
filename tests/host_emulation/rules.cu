// The dispatch rules of the whole-plane kernels and the launches they lead to, for the unit tests: host code only, compiled by
// tests/test_dispatch_rules_host.py.
#include "box_plane_kernels.cuh"

namespace bc {

// Threads of the pair backward's launch, the bound of the kernel that is launched and the tensor-memory columns of a CTA;
// 0 where the rule sends the plane elsewhere.
extern "C" int rule_pair_backward(int64_t planes, int F, int h, int w, int wide, int *bound, int *columns)
{
    if (!quad_pair_suits_backward(planes, F, h, w, wide != 0)) return 0;
    const int warps = quad_row_tiles(h) * quad_col_tiles(w) / 2;
    *bound = quad_pair_max_threads(quad_col_tiles(w), warps);
    *columns = (int)tmem_columns<2>(warps);
    return warps * 32;
}

// Which kernel the backward of an aligned plane runs in: 0 pairs of tiles, 1 one tile a warp, 2 square tiles, 3 strips.
extern "C" int rule_backward(int64_t planes, int F, int h, int w, int wide)
{
    const bool fast = h % kTileRows == 0 && w % kStrip == 0;
    return plane_backward_choice(planes, F, h, w, wide != 0, fast, fast);
}

// Backward from the input's integral image: by slabs?
extern "C" int rule_slabs_backward(int64_t planes, int F, int h, int w) { return plane_prefers_slabs_backward(planes, F, h, w); }

// Does the forward through tensor memory serve the plane?  If so, the tiles of a plane, the warps that build it and the
// tensor-memory columns of a CTA.
extern "C" int rule_tmem_forward(int64_t planes, int F, int h, int w, int *tiles, int *warps, int *columns)
{
    if (!tmem_suits_forward(planes, F, h, w)) return 0;
    *tiles = quad_row_tiles(h) * quad_col_tiles(w);
    *warps = tmem_forward_warps(h, w);
    *columns = h * kStrip;
    return 1;
}

}  // namespace bc
