// Layout and launches of the whole-plane kernels that deal out strips, for the unit tests: host code only, compiled by
// tests/test_flat_host.py.
#include "bc_flat.cuh"

namespace bc {

// warps, tiles a warp, planes, split, columns, shared memory, strips a row, row groups, bytes of a plane's image, offset of its last row, bytes from row to row and
// of a sub-row, words from row group to row group and from plane to plane beyond what its strips take
extern "C" void flat_backward(int N, int C, int F, int h, int w, int write_gin, int64_t *out)
{
    const FlatPlan p = flat_backward_plan(N, C, F, h, w, write_gin != 0);
    const FlatShape &s = p.sh;
    const int64_t v[] = {p.warps, p.tiles_a_warp, s.planes, s.split, s.columns, (int64_t)p.smem, s.strips, s.groups, s.plane, s.last, s.row, s.sub,
                         (flat_row_at(8, s.row, s.skew) / 4 - s.strips) % 32, (s.plane / 4 - s.cells) % 32, s.tiles, flat_image_bytes(s)};
    for (int i = 0; i < 16; ++i) out[i] = v[i];
}
// warps, planes, parts of the filters, parts of the tiles, shared memory, strips a row, row groups
extern "C" void flat_forward(int N, int C, int F, int h, int w, int64_t *out)
{
    const FlatForwardPlan p = flat_forward_plan(N, C, F, h, w);
    const int64_t v[] = {p.warps, p.sh.planes, p.fsplit, p.tsplit, (int64_t)p.smem, p.sh.strips, p.sh.groups, flat_image_bytes(p.sh), p.tight};
    for (int i = 0; i < 9; ++i) out[i] = v[i];
}
// Offsets, as the kernels add them up, of the tap row `row` less than 16 below the start of row group `group`'s first one at `a`.
extern "C" int flat_offset(int h, int w, int group, int a, int j)
{
    const FlatShape s = flat_shape(h, w, 1);
    const int first = flat_row_at(group * kFlatRows + (a & ~7), s.row, s.skew), at = first + s.offset[(a & 7) + j];
    return at < 0 ? 0 : at > s.last ? s.last : at;
}
extern "C" int flat_row(int h, int w, int a)
{
    const FlatShape s = flat_shape(h, w, 1);
    return flat_row_at(a, s.row, s.skew);
}

}  // namespace bc
