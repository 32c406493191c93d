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
// Walks all sizes of at most 32 tiles of 32 x 32 whose padded integral image and two rows of sums a tile take at most 200 KB, which is what the
// whole-plane kernels serve: the number of wrong launches, the first of which is put into `at` (rows, columns).
template <class Wrong>
int64_t walk(int64_t *at, int64_t *sizes, Wrong &&wrong)
{
    int64_t n = 0;
    *sizes = 0;
    for (int h = 1; h <= 1024; ++h)
        for (int w = 1; w <= 1024; ++w) {
            const int tiles = ((h + 31) / 32) * ((w + 31) / 32);
            if (tiles > 32 || ((h + 1) * (w + 9) + h / 8 + 7 + 64 * tiles) * 4 > 200 * 1024) continue;
            ++*sizes;
            if (wrong(h, w) && !n++) at[0] = h, at[1] = w;
        }
    return n;
}
extern "C" int64_t flat_walk_backward(int N, int C, int F, int write_gin, int64_t *at, int64_t *sizes)
{
    return walk(at, sizes, [&](int h, int w) {
        const FlatPlan p = flat_backward_plan(N, C, F, h, w, write_gin != 0);
        const FlatShape &s = p.sh;
        const int T = p.tiles_a_warp, slots = 64 * T * ((p.warps + 3) / 4);
        return p.warps > (T == 1 ? 24 : 16) || s.tiles != p.warps * T || s.tiles * 32 < s.cells * s.planes || p.smem > kFlatMaxSmem ||
               (int64_t)p.smem < flat_image_bytes(s) + s.tiles * (544 + (T == 1 ? kFlatScanBytes : 0)) + F * (48 + p.warps * 20) || s.planes < 1 || s.planes > 255 ||
               s.planes > N || s.strips > 1023 || s.groups > 1023 || s.split < 1 || s.split > 8 || s.split > F || p.each != (F + s.split - 1) / s.split ||
               (s.columns & (s.columns - 1)) || s.columns < 64 || s.columns > 512 || slots * (s.split > 1 ? p.each : 1) > s.columns ||
               (write_gin && s.split > 1 && (int64_t)p.smem < (int64_t)s.tiles * 4096 * p.each);
    });
}
extern "C" int64_t flat_walk_forward(int N, int C, int F, int64_t *at, int64_t *sizes)
{
    return walk(at, sizes, [&](int h, int w) {
        const FlatForwardPlan p = flat_forward_plan(N, C, F, h, w);
        const FlatShape &s = p.sh;
        const int corners = p.warps * kFlatScanBytes;
        return p.warps > 32 || p.warps * 32 < s.cells * s.planes || s.planes < 1 || s.planes > N || p.smem > kFlatMaxSmem || p.fsplit < 1 || F % p.fsplit ||
               (p.tsplit != 1 && p.tsplit != 2 && p.tsplit != 4) || (p.tight && flat_image_bytes(s) < corners) ||
               (int64_t)p.smem < flat_image_bytes(s) + p.warps * 544 + F * 48 + (p.tight ? 0 : corners);
    });
}
extern "C" int64_t flat_walk_layout(int64_t *at, int64_t *sizes)
{
    return walk(at, sizes, [&](int h, int w) {
        const FlatShape s = flat_shape(h, w, 1);
        bool wrong = (flat_row_at(8, s.row, s.skew) / 4 - s.strips) % 32 || (s.plane / 4 - s.cells) % 32 || s.row != 4 * s.sub || s.sub != 4 * (s.strips + 4) ||
                     s.last != flat_row_at(h, s.row, s.skew) || s.last + s.row > s.plane;
        for (int group : {0, s.groups - 1})
            for (int a : {-h - 17, -9, -8, -1, 0, 1, 5, 7, 8, h, h + 16})
                for (int j = 0; j < 9; ++j) {
                    const int first = flat_row_at(group * kFlatRows + (a & ~7), s.row, s.skew), off = first + s.offset[(a & 7) + j], row = group * 8 + a + j;
                    wrong |= (off < 0 ? 0 : off > s.last ? s.last : off) != flat_row_at(row < 0 ? 0 : row > h ? h : row, s.row, s.skew);
                }
        return wrong;
    });
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
