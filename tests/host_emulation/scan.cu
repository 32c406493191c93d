// How the integral image's tiles are dealt out, for the unit tests: host code only, compiled by tests/test_scan_shape_host.py.
#include "scan_shape.cuh"

namespace bc {

// Checks every launch of up to `planes` planes of up to `tiles` tiles and `warps` warps a row; how many clusters of fewer than eight
// CTAs there are among those of several steps, or the negated number of wrong launches.
extern "C" int scan_shapes(int planes, int tiles, int warps)
{
    int smaller = 0, wrong = 0;
    for (int p = 1; p <= planes; ++p)
        for (int t = 1; t <= tiles; ++t)
            for (int w = 1; w <= warps; ++w) {
                const ScanShape was = scan_shape(p, t, w), s = scan_clusters_that_fit(was, p, t, w, false), quad = scan_clusters_that_fit(was, p, t, w, true);
                const bool same = s.G == was.G && s.ctas == was.ctas && s.steps == was.steps;
                wrong += s.G < 1 || s.G * w > kScanWarps || s.ctas < 1 || s.ctas > 8 || s.steps < 1 || s.G * s.ctas * s.steps < t;
                wrong += !same && (p >= 148 || (was.ctas > 1 && was.steps == 1) || s.ctas < 2 || s.steps < 2);
                const ScanShape &as = was.ctas == 1 ? was : s;
                wrong += quad.G != as.G || quad.ctas != as.ctas || quad.steps != as.steps;
                smaller += !same;
            }
    return wrong ? -wrong : smaller;
}

}  // namespace bc
