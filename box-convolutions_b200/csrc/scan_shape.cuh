// How the integral image's tiles are dealt out to CTAs and clusters of them; host code.
#pragma once
#include <cstdint>

namespace bc {

namespace {

constexpr int kScanWarps = 16;             // warps a CTA

// How a plane of `tiles` warps' rows and `warps` warps a row is dealt out.  Few planes: to a cluster of at most 8 CTAs of
// up to 16 warps, which hold it whole if they can (steps = 1; else they read it twice).  Many: to one CTA of 8 warps,
// which walks down it ((512,256,512): 102 us against 148 as clusters; CTAs of 16 warps 109), or of 16 where there are
// fewer planes than SMs and a cluster would read them twice in two steps ((130,161,715): 64 us, clusters 78; in three
// steps, (108,260,860): 92, 81).  `many16`: planes up to which the CTAs that walk have 16 warps.
struct ScanShape {
    int G, ctas, steps;
};
inline ScanShape scan_shape(int64_t planes, int tiles, int warps, int many16 = 148)
{
    ScanShape s;
    const int most = kScanWarps / warps;
    s.ctas = (tiles + most - 1) / most;
    s.steps = 1;
    if (s.ctas > 1 && (planes >= 148 || (planes >= 100 && s.ctas > 8 && s.ctas <= 16))) {
        s.ctas = 1;
        const int fit = planes < many16 ? most : (8 / warps > 1 ? 8 / warps : 1);
        s.steps = (tiles + fit - 1) / fit;
    } else if (s.ctas > 8) {
        s.steps = (s.ctas + 7) / 8;
        s.ctas = 8;
    }
    const int parts = s.ctas * s.steps;
    s.G = (tiles + parts - 1) / parts;
    return s;
}

// Clusters of eight CTAs of up to 16 warps: an SM runs two, a GPU 33, and 37, 45, 56, 71, 93 and 140 of those of seven to two CTAs (as asked of
// the occupancy calculator; `fit` is within three of that).  With a few planes more than fit, eight CTAs take as long again for the
// rest.  Planes that a cluster reads twice, in two steps or more, are therefore shared by as many CTAs (eight, or the fewest below) as make
// rounds times steps least, where that saves more than a quarter: (41,160,872) 27.7 us with clusters of 8, 16.6 with 5; (48,136,668) 24.1,
// 14.5; (85,272,528) 47.4, 32.4; (53,612,1077) 159, 124; (133,542,669) 188, 155; 42 of 115 drawn ones 0.79 of the time, none above 1.03.  In place of
// the walk of a CTA a plane (102,467,279) 84, 66, but not in the quad layout (140 planes of 364 x 430: 11 us more).  Planes that eight CTAs hold whole stay as they are: read twice they take 1.3 to
// 1.5 times as long.
inline ScanShape scan_clusters_that_fit(ScanShape s, int64_t planes, int tiles, int warps, bool quad)
{
    const int most = kScanWarps / warps, sets = (tiles + most - 1) / most;
    if (planes >= 148 || sets <= 8 || (quad && s.ctas == 1)) return s;
    auto dealt = [&](int ctas) {
        ScanShape d;
        d.ctas = ctas;
        d.steps = (sets + ctas - 1) / ctas;
        d.G = (tiles + ctas * d.steps - 1) / (ctas * d.steps);
        return d;
    };
    auto cost = [&](const ScanShape &d) {
        const int an_sm = 32 / (d.G * warps), fit = (2 * 142 * an_sm - 5 * (d.ctas - 1)) / (2 * d.ctas);      // (64 registers a thread)
        return (int)((planes + fit - 1) / fit) * d.steps * 4;
    };
    ScanShape best = dealt(8);
    int least = cost(best) / 4 * 3;
    for (int ctas = 2; ctas < 8; ++ctas) {
        const ScanShape d = dealt(ctas);
        if (cost(d) < least) best = d, least = cost(d);
    }
    return best.ctas < 8 ? best : s;
}

}  // namespace

}  // namespace bc
