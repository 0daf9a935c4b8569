// How the rows kernel's tiles go into launches: arithmetic for the host alone, without CUDA, so that a test without a GPU can ask for the plan of a shape.
#pragma once

#include "../../include/jitnn_b200.h"

namespace jq {
namespace rows {

// Clusters of ks thread blocks that run at a time, one thread block per SM (cudaOccupancyMaxActiveClusters; the SMs of a GPC are not all a multiple of
// 4 or 8).
inline int clusters_of(int ks) { return ks == 1 ? 148 : (ks == 2 ? 74 : (ks == 4 ? 33 : 15)); }

// What a unit takes a thread block in nanoseconds, 16 rows of x, measured on 32000 x 4096. Q4_0 and Q8_0 take 720 and 770, a little less than is said here,
// and 8 rows of x a fifth less throughout: that would move a tile or two of shapes at a wave's edge from one launch to another, which gained nothing.
inline double unit_ns(int type) { return type == JQ_TYPE_Q4_K ? 630.0 : (type == JQ_TYPE_Q5_K ? 870.0 : (type == JQ_TYPE_Q4_0 || type == JQ_TYPE_Q8_0 ? 830.0 : (type == JQ_TYPE_Q4_1 ? 915.0 : 1010.0))); }

// A product's tiles in up to three launches, each with its own number of thread blocks per tile: whole waves first, then what is left, which alone would
// leave most of the chip idle for a whole contraction, with its contraction split over clusters (57344 x 8192: 448 tiles are three waves and four
// tiles: 85.5 us in one launch, 71.7 in two). The launch behind starts where SMs become free; GAP_NS is its own start.
// The cost of a launch is its waves' units and 1700 ns a wave, for a cluster 1600 more, which are rounder than what 16 rows of x take, us: one wave of 8, 16 and 32
// units 10.9, 15.7 and 25.6 (Q4_K), 14.4, 22.4 and 38.2 (Q6_K) and 13.2, 19.0 and 30.6 (Q8_0), that is 0.62, 0.99 and 0.73 a unit and 5.7 to 7.3 beside the units,
// the image kernel in front among them; a second wave of 16 in the same launch 10.5, 16.8 and 12.8; 16 units a thread block in clusters of 2, 4 and 8 2.5, 2.8 and 3.2
// (Q4_K), 5.3, 3.0 and 2.6 (Q6_K) and 1.7, 2.1 and 2.7 (Q8_0) more than alone. (8 rows of x: Q6_K 0.86 a unit, Q8_0 0.74.)
constexpr int MAX_PARTS = 3;
constexpr double GAP_NS = 2500.0;
struct Parts {
    int count;
    int tiles[MAX_PARTS], ksplit[MAX_PARTS];
};
inline double cut(int tiles, int units, double unit, int most, Parts& out) {
    double best = 1e30;
    for (int ks = 1; ks <= 8 && (ks == 1 || units >= 2 * ks); ks *= 2) {
        const int slots = clusters_of(ks), waves = (tiles + slots - 1) / slots;
        auto cost_of = [&](int w) { return w * (((units + ks - 1) / ks) * unit + 1700.0) + (ks > 1 ? 1600.0 : 0.0); };
        if (ks == 1 || waves == 1) {
            const double cost = cost_of(waves);
            if (cost < best) {
                best = cost;
                out.count = 1;
                out.tiles[0] = tiles;
                out.ksplit[0] = ks;
            }
        }
        const int whole = ks == 1 ? tiles / slots : 1, front = whole * slots;
        if (most > 1 && front > 0 && front < tiles) {
            Parts rest;
            const double cost = cost_of(whole) + GAP_NS + cut(tiles - front, units, unit, most - 1, rest);
            if (cost < best) {
                best = cost;
                out.count = 1 + rest.count;
                out.tiles[0] = front;
                out.ksplit[0] = ks;
                for (int i = 0; i < rest.count; i++) {
                    out.tiles[1 + i] = rest.tiles[i];
                    out.ksplit[1 + i] = rest.ksplit[i];
                }
            }
        }
    }
    return best;
}

}  // namespace rows
}  // namespace jq
