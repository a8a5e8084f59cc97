// Host-side rules and keys of the launches.  Plain C++ without CUDA, so that
// they are checked on the host alone.
#pragma once

#include <cmath>
#include <cstdint>
#include <vector>

namespace kpt {

// What a captured interval loop of a batch holds by value: the loop's shape,
// and of every run the particle count and the buffers of its cell sort.  A
// graph may be replayed only while all of them are the same; a store that
// grew or shrank, or whose sort buffers moved, needs a new capture.
struct BatchGraphShape {
    uint32_t intervals;
    int sort_tile, blocks_per_sm, sort_every, threads, particles_per_lane;
    bool records;
};
struct BatchGraphRun {
    uint64_t count;
    const void *order, *keys, *tile_counts;
};

inline std::vector<uint64_t> batch_graph_key(const BatchGraphShape& shape,
                                             const std::vector<BatchGraphRun>& runs) {
    std::vector<uint64_t> key = {shape.intervals,
                                 static_cast<uint64_t>(shape.sort_tile),
                                 static_cast<uint64_t>(shape.blocks_per_sm),
                                 static_cast<uint64_t>(shape.sort_every),
                                 static_cast<uint64_t>(shape.threads),
                                 static_cast<uint64_t>(shape.particles_per_lane),
                                 shape.records ? 1u : 0u};
    for (const BatchGraphRun& run : runs) {
        key.push_back(run.count);
        for (const void* p : {run.order, run.keys, run.tile_counts}) {
            key.push_back(static_cast<uint64_t>(reinterpret_cast<uintptr_t>(p)));
        }
    }
    return key;
}

// ---- cell records of a single push (KPT_RECORDS_AUTO)

struct RecordsCase {
    bool focused, learned;       // learned: the network's closure
    uint64_t particles, points;  // of the store, of a table
    double dt_min_rel, dt_max_rel;
    int sm_count;
};

// Whether a push gains from cell records.  They cost about 0.15 ns per table
// point to build, and a push that reads most of them from memory more than
// the point tables' rows.
//  * A quarter as many particles as points and more: always.
//  * Fewer, if they fill the chip (1.25 times the 640 lanes of the record
//    kernel's five blocks per SM, four times with the learned closure, whose
//    network hides more of the gathers):
//    - learned: from ten particle-steps a point on (counted with the fewest
//      substeps an interval can take).  421 891 particles on 1024 x 2048, 100
//      steps 4.85 -> 3.85 ms; 1 009 584 on 2048 x 4096, 100 steps 10.25 / 10.20.
//    - adaptive steps: likewise, and twice as many or two lanes' worth of
//      particles.  253 134 Parker on 1024 x 2048 17.97 -> 17.06 ms, 126 814 on
//      1024 x 1024 11.04 / 11.82.
//    - fixed steps run in rounds of the resident lanes: of three blocks per SM
//      on the point tables, of five, each 1.2 to 1.7 (Parker), 1.3 to 1.5
//      (focused) times as long with the table's size, on records.  What the
//      rounds save has to pay for the build.  Tables new in the interval, ms,
//      point tables / records: Parker 253 628 on 1024 x 1024, 100 steps 1.36 /
//      1.27; 506 269 on 1024 x 2048, 200 steps 5.12 / 4.56, 100 steps 2.57 /
//      2.60; 1 009 584 on 2048 x 4096, 100 steps 5.13 / 7.25, 400 steps 19.98 /
//      22.90; focused 253 628 on 1024 x 1024, 200 steps 4.06 / 3.58; 211 356 on
//      it, 200 steps 3.26 / 3.46.
inline bool records_pay(const RecordsCase& c) {
    if (c.particles * 4 >= c.points) return true;
    const double lanes = 640.0 * c.sm_count;
    const double particles = static_cast<double>(c.particles);
    const double points = static_cast<double>(c.points);
    if (particles < (c.learned ? 4.0 : 1.25) * lanes) return false;
    const double steps = 1.0 / c.dt_max_rel;  // the fewest
    if (c.learned) return particles * steps >= 10.0 * points;
    if (c.dt_min_rel != c.dt_max_rel) {
        return particles * steps >= (particles >= 2.0 * lanes ? 10.0 : 20.0) * points;
    }
    const double point_rounds = std::ceil(particles / (384.0 * c.sm_count));
    const double record_rounds = std::ceil(particles / lanes);
    const double longer = c.focused ? 1.3 + 0.025e-6 * points : 1.13 + 0.07e-6 * points;
    return steps * (0.97 * point_rounds - longer * record_rounds) >=
           (c.focused ? 0.8e-4 : 1.0e-4) * points;
}

}  // namespace kpt
