// Host-side rules and keys of the launches.  Plain C++ without CUDA, so that
// they are checked on the host alone.
#pragma once

#include <cmath>
#include <cstddef>
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
//    - learned: from 16 particle-steps a point on (counted with the fewest
//      substeps an interval can take).  Width 64, point tables / records:
//      421 891 particles on 1024 x 2048, 100 steps 4.11 / 3.97 ms, 400 steps
//      15.8 / 13.9; 506 269, 50 steps (12 a point) 2.48 / 2.57.
//    - adaptive steps: from ten, for two particles a lane and more (with fewer
//      the longest particles' chains are the time, and they are shorter on
//      the point tables).  253 134 Parker on 1024 x 2048 17.97 -> 17.06 ms, 361
//      922 on 1500 x 1500 51.3 -> 42.8; 126 814 on 1024 x 1024 11.04 / 11.82,
//      133 013 on 700 x 800 5.31 / 6.06, 124 655 on 512 x 1024 2.83 / 3.30.
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
    if (c.learned) return particles * steps >= 16.0 * points;
    if (c.dt_min_rel != c.dt_max_rel) {
        return particles * steps >= 10.0 * points && particles >= 2.0 * lanes;
    }
    const double point_rounds = std::ceil(particles / (384.0 * c.sm_count));
    const double record_rounds = std::ceil(particles / lanes);
    const double longer = c.focused ? 1.3 + 0.025e-6 * points : 1.13 + 0.07e-6 * points;
    return steps * (0.97 * point_rounds - longer * record_rounds) >=
           (c.focused ? 0.8e-4 : 1.0e-4) * points;
}

// ---- cell records of a batch (KPT_RECORDS_AUTO)

struct BatchRecordsCase {
    bool focused, learned;
    bool fixed;        // every run's step is fixed
    size_t runs;
    double particles;  // of all runs
    double points;     // of all runs' tables
    double steps;      // particle-steps of an interval, at least
    int sm_count;
};

// Whether a batch gains from cell records.  They are built once for a batch's
// tables and read by every interval; an interval reads each record it meets
// from DRAM, so a particle has to make enough substeps and the points enough
// particle-steps, more of them on a finer table, where a particle stays in a
// cell for less time.  As a rule a batch takes records from a quarter as many
// particles as points on; with fixed steps, where the substeps are known, a
// population that fills the chip goes by both: a dense one falls back to the
// point tables below the lower line, a thin one takes records above the higher
// one.  Particles as many as points: always.  Adaptive runs only add to their
// fewest substeps.  First interval / later ones in ms, point tables against
// records (runs x table, particles, substeps):
//   Parker   16 x  512 x  512, 2.50 M x  25   6.32 /  5.37    7.90 /  6.49
//                              2.50 M x  50   8.20 /  7.22    8.43 /  6.80
//                              0.99 M x 100   7.19 /  5.75    7.83 /  5.26
//             4 x 1024 x 2048, 2.52 M x  50   8.33 /  7.86   11.27 / 10.02
//                              2.52 M x 100  15.77 / 14.77   14.85 / 13.41
//            48 x  256 x  256, 1.89 M x  50   6.82 /  5.73    8.18 /  5.14
//   focused   4 x 1024 x 2048, 2.01 M x  50   9.67 /  9.22   11.76 /  9.92
//                              2.01 M x 100  18.02 / 17.57   17.32 / 15.61
//            16 x 1024 x 1024, 4.03 M x  50  19.37 / 18.29   22.97 / 19.23
//            48 x  256 x  256, 1.89 M x  25   6.68 /  5.58    8.16 /  5.06
//            16 x  512 x  512, 0.99 M x 100   9.81 /  9.16    9.23 /  7.60
inline bool batch_records_pay(const BatchRecordsCase& c) {
    const bool dense = c.particles * 4.0 >= c.points;
    if (c.learned || c.particles < 1.25 * 640.0 * c.sm_count || c.particles >= c.points) {
        return dense;
    }
    const double side = std::sqrt(c.points / static_cast<double>(c.runs));
    double substeps, per_point;
    if (c.focused) {
        substeps = dense ? 20.0 : 40.0;
        per_point = dense ? 0.006 * side + 8.0 : 0.0085 * side + 10.0;
    } else {
        substeps = dense ? 40.0 : 70.0;
        per_point = 0.014 * side + 8.0;
        if (!dense && per_point < 18.0) per_point = 18.0;
    }
    const bool pays = c.steps >= substeps * c.particles && c.steps >= per_point * c.points;
    return pays || (dense && !c.fixed);
}

// ---- residency of a push on the point tables

// Blocks of 128 threads per SM for a population above the build for few, plain
// closures: the build for points holds up to three, the record build (on the
// point tables) five.  Adaptive steps: three.  Fixed steps run in rounds of the
// resident lanes, each about as long as it is wide, so what counts is how full
// the last one is; tables far larger than the L2 cache punish more than three
// blocks, whose gathers evict each other.  100 steps, ms with 2 / 3 / 4 / 5
// blocks: Parker on 512 x 1024 75 000 0.43 / 0.51 / 0.41 / 0.50, 95 000 0.62 /
// 0.60 / 0.63 / 0.49, 110 000 0.62 / 0.62 / 0.70 / 0.74, 190 000 1.00 / 1.05 /
// 1.05 / 0.95; on 1024 x 2048 75 000 0.55 / 0.58 / 0.59 / 0.67, 95 000 0.73 /
// 0.62 / 0.80 / 0.92; focused QLT on 1024 x 2048 62 000 0.86 / 1.07 / 0.83 /
// 0.89, 110 000 1.22 / 1.07 / 1.47 / 1.83.
inline int point_blocks(uint64_t particles, bool fixed, double table_bytes, double l2_bytes,
                        int sm_count) {
    const int usual = 3;
    const uint64_t lanes = 128 * static_cast<uint64_t>(sm_count);  // of a block per SM
    if (!fixed || particles > 8 * usual * lanes) return usual;
    const bool fits = table_bytes <= 1.7 * l2_bytes;
    const double near[4] = {2.08, 3.0, 3.9, 4.75}, far[2] = {2.5, 3.0};
    int best = usual;
    double least = 0.0;
    for (int b = 2; b <= (fits ? 5 : 3); ++b) {
        const uint64_t resident = lanes * static_cast<uint64_t>(b);
        const uint64_t rounds = (particles + resident - 1) / resident;
        const double cost = static_cast<double>(rounds) * (fits ? near[b - 2] : far[b - 2]);
        if (b == 2 || cost < least) {
            best = b;
            least = cost;
        }
    }
    return best;
}

// ---- residency of a batch on the point tables

// Threads per SM for a batch that samples the point tables, of the `fit` that
// the batch's registers admit.  With fixed steps a batch runs in rounds of the
// resident lanes.  Three blocks of 128 share the tables' rows through L1
// better than five, whose rounds take 1.5 (few rounds) to 1.65 times as long,
// so they win where they need few more rounds: ms at 384 / 640 threads, 50
// steps, 980 000 Parker particles 3.31 / 3.60, 223 000 1.16 / 1.21 (focused
// 1.59 / 1.64), 112 000 0.59 / 0.66 (0.82 / 0.90); and lose where the last of
// the rounds is nearly empty: 190 000 1.02 / 0.96 (1.48 / 1.28), 84 000 0.54 /
// 0.49 (0.77 / 0.64), 64 000 0.46 / 0.41 (0.62 / 0.58).  Adaptive steps have no
// rounds and want the lanes: 192 000 Parker particles 9.40 / 8.97.  A population
// that one or two blocks hold takes no more: its warps then spread evenly, and
// share an L1 with fewer.  1 / 2 / 3 / 5 blocks, focused: 8 000 particles 0.20 /
// 0.25 / 0.33 / 0.27, 32 000 0.34 / 0.29 / 0.34 / 0.46.
inline int batch_point_threads(uint64_t particles, bool fixed, int fit, int sm_count) {
    const int few = 3 * 128;
    if (fit <= few || !fixed) return fit;
    const auto rounds = [&](int threads) {
        const uint64_t lanes = static_cast<uint64_t>(threads) * static_cast<uint64_t>(sm_count);
        return static_cast<double>((particles + lanes - 1) / lanes);
    };
    for (int threads = 128; threads < few; threads += 128) {
        if (rounds(threads) <= 1.0) return threads;
    }
    const double longer = rounds(fit) <= 4.0 ? 1.48 : 1.65;
    return longer * rounds(fit) < rounds(few) ? fit : few;
}

// ---- residency of the FP64 push

// Blocks per SM (each one warp per sub-partition).
//  * Every particle takes the same steps (dt_min = dt_max): the time is the
//    number of rounds of the population times the warps that share a
//    sub-partition, over how well that many keep its FP64 pipe busy (0.80,
//    0.92, 0.97, 1.0 of the best for 1 to 4 warps, measured at 400 000
//    particles).  A last round of a few has only the warps that they fill.
//    60 000 focused particles, 50 steps: 10.1 / 7.6 / 8.8 / 7.9 ms with 1 / 2 /
//    3 / 4 blocks; 25 000: 5.2 / 3.4 / 4.4 / 5.5 ms.
//  * Adaptive steps: the interval ends with its longest particles (6 840 of
//    a mean of 1 095 substeps on the driver's uniform field), whose substeps
//    take as long as the warps beside them allow: one block up to eight
//    populations of its lanes, two beyond.  40 000 Parker particles: 111 /
//    135 / 163 / 188 ms with 1 / 2 / 3 / 4 blocks, 131 072: 254 / 257 / 274 /
//    300, 400 000: 693 / 639 / 659 / 685.
// A request (blocks_per_sm of the push schedule, 0: none) is taken as it is,
// up to the `most` that fit.
inline int f64_blocks_per_sm(uint64_t particles, bool fixed, uint64_t lanes, int most,
                             int requested) {
    if (requested > 0) return requested < most ? requested : most;
    if (!fixed) return particles <= 8 * lanes || most < 2 ? 1 : 2;
    const double busy[4] = {0.80, 0.92, 0.97, 1.0};
    int best = 1;
    double least = 0.0;
    const auto round = [&](int warps) { return warps / busy[warps < 4 ? warps - 1 : 3]; };
    for (int b = 1; b <= most; ++b) {
        const uint64_t resident = lanes * static_cast<uint64_t>(b);
        const uint64_t full = particles / resident, rest = particles - full * resident;
        // a population of less than one round is spread over all warps
        double cost = static_cast<double>(full > 0 ? full : 1) * round(b);
        if (full > 0 && rest > 0) cost += round(static_cast<int>((rest + lanes - 1) / lanes));
        if (b == 1 || cost <= least) {
            best = b;
            least = cost;
        }
    }
    return best;
}

}  // namespace kpt
