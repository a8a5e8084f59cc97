// Host-side rules and keys of the launches.  Plain C++ without CUDA, so that
// they are checked on the host alone.
#pragma once

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

}  // namespace kpt
