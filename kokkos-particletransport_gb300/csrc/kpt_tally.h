// Counters of one block of a push, in shared memory: they change when a
// particle finishes, is judged or falls back, so keeping them out of the
// registers costs nothing per substep and leaves 7 (14 with the network's)
// registers to the warps.  Host builds (the tests) add without atomics.
#pragma once

#ifdef __CUDACC__
#define KPT_TALLY_FN __device__ __forceinline__
#else
#define KPT_TALLY_FN static inline
static inline unsigned atomicAdd(unsigned* word, unsigned v) {
    const unsigned old = *word;
    *word = old + v;
    return old;
}
static inline void atomicMax(unsigned* word, unsigned v) { *word = *word < v ? v : *word; }
#endif

namespace kpt {

struct BlockTally {
    unsigned steps[2], fallbacks[2];  // low and high words
    unsigned pushed, failed, max_steps, judged;
    unsigned max_error;  // float bits (non-negative floats order like them)
};

KPT_TALLY_FN void tally_add(unsigned (&word)[2], unsigned v) {
    const unsigned old = atomicAdd(&word[0], v);
    if (old + v < old) atomicAdd(&word[1], 1u);
}

KPT_TALLY_FN unsigned long long tally_word(const unsigned (&word)[2]) {
    return (static_cast<unsigned long long>(word[1]) << 32) | word[0];
}

// A particle the block loaded has reached its last substep.
KPT_TALLY_FN void tally_finish(BlockTally& b, int steps, int status) {
    tally_add(b.steps, static_cast<unsigned>(steps));
    atomicAdd(&b.pushed, 1u);
    if (status != 0) atomicAdd(&b.failed, 1u);
    atomicMax(&b.max_steps, static_cast<unsigned>(steps));
}

// A particle the block loaded and gives up: `served` of its substeps had their
// closure served, and are counted, as their fallbacks have been.
KPT_TALLY_FN void tally_abandon(BlockTally& b, int served) {
    tally_add(b.steps, static_cast<unsigned>(served));
    atomicAdd(&b.pushed, 1u);
}

// Substeps whose closure the network served: every substep of a particle is
// served by the network or falls back.
KPT_TALLY_FN unsigned long long tally_evaluations(const BlockTally& b) {
    return tally_word(b.steps) - tally_word(b.fallbacks);
}

}  // namespace kpt
