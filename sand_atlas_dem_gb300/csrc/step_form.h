// How a call's steps are dealt to persistent launches.  Plain host code.
#pragma once
#include <algorithm>
#include <cstdint>

namespace sdg {

// Steps of one persistent launch (even: each starts on the same history side): a
// few milliseconds at a time, so that a long chunk shares the GPU.
constexpr uint32_t RUN_STEPS = 64;

// Issues `steps` steps by `run(n)`, the next n in one launch, until it refuses one;
// returns how many were issued.  The rest, an even number on, is the caller's.
template <class Run>
uint32_t runSteps(uint32_t steps, Run&& run) {
    uint32_t done = 0;
    while (done < steps) {
        const uint32_t n = std::min(RUN_STEPS, steps - done);
        if (!run(n)) break;
        done += n;
    }
    return done;
}

}  // namespace sdg
