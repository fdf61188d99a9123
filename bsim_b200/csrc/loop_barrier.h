// What the host keeps of the many-cycle launches' grid barrier (step.cu).
//
// The barrier's counters only grow: every block adds one per passage, and LOOP_ERR with it when it has
// seen an error. The arrivals of a long simulation would reach the error bits after 2^40 (about a day of
// 3 us cycles on 148 SMs), so the counters are set to zero, in stream order between two launches, before
// LOOP_MAX_BARRIERS barriers have been passed since the last time. (Counters that the kernel itself
// zeroes or that may wrap made 10 x 1,000 neurons 3.16 -> 3.27 and 3.32 us per cycle.)
#pragma once
#include <stdint.h>

namespace bsim {

constexpr unsigned long long LOOP_ERR = 1ull << 40;  // one block's error in a barrier counter; arrivals are below
constexpr int64_t LOOP_MAX_BARRIERS = 1ll << 30;     // of up to 1,023 blocks: below 2^40 arrivals

struct LoopBarriers {
    int64_t passed = 0;  // since the counters were last zero, at most

    // Before a launch of up to n barriers: whether the counters start over.
    bool start_over(int64_t n)
    {
        const bool over = passed + n > LOOP_MAX_BARRIERS;
        passed = (over ? 0 : passed) + n;
        return over;
    }
};

}  // namespace bsim
