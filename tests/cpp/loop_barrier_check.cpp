// Arrivals in the many-cycle launches' barrier counters over a simulation of argv[1] launches of argv[2]
// cycles (a barrier each at most) on 1,023 blocks: never up to the error bits, and the counters start
// over as seldom as that allows.
#include <cstdio>
#include <cstdlib>

#include "../../bsim_b200/csrc/loop_barrier.h"

int main(int, char **argv)
{
    const int64_t launches = atoll(argv[1]), cycles = atoll(argv[2]);
    const unsigned long long blocks = 1023;
    bsim::LoopBarriers b;
    unsigned long long arrivals = 0, most = 0, resets = 0;
    for (int64_t l = 0; l < launches; l++) {
        if (b.start_over(cycles)) {
            arrivals = 0;
            resets++;
        }
        arrivals += blocks * (unsigned long long)cycles;  // as if one counter took every barrier
        most = arrivals > most ? arrivals : most;
        if (arrivals >= bsim::LOOP_ERR) return 1;
    }
    printf("%llu arrivals at most, %llu resets\n", most, resets);
    return resets == (unsigned long long)((launches - 1) / (bsim::LOOP_MAX_BARRIERS / cycles)) ? 0 : 2;
}
