// Timing of launch variants against one another (glac_autotune, glac_ensemble_autotune).
#pragma once

#include <cuda_runtime.h>

namespace glac {

// seconds[v]: mean time of a call as variant v, over `reps` calls or a few more;
// returns the fastest.  Variants alike (same[v] < v, first_alike) share one time.
// call(v) makes one call, reset() puts back what calls change, check(status, what)
// raises.
//
// The variants take turns, in two or four rounds of which every second one goes
// backwards, after a call each that warms up.  Timed one after the other, they
// also differed by where the card was between its burst clock and its power cap:
// two numbers of one FP32 flow kernel at 32^3 x 64 on B200 got 2.41 and 2.56 ms, and
// of the Metropolis forms the slower one won (2.44 ms against 2.28; 2.25 and 2.28 at
// one clock).
template <typename Call, typename Reset, typename Check>
int time_variants(int n, const int *same, int reps, cudaStream_t st, Call call, Reset reset, Check check,
                  double *seconds) {
    struct Events {
        cudaEvent_t e[2] = {nullptr, nullptr};
        ~Events() {
            for (cudaEvent_t v : e)
                if (v) cudaEventDestroy(v);
        }
    } ev;
    for (cudaEvent_t &v : ev.e) check(cudaEventCreate(&v), "event");
    const int rounds = reps >= 4 ? 4 : 2, calls = (reps + rounds - 1) / rounds;
    for (int v = 0; v < n; v++) {
        seconds[v] = 0.0;
        if (same[v] == v) call(v);
    }
    reset();
    for (int round = 0; round < rounds; round++)
        for (int i = 0; i < n; i++) {
            const int v = round & 1 ? n - 1 - i : i;
            if (same[v] != v) continue;
            check(cudaEventRecord(ev.e[0], st), "event");
            for (int k = 0; k < calls; k++) call(v);
            check(cudaEventRecord(ev.e[1], st), "event");
            check(cudaEventSynchronize(ev.e[1]), "event sync");
            float ms = 0.f;
            check(cudaEventElapsedTime(&ms, ev.e[0], ev.e[1]), "elapsed");
            seconds[v] += ms * 1e-3 / (rounds * calls);
            reset();
        }
    int best = 0;
    for (int v = 0; v < n; v++) {
        seconds[v] = seconds[same[v]];
        if (seconds[v] < seconds[best]) best = v;
    }
    return best;
}

}  // namespace glac
