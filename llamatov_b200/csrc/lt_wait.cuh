// The loop of a bounded wait, apart from what it waits for, so that it can also be compiled for the host and tested there.
#pragma once
#ifdef __CUDACC__
#define LT_WAIT_FN __device__ __forceinline__
#else
#define LT_WAIT_FN inline
#endif

namespace lt {
namespace tc {

// sleep(): true once the barrier has completed, else after a while.  *abort_flag is set by the first wait of the CTA that runs
// out of time, and looked at before every sleep: from then on a wait returns at once, however many are left.
template <class Sleep, class Clock, class GiveUp>
LT_WAIT_FN void bounded_wait(Sleep sleep, Clock now, long long limit, const volatile int* abort_flag, GiveUp give_up) {
    if (*abort_flag || sleep()) return;
    const long long t0 = now();
    while (!*abort_flag && !sleep()) {
        if (now() - t0 > limit) {
            give_up();
            return;
        }
    }
}

}  // namespace tc
}  // namespace lt
