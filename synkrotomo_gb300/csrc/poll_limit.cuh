// Time limit of a polling wait, in plain integers so that a host test can
// evaluate it.
#pragma once

#ifndef SYNK_HD
#ifdef __CUDACC__
#define SYNK_HD __host__ __device__ __forceinline__
#else
#define SYNK_HD inline
#endif
#endif

namespace synk {

// Counts the time the waiter has polled: of the time between two looks at most
// kPollGapNs.  A longer gap is time in which the GPU ran another process (the whole
// kernel, and whom it waits for, stood still), not time the wait has lasted.
constexpr unsigned long long kPollGapNs = 1000000ull;

struct PollLimit {
    unsigned long long last, spent;
    SYNK_HD void start(unsigned long long now) {
        last = now;
        spent = 0;
    }
    SYNK_HD bool over(unsigned long long now, unsigned long long limit_ns) {
        const unsigned long long gap = now - last;
        last = now;
        spent += gap < kPollGapNs ? gap : kPollGapNs;
        return spent > limit_ns;
    }
};

}  // namespace synk
