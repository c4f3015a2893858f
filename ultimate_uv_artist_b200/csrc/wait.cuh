// Polling with a limit, shared by the kernels' mbarrier waits.
#pragma once

#ifdef __CUDACC__
#define UVA_WAIT_FN __host__ __device__ __forceinline__
#else
#define UVA_WAIT_FN inline
#endif

namespace uva {

// Calls of poll() until it is true, `limit` of them at most; a wait that runs
// out sets `out`, the flag of all that wait with it, after which every other
// wait ends within kWaitBurst polls: many waits end soon after the first, and
// not after the sum of their limits. (A look at the flag between every two polls
// costs ARAP 0.5 %.)
constexpr int kWaitBurst = 64;

template <typename Poll>
UVA_WAIT_FN bool bounded_wait(Poll poll, int limit, volatile int& out) {
    for (int it = 1; it <= limit; ++it) {
        if (poll()) return true;
        if (it % kWaitBurst == 0 && out != 0) break;
    }
    out = 2;
    return false;
}

}  // namespace uva
