// CPU check of trial_end (csrc/sms_trials.cuh): prints the Newton iterations
// counted after each of a fixed sequence of trial ends of one query.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>

using std::max;
using std::min;
#undef __launch_bounds__
#define __launch_bounds__(...)
struct Dim { unsigned x; };
static Dim threadIdx{0}, blockIdx{0}, blockDim{32}, gridDim{1};
template <class T, class U> static T atomicAdd(T *p, U v) { T o = *p; *p = o + (T)v; return o; }
template <class T, class U> static T atomicMin(T *p, U v) { T o = *p; *p = std::min(o, (T)v); return o; }
template <class T, class U> static T atomicMax(T *p, U v) { T o = *p; *p = std::max(o, (T)v); return o; }
template <class T, class U> static T atomicOr(T *p, U v) { T o = *p; *p = o | (T)v; return o; }
template <class T> static T __ldg(const T *p) { return *p; }
template <class T> static T __shfl_sync(unsigned, T v, int) { return v; }
template <class T> static T __shfl_xor_sync(unsigned, T, int) { return T(0); }
static unsigned __ballot_sync(unsigned, int p) { return p ? 1u : 0u; }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static void __syncwarp() {}

#include "sms_trials.cuh"

int main() {
    using namespace sms;
    DevCounters ctr{};
    LaneStats st;
    int count = kTrialOpen;
    const struct { int t, succ, it; } ends[] = {{4, 0, 1}, {5, 1, 10}, {7, 1, 100}, {6, 0, 1000},
                                                {2, 0, 10000}, {3, 1, 100000}, {5, 0, 1000000}};
    for (const auto &e : ends) {
        trial_end(&count, &ctr, 0, e.t, e.succ != 0, e.it, st);
        std::printf("%llu ", st.newton);
    }
    std::printf("%d %u %llu\n", count, ctr.trial_done, st.spec);
    return 0;
}
