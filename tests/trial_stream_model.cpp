// CPU model of the Bernoulli trials' stream (csrc/sms_trials.cuh): the header's
// own code, a warp of one lane per fiber, under randomly drawn interleavings.
// Fibers change at every atomic, before it and after it, and while a trial
// runs.  Prints the number of queries, over all runs, whose count is not their
// smallest successful trial.
//   trial_stream_model runs warps queries cap success_percent chunk
#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

static void yield();

// ------------------------------------------------ the device's vocabulary
using std::max;
using std::min;
#undef __launch_bounds__
#define __launch_bounds__(...)
struct Dim { unsigned x; };
static Dim threadIdx{0}, blockIdx{0}, blockDim{32}, gridDim{1};
template <class T, class U> static T atomicAdd(T *p, U v) { yield(); T o = *p; *p = o + (T)v; yield(); return o; }
template <class T, class U> static T atomicMin(T *p, U v) { yield(); T o = *p; *p = std::min(o, (T)v); yield(); return o; }
template <class T, class U> static T atomicMax(T *p, U v) { T o = *p; *p = std::max(o, (T)v); return o; }
template <class T, class U> static T atomicOr(T *p, U v) { T o = *p; *p = o | (T)v; return o; }
template <class T> static T __ldg(const T *p) { return *p; }
template <class T> static T __shfl_sync(unsigned, T v, int) { return v; }
template <class T> static T __shfl_xor_sync(unsigned, T, int) { return T(0); }
static unsigned __ballot_sync(unsigned, int p) { return p ? 1u : 0u; }
static int __popc(unsigned v) { return __builtin_popcount(v); }
static void __syncwarp() {}
static void __threadfence() {}

#include "sms_trials.cuh"

using namespace sms;

// ------------------------------------------------------------------ fibers
static ucontext_t g_main;
static std::vector<ucontext_t> g_ctx;
static std::vector<std::vector<char>> g_stack;
static std::vector<int> g_runnable;
static int g_now = -1;
static std::mt19937 g_rng;

static void yield() { swapcontext(&g_ctx[g_now], &g_main); }

// ------------------------------------------------------------------- model
static DevCounters g_ctr;
static std::vector<uint32_t> g_list;
static std::vector<int> g_count;
static std::vector<std::vector<char>> g_succ;
static int g_cap, g_chunk, g_pass;

static void warp() {
    TrialStream ts((unsigned)g_list.size(), g_cap, g_pass, 1);
    TrialBuffer buf;
    LaneStats st;
    uint32_t qi;
    int t;
    while (ts.next(buf, g_list.data(), g_count.data(), &g_ctr, g_pass, g_chunk, 1, 0, qi, t)) {
        for (unsigned k = g_rng() % 4; k > 0; --k) yield();   // the walk
        trial_end(g_count.data(), &g_ctr, qi, t, g_succ[qi][t] != 0, 1, st);
    }
    g_runnable.erase(std::find(g_runnable.begin(), g_runnable.end(), g_now));
    swapcontext(&g_ctx[g_now], &g_main);
}

static void run_pass(int warps) {
    g_ctx.assign(warps, ucontext_t());
    g_stack.assign(warps, std::vector<char>(64 * 1024));
    g_runnable.clear();
    for (int w = 0; w < warps; ++w) {
        getcontext(&g_ctx[w]);
        g_ctx[w].uc_stack.ss_sp = g_stack[w].data();
        g_ctx[w].uc_stack.ss_size = g_stack[w].size();
        g_ctx[w].uc_link = nullptr;
        makecontext(&g_ctx[w], warp, 0);
        g_runnable.push_back(w);
    }
    // one fiber at a time is held back for a while
    int held = -1, left = 0;
    while (!g_runnable.empty()) {
        if (left-- <= 0) {
            held = g_runnable[g_rng() % g_runnable.size()];
            left = (int)(g_rng() % 60);
        }
        g_now = g_runnable[g_rng() % g_runnable.size()];
        if (g_now == held && g_runnable.size() > 1) continue;
        swapcontext(&g_main, &g_ctx[g_now]);
    }
}

int main(int argc, char **argv) {
    if (argc != 7) return 2;
    const int runs = std::atoi(argv[1]), warps = std::atoi(argv[2]), n = std::atoi(argv[3]);
    const int percent = std::atoi(argv[5]);
    g_cap = std::atoi(argv[4]);
    g_chunk = std::atoi(argv[6]);
    gridDim.x = (unsigned)warps;
    long wrong = 0;
    for (int r = 0; r < runs; ++r) {
        g_rng.seed((unsigned)r);
        g_ctr = DevCounters{};
        g_list.resize(n);
        for (int i = 0; i < n; ++i) g_list[i] = (uint32_t)i;
        std::shuffle(g_list.begin(), g_list.end(), g_rng);
        g_count.assign(n, kTrialOpen);
        g_succ.assign(n, std::vector<char>(g_cap + 1, 0));
        for (auto &s : g_succ)
            for (int t = 1; t <= g_cap; ++t) s[t] = (int)(g_rng() % 100) < percent;
        for (g_pass = 0; g_pass < 2; ++g_pass) run_pass(warps);
        for (int i = 0; i < n; ++i) {
            int first = kTrialOpen;
            for (int t = g_cap; t >= 1; --t)
                if (g_succ[i][t]) first = t;
            wrong += g_count[i] != first;
        }
    }
    std::printf("%ld\n", wrong);
    return 0;
}
