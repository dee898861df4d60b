// sms_trials.cuh -- scheduling of the unbiased estimators' Bernoulli trials.
//
// After the first walks, n_list queries wait for trials t = 1, 2, ... until
// the first success or the cap.  A trial is a walk of its own with its own run
// of random numbers, so any number of a query's trials can run at once; the
// answer is the smallest successful t, which count[q] holds while the trials
// run (kTrialOpen: none yet).  The trials form one stream in trial-major
// order -- every open query's t before anyone's t + 1 -- that the warps of a
// persistent grid consume lane by lane; a trial whose query is known to
// succeed earlier is dropped when it is drawn.  Large lists thus run few
// trials past a success (about lanes / n_list per query), and short lists
// spread over the whole chip: the last query's 256 trials are 256 lanes' work
// in one go instead of eight 32-trial rounds of one warp.
//
// What it costs is trials past a success: up to the grid's lanes / n_list per
// query.  Holding a query to 32 or 64 trials in flight was slower (points of the
// 512^2 water, GB300; one warp per query with 32 trials at a time before):
//   points             before    32     64    no limit
//   32,003              6.5 ms   3.6    3.3    3.2
//   7,321 (64^2, 100)   2.2      1.25   1.1    0.84
//   300 (host)          3.5      0.59   0.59   0.59
// (1M points: 40.5 -> 36.1 ms.)
//
// Where most queries succeed at their first trial, that is most of the work:
// pass 0 then runs t = 1 alone and pass 1 the rest (TrialRule).
#pragma once
#include "sms_device.cuh"
#include "sms_estimator.cuh"

namespace sms {

constexpr int kTrialOpen = 0x7fffffff;
// When the first trials run in a pass of their own (lists shorter than the
// grid's lanes only; longer ones run few trials past a success anyway).  A pass
// costs the latency of its longest walk; what it saves is the speculative
// trials of the queries that succeed at once.
//   kSplitNever   single scatter: 60,000 pane points x 64 0.61 ms in two passes,
//                 0.55 in one; 600,000 points of the 512^2 water x 100 17.6 and
//                 17.0
//   kSplitLong    chains and the two-stage solver, whose walks are long, for more
//                 than kTrialSinglePass grids' worth of trials: 20,011 slab
//                 points x 128 (14,529 listed, 32 grids of 3 blocks) 3.2 ms in
//                 two passes, 3.6 in one; two-stage pane, 90,000 x 32 (19 grids)
//                 0.90 and 0.96, 30,000 x 64 (12) 0.60 in one
//   kSplitAlways  deterministic seeds (mnee_init): every trial of a query is the
//                 same walk, so that the first one decides: 45,000 points of
//                 the 128^2 water x 32 1.53 ms in one pass, 0.82 in two
enum TrialSplit : int { kSplitNever, kSplitLong, kSplitAlways };
constexpr unsigned kTrialSinglePass = 16;

// How a launch runs its stream.
struct TrialRule {
    TrialSplit split = kSplitLong;
    // Warps over which a stream of less than 32 trials a warp spreads, 0: the
    // grid's (lanes of one warp wait for each other's rays, so the fewer the
    // better while walks wait for tree nodes).
    int warps = 0;
    // Whether next() may hand out fewer trials than wanted before the pass ends.
    bool even_end = false;
    // Size of a claim: by what a trial of every query is to all warps, growing
    // while a warp finds no open trial (30,000 two-stage pane points 0.75 ms,
    // 0.60), or by the warp's share of the whole stream (chains: 20,011 slab
    // points 3.22 ms, 3.19).
    bool claim_by_row = false;
};
// Single-scatter scenes of at most this many triangles spread over
// kSmallTreeWarps warps an SM: their walks wait for little and are bound by
// instruction issue, where more warps only get in each other's way.  3,000
// points x 32, over the grid's 36 warps an SM / 8 / 4 / 2: sphere 0.208 / 0.192
// / 0.175 / 0.178 ms, water of 18 triangles 0.398 / 0.360 / 0.340 / 0.325, of
// 450 0.422 / 0.414 / 0.403 / 0.390, of 1,922 0.486 / 0.483 / 0.484 / 0.504.
constexpr uint32_t kSmallTree = 512;
constexpr int kSmallTreeWarps = 2;
// Rounds a claim grows to while a warp finds no open trial.
constexpr unsigned kTrialClaimMax = 8;

// Trials [lo, hi] of one pass, and the lanes of a warp that take part (`most`
// at most).
struct TrialPlan {
    int lo, hi;
    int lanes;
};

SMS_D TrialPlan trial_plan(unsigned n_list, int cap, int pass, int most, TrialRule rule) {
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x / 32), all = 32ull * warps;
    const unsigned long long jobs = (unsigned long long)n_list * (unsigned)cap;
    const bool split = n_list < all && (rule.split == kSplitAlways ||
                                        (rule.split == kSplitLong && jobs > kTrialSinglePass * all));
    TrialPlan p;
    p.lo = 1;
    p.hi = cap;
    if (pass == 0) p.hi = split ? 1 : 0;
    else if (split) p.lo = 2;
    const unsigned long long mine = (unsigned long long)n_list * (unsigned)max(0, p.hi - p.lo + 1);
    const unsigned long long over = rule.warps > 0 ? min(warps, (unsigned long long)rule.warps) : warps;
    p.lanes = (int)min((unsigned long long)most, max(1ull, (mine + over - 1) / over));
    return p;
}

// A warp's end of the stream: a claimed range of the pass's trial indices and
// the drawn trials that wait for a lane.
struct TrialBuffer {
    uint32_t qi[64];
    int t[64];
};

struct TrialStream {
    unsigned long long cur = 0, end = 0;   // claimed range
    unsigned long long total;
    unsigned n_list;
    TrialPlan plan;
    TrialRule rule;
    int ready = 0;       // buffered trials
    unsigned rounds = 1; // of the last claim
    bool claimed = false, found = true;   // whether there was one, and an open trial in it
    bool drained = false;

    SMS_D TrialStream(unsigned n, int cap, int pass, int most = 32, TrialRule r = TrialRule())
        : n_list(n), plan(trial_plan(n, cap, pass, most, r)), rule(r) {
        total = (unsigned long long)n * (unsigned)max(0, plan.hi - plan.lo + 1);
    }

    // Draw up to `want` trials (at most 32), in stream order, for the lanes
    // of rank < want; returns whether this lane got one.  Called by the whole
    // warp.  Fewer than want: the pass has no more (or rule.even_end).
    SMS_D bool next(TrialBuffer &buf, const uint32_t *list, const int *count, DevCounters *ctr, int pass,
                    int chunk, int want, int rank, uint32_t &qi, int &t) {
        const unsigned full = 0xffffffffu;
        const int lane = (int)(threadIdx.x & 31);
        const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x / 32);
        int goal = want;
        while (ready < goal && !drained) {
            if (cur >= end) {
                // A claim is one to four rounds of the warp, chunk at least.
                const unsigned long long grid = warps * (unsigned)plan.lanes;
                const unsigned share = (unsigned)min(4ull, rule.claim_by_row ? n_list / grid : total / (4ull * grid));
                rounds = max(max(found || !rule.claim_by_row ? 1u : min(2u * rounds, kTrialClaimMax), share),
                             (unsigned)chunk);
                found = false;
                unsigned claim = (unsigned)plan.lanes * rounds;
                // Once every query has a success the warp stops, and it looks
                // before it claims: a claimed range is never dropped, because it
                // can hold a trial before a success that another warp found in
                // a later range in the meantime.  All ranges before a success
                // then belong to warps that run them.  The first claim does not
                // look: all warps make it at once, and with a look before it
                // those near the counter took the whole of a short stream
                // (100 points of the 512^2 water 0.60 ms, without 0.53).
                unsigned long long got = total;
                if (lane == 0) {
                    bool more = true;
                    if (claimed) {
                        more = *(volatile unsigned *)&ctr->trial_done < n_list;
                        // The last part of a short stream goes to all warps, a
                        // few trials each, instead of full warps that run it for
                        // a whole walk of 32 diverging lanes (115,000 points of
                        // the 512^2 water x 32, 1.06 grids of trials: 3.73 ms,
                        // shared out 2.95).
                        if (rule.even_end && total <= 64ull * warps) {
                            const unsigned long long at = *(volatile unsigned long long *)&ctr->trial_jobs[pass];
                            const unsigned long long left = at < total ? 4ull * (total - at) / warps : 0ull;
                            if (left < claim) claim = (unsigned)max(1ull, left);
                        }
                    }
                    if (more) got = atomicAdd(&ctr->trial_jobs[pass], (unsigned long long)claim);
                }
                claimed = true;
                claim = __shfl_sync(full, claim, 0);
                if (rule.even_end) goal = min(goal, (int)claim);
                cur = __shfl_sync(full, got, 0);
                end = min(cur + claim, total);
                if (cur >= total) { drained = true; break; }
            }
            const int k = (int)min((unsigned long long)plan.lanes, end - cur);
            bool open = false;
            uint32_t q = 0;
            int tt = 0;
            if (lane < k) {
                const unsigned long long j = cur + (unsigned)lane;
                const unsigned long long row = (j >> 32) == 0 ? (unsigned)j / n_list : j / n_list;
                tt = plan.lo + (int)row;
                q = list[(unsigned)(j - row * n_list)];
                open = *(volatile const int *)(count + q) > tt;
            }
            const unsigned m = __ballot_sync(full, open);
            found = found || m != 0u;
            if (open) {
                const int at = ready + __popc(m & ((1u << lane) - 1u));
                buf.qi[at] = q;
                buf.t[at] = tt;
            }
            ready += __popc(m);
            cur += (unsigned)k;
        }
        __syncwarp();
        const int take = min(ready, want);
        const bool mine = rank < take;
        if (mine) { qi = buf.qi[rank]; t = buf.t[rank]; }
        // what is left moves to the front (fewer than 32 entries)
        uint32_t q2 = 0;
        int t2 = 0;
        const bool move = take + lane < ready;
        if (move) { q2 = buf.qi[take + lane]; t2 = buf.t[take + lane]; }
        __syncwarp();
        if (move) { buf.qi[lane] = q2; buf.t[lane] = t2; }
        ready -= take;
        __syncwarp();
        return mine;
    }
};

// Record the end of trial t of query qi.
SMS_D void trial_end(int *count, DevCounters *ctr, uint32_t qi, int t, bool succ, int it, LaneStats &st) {
    st.spec++;   // the trials up to each query's first success are taken out at the end
    const int before = succ ? atomicMin(count + qi, t) : *(volatile const int *)(count + qi);   // the success known so far
    if (succ && before == kTrialOpen) atomicAdd(&ctr->trial_done, 1u);
    if (before > t) st.newton += (unsigned)it;
}

// The estimate's trial statistics once all trials have run: f the first
// success or kTrialOpen.
SMS_D void trial_stats(int f, int cap, bool unbounded, uint32_t &err, LaneStats &st) {
    const bool found = f != kTrialOpen;
    const unsigned long long w = (unsigned long long)(found ? f : cap);
    if (!found && unbounded) err |= kErrTrialLimit;
    st.walks += w;
    st.spec -= w;
    st.calls++;
    st.iters += found ? w : w + 1;
    st.imax = max(st.imax, found ? w : w + 1);
}

// A result of n_list queries after their trials: value += first-walk
// contribution x trial count (over the template's offset density pdf, where
// given), the query's stream position behind its trials.
static __global__ void __launch_bounds__(128) trials_finish_kernel(uint32_t n, float *__restrict__ value,
                                                                   int *__restrict__ count, int *__restrict__ walks,
                                                                   SsScratch scr, const float *__restrict__ pdf,
                                                                   int cap, int unbounded, uint32_t stride, int phase,
                                                                   DevCounters *ctr) {
    LaneStats st;
    uint32_t err = 0;
    const unsigned n_list = *(volatile unsigned *)&ctr->trial_count;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n_list; i += gridDim.x * blockDim.x) {
        const uint32_t qi = scr.list[i];
        const int f = count[qi];
        const bool found = f != kTrialOpen;
        const float inv_prob = found ? (float)f : 0.f;
        const int trial_walks = found ? f : cap;
        trial_stats(f, cap, unbounded != 0, err, st);
        f3 cur = mk(scr.val[qi], scr.val[(size_t)n + qi], scr.val[2 * (size_t)n + qi]) * inv_prob;
        if (pdf) cur = mk(cur.x / pdf[qi], cur.y / pdf[qi], cur.z / pdf[qi]);
        value[qi] += cur.x;
        value[(size_t)n + qi] += cur.y;
        value[2 * (size_t)n + qi] += cur.z;
        count[qi] = found ? f : -1;
        walks[qi] += trial_walks;
        scr.pos[qi] += stride * (uint32_t)trial_walks;
    }
    flush_stats(st, ctr, err, phase);
}

// Lanes of a warp that run first walks, one query each.  Lanes of one warp
// wait for each other's rays, so a batch below kFirstWarps full warps per SM
// (two per scheduler, enough to hide each other's latency) takes that many
// warps with fewer queries each: 300 points 0.67 -> 0.20 ms; spread over all
// resident warps instead, larger batches lose to the extra instructions (pane
// of 30,000 points, 32 / 25 / 6 queries a warp: 0.19 / 0.19 / 0.44 ms).
constexpr int kFirstWarps = 8;
inline int first_walk_lanes(uint32_t n, int num_sms) {
    const uint32_t warps = (uint32_t)(num_sms * kFirstWarps), l = n / warps + (n % warps != 0);
    return (int)(l < 1 ? 1 : l > 32 ? 32 : l);
}
inline uint32_t first_walk_blocks(uint32_t n, int lanes) { return ((n - 1) / (uint32_t)lanes + 1 + 3) / 4; }

// Whether a pass of first trials may run at all for a batch of n queries on a
// grid of `blocks` blocks (trial_plan decides by the list's length).
inline bool trial_split_possible(TrialRule rule, uint32_t n, int cap, int blocks) {
    if (rule.split != kSplitLong) return rule.split == kSplitAlways;
    return (unsigned long long)n * (unsigned)cap > (unsigned long long)kTrialSinglePass * 128u * (unsigned)blocks;
}

inline uint32_t finish_blocks(uint32_t n, int num_sms) {
    const uint32_t b = (n - 1) / 128 + 1, most = 8 * (uint32_t)num_sms;
    return b < most ? b : most;
}

}  // namespace sms
