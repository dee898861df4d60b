// sms_ss_kernels.cuh -- the single-scatter estimator kernels (biased, unbiased
// first walks, Bernoulli trials) and their per-caster launchers, templated on
// the caster variant kVar: bit 0 rough (offset normals), bit 1 two-stage
// solver, bit 2 normal-mapped manifold vertices.  sms_ss.cu instantiates the
// plain and rough variants, sms_ss_nm.cu the normal-mapped ones, so neither
// translation unit carries all of them.
//
// Random-number layout: query i owns stream (seed, stream) -- 3 numbers for
// the emitter sample, then per caster its offset normal (2, rough casters)
// and per walk the seed (2; 3 with a learned proposal) and, with the
// two-stage solver, the slope of its smoothed first solve (2, drawn for every
// walk so that walk m always starts at the same position).
#pragma once
#include <algorithm>

#include "sms_device.cuh"
#include "sms_estimator.cuh"
#include "sms_kernels.h"
#include "sms_mlp.cuh"
#include "sms_trials.cuh"

namespace sms {

// Resident blocks per SM the first-walk and trial kernels are compiled for
// (128 threads each): 9 gives 56 registers per thread, the measured optimum of
// the latency-bound walks (the headline step at 4 / 6 / 7 / 8 / 10 blocks:
// 62.4 / 53.3 / 50.6 / 49.7 / 57.8 ms; with the current traversal loop 8 and
// 9 blocks: 42.9 and 42.1 ms).
#ifndef SMS_SS_WALK_MIN_BLOCKS
#define SMS_SS_WALK_MIN_BLOCKS 9
#endif
// Normal-mapped casters: the map's frame and the two-stage solver add
// arithmetic, not traversal, so what counts is that the step stays in
// registers.  4 blocks (128 registers); pane of 30,000 points with the
// two-stage solver at 4 / 5 / 6 / 9 blocks: 0.60 / 0.75 / 0.86 / 1.05 ms.
constexpr int ss_walk_blocks(int var) { return (var & 4) ? 4 : SMS_SS_WALK_MIN_BLOCKS; }

// The same of the biased estimator's kernel for large batches (see below), and
// the blocks per SM from which a batch is large.  4 / 6 / 8 blocks, biased:
//   sphere, 13,355 points x 32 walks (22 blocks per SM)     374 / 348 / 376 us
//   sphere, 3,745 x 24 (6)                                  130 / 136 / 127 us
//   water 256^2, 16,000 x 32 (26)                           4.7 / 3.8 ms
//   pane, two-stage, 82,185 x 64 (135)                      22.4 / 19.8 / 18.5 ms
//   pane, two-stage, 11,000 x 16 (9); 12,000 x 32 (20)      0.48 / - / 0.55; 1.36 / - / 1.38 ms
//   pane, one stage, 51,728 x 64 (85)                       4.9 / 5.0 / 5.0 ms
constexpr int ss_biased_blocks(int var) { return var == 0 ? 6 : var == 6 ? 8 : 4; }
constexpr uint32_t ss_biased_large(int var) { return var == 0 ? 8u : 32u; }

// ------------------------------------------------------ biased estimator
// Group of G lanes per query; walk m of caster c sits at stream position
// 3 + 2 (c M + m).  Contributions are summed in walk order over the first
// occurrences of each solution direction, exactly as manifold_ss.cpp:146-196.
// Compiled for kBlocks resident blocks per SM (128 threads): 4 hold the Newton
// step in registers, which is what counts while the batch fits the chip; more
// hide more of its latency in larger batches (ss_biased_blocks).
template <int G, int kVar, int kBlocks>
__global__ void __launch_bounds__(128, kBlocks) ss_biased_kernel(DevScene sc, SolverCfg cfg, const float *__restrict__ qs,
                                                        uint32_t n, uint64_t seed, uint64_t stream_off,
                                                        float *__restrict__ value, int *__restrict__ count,
                                                        int *__restrict__ walks, DevCounters *ctr) {
    constexpr bool kRough = (kVar & 1) != 0, kTwo = (kVar & 2) != 0, kNM = (kVar & 4) != 0;
    constexpr uint32_t kWalk = kTwo ? 4u : 2u;   // numbers per walk: seed position (+ two-stage slope)
    constexpr int kGroupsPerBlock = 128 / G;
    __shared__ f3 rec[kGroupsPerBlock][kMaxSolutions];
    const unsigned full = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31;
    const int gl = (int)(threadIdx.x % G);             // lane within group
    const int gib = (int)(threadIdx.x / G);            // group within block
    const int gbase = (int)(lane & ~(unsigned)(G - 1));
    const unsigned gmask = (G == 32) ? full : (((1u << G) - 1u) << gbase);
    LaneStats st;
    uint32_t err = 0;
    const int M = cfg.max_trials > 0 ? cfg.max_trials : 0;
    const uint32_t groups_total = gridDim.x * kGroupsPerBlock;
    // every group of the grid runs the same number of rounds (full-warp syncs)
    const uint32_t rounds = (n + groups_total - 1) / groups_total;
    for (uint32_t r = 0; r < rounds; ++r) {
        uint32_t qi = (r * gridDim.x + blockIdx.x) * kGroupsPerBlock + gib;
        bool live = qi < n;
        Query Q{};
        Light L{};
        bool have_light = false;
        if (live) {
            Q = load_query(qs, n, qi);
            Pcg32 rng = query_rng(seed, query_stream(cfg, stream_off, qi), 0);
            have_light = sample_emitter(sc, sc.emitters_ss, sc.n_emitters_ss, rng, Q.x, L);
        }
        bool work = live && have_light && sc.n_casters_ss > 0;
        if (work && gl == 0) st.conns++;
        f3 acc = splat(0.f);
        int n_unique = 0;
        uint64_t cpos = 3u;   // stream position of the caster's first draw
        for (int c = 0; c < sc.n_casters_ss; ++c) {
            int caster = sc.casters_ss[c];
            const DevShape &cs = sc.shapes[caster];
            float p_off = 1.f;
            f3 no = mk(0.f, 0.f, 1.f);
            if (kRough && work && cs.alpha > 0.f) {
                Pcg32 r0 = query_rng(seed, query_stream(cfg, stream_off, qi), cpos);
                no = caster_offset(cs, r0, p_off);
            }
            const uint64_t wpos = cpos + caster_draws(cs);
            int nrec = 0;
            f3 cur = splat(0.f);
            for (int m0 = 0; m0 < M; m0 += G) {
                int m = m0 + gl;
                bool cand = false;
                f3 dir = splat(0.f), contrib = splat(0.f);
                if (work && m < M) {
                    Pcg32 rng = query_rng(seed, query_stream(cfg, stream_off, qi), wpos + kWalk * (uint64_t)m);
                    float sx = rng.next_f32(), sy = rng.next_f32();
                    f3 sp = sample_position(sc, cs, sx, sy);
                    float g0 = 0.f, g1 = 0.f;
                    if (kTwo) { g0 = rng.next_f32(); g1 = rng.next_f32(); }
                    Vtx v;
                    int it;
                    bool ok = ss_walk<kRough, kTwo, kNM>(sc, cfg, caster, Q.x, L.p, sp, v, it, err, st, nullptr, no,
                                                         g0, g1);
                    st.walks++;
                    st.newton += (unsigned)it;
                    if (ok) {
                        st.succ++;
                        if (visible(sc, L.p, v.p, err, st)) {
                            cand = true;
                            dir = normalize(v.p - Q.x);
                            // evaluated for every visible solution; only first
                            // occurrences are kept below
                            contrib = receiver_eval(sc, Q, dir, err) * contribution<kNM>(sc, Q.x, L, v, err, st);
                        }
                    } else {
                        st.fail++;
                    }
                }
                // walk-ordered deduplication within the group, one pass per candidate
                unsigned pend = __ballot_sync(full, cand) & gmask;
                while (__any_sync(full, pend != 0u)) {
                    const int src = pend ? __ffs(pend) - 1 : (int)lane;
                    f3 dk = mk(__shfl_sync(full, dir.x, src), __shfl_sync(full, dir.y, src),
                               __shfl_sync(full, dir.z, src));
                    f3 vk = mk(__shfl_sync(full, contrib.x, src), __shfl_sync(full, contrib.y, src),
                               __shfl_sync(full, contrib.z, src));
                    bool dup = false;
                    if (pend)
                        for (int j = gl; j < nrec; j += G)
                            if (fabsf(dot(dk, rec[gib][j]) - 1.f) < cfg.uniqueness_threshold) dup = true;
                    unsigned anydup = __ballot_sync(full, dup) & gmask;
                    __syncwarp();
                    if (pend && !anydup) {
                        if (nrec < kMaxSolutions) {
                            if (gl == 0) rec[gib][nrec] = dk;
                            nrec++;
                            cur = cur + vk;
                        } else {
                            err |= kErrSolutionOverflow;
                        }
                    }
                    pend &= pend - 1u;
                    __syncwarp();
                }
            }
            acc = kRough ? acc + cur * (1.f / p_off) : acc + cur;
            n_unique += nrec;
            cpos = wpos + kWalk * (uint64_t)M;
        }
        if (live && gl == 0) {
            value[qi] = acc.x;
            value[(size_t)n + qi] = acc.y;
            value[2 * (size_t)n + qi] = acc.z;
            count[qi] = n_unique;
            walks[qi] = work ? M * sc.n_casters_ss : 0;
        }
    }
    flush_stats(st, ctr, err, kPhaseSsBiased);
}

// --------------------------------------------------- unbiased: first walks
// kLearned: seeds come from the query's learned mixture (three draws per walk,
// mlp::proposal_seed, mixture from ss_proposal_kernel) instead of two-draw
// uniform seeding.
template <bool kLearned, int kVar>
__global__ void __launch_bounds__(128, ss_walk_blocks(kVar)) ss_first_kernel(DevScene sc, SolverCfg cfg, int c, const float *__restrict__ qs,
                                                       uint32_t n, uint64_t seed, uint64_t stream_off,
                                                       float *__restrict__ value, int *__restrict__ count,
                                                       int *__restrict__ walks, SsScratch scr, DevCounters *ctr,
                                                       mlp::SeedProposal pr, int lanes) {
    constexpr bool kRough = (kVar & 1) != 0, kTwo = (kVar & 2) != 0, kNM = (kVar & 4) != 0;
    const unsigned lane = threadIdx.x & 31;
    const uint32_t qi = (blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * (uint32_t)lanes + lane;
    const bool active = (int)lane < lanes && qi < n;
    LaneStats st;
    uint32_t err = 0;
    bool enqueue = false;
    Query Q;
    Pcg32 rng;
    Light L;
    bool have_light = false;
    if (active) {
        Q = load_query(qs, n, qi);
        rng = query_rng(seed, query_stream(cfg, stream_off, qi), 0);
        have_light = sample_emitter(sc, sc.emitters_ss, sc.n_emitters_ss, rng, Q.x, L);
    }
    if (active) {
        uint32_t pos = 3u;
        f3 acc = splat(0.f);
        int nw = 0;
        if (c == 0) {
            if (have_light) st.conns++;
        } else {
            pos = scr.pos[qi];
            acc = mk(value[qi], value[(size_t)n + qi], value[2 * (size_t)n + qi]);
            nw = walks[qi];
        }
        if (have_light) {
            const int caster = sc.casters_ss[c];
            rng.advance(pos - 3u);
            float p_off = 1.f;
            f3 no = mk(0.f, 0.f, 1.f);
            if (kRough) {
                no = caster_offset(sc.shapes[caster], rng, p_off);
                pos += caster_draws(sc.shapes[caster]);
            }
            f3 sp;
            if constexpr (kLearned) {
                const float us = rng.next_f32(), sx = rng.next_f32(), sy = rng.next_f32();
                pos += 3u;
                sp = mlp::proposal_seed(sc, pr, sc.shapes[caster], pr.gmm + qi, n, us, sx, sy);
            } else {
                const float sx = rng.next_f32(), sy = rng.next_f32();
                pos += 2u;
                sp = sample_position(sc, sc.shapes[caster], sx, sy);
            }
            float g0 = 0.f, g1 = 0.f;
            if (kTwo) {
                g0 = rng.next_f32();
                g1 = rng.next_f32();
                pos += 2u;
            }
            Vtx v;
            int it;
            bool ok = ss_walk<kRough, kTwo, kNM>(sc, cfg, caster, Q.x, L.p, sp, v, it, err, st, nullptr, no, g0, g1);
            st.walks++;
            st.newton += (unsigned)it;
            nw++;
            if (ok) {
                st.succ++;
                if (visible(sc, L.p, v.p, err, st)) {
                    f3 dir = normalize(v.p - Q.x);
                    f3 spec = contribution<kNM>(sc, Q.x, L, v, err, st);
                    // the caster's estimate is divided by the offset density (manifold_ss.cpp:199)
                    f3 val = kRough ? receiver_eval(sc, Q, dir, err) * spec * (1.f / p_off) : receiver_eval(sc, Q, dir, err) * spec;
                    scr.dir0[qi] = dir.x; scr.dir0[(size_t)n + qi] = dir.y; scr.dir0[2 * (size_t)n + qi] = dir.z;
                    scr.val[qi] = val.x; scr.val[(size_t)n + qi] = val.y; scr.val[2 * (size_t)n + qi] = val.z;
                    enqueue = true;
                }
            } else {
                st.fail++;
            }
        }
        scr.pos[qi] = pos;
        value[qi] = acc.x;
        value[(size_t)n + qi] = acc.y;
        value[2 * (size_t)n + qi] = acc.z;
        count[qi] = enqueue ? kTrialOpen : 0;
        walks[qi] = nw;
    }
    // warp-aggregated append to the trial queue
    unsigned want = __ballot_sync(0xffffffffu, enqueue);
    if (want) {
        unsigned leader = __ffs(want) - 1;
        unsigned base = 0;
        if (lane == leader) base = atomicAdd(&ctr->trial_count, (unsigned)__popc(want));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (enqueue) scr.list[base + __popc(want & ((1u << lane) - 1u))] = qi;
    }
    flush_stats(st, ctr, err, kPhaseSsFirst);
}

// ------------------------------------------------ unbiased: Bernoulli trials
// For query q with first-walk direction dir0 the trials are t = 1, 2, ...;
// trial t draws stream positions pos + S(t-1) .. (S = 2 draws per walk, 3 with
// a learned proposal), so the smallest successful t is exactly the reference's
// sequential trial count (manifold_ss.cpp:115-135), whichever trials ran side
// by side.  Every trial redraws its seed from the same per-query proposal as
// the first walk, so the count still estimates the inverse probability of
// reaching dir0.  One lane per trial, drawn from the stream of sms_trials.cuh.
template <bool kLearned, int kVar, bool kTree = false>
__global__ void __launch_bounds__(128, ss_walk_blocks(kVar)) ss_trials_kernel(DevScene sc, SolverCfg cfg, int c, const float *__restrict__ qs,
                                                        uint32_t n, uint64_t seed, uint64_t stream_off,
                                                        int *__restrict__ count, SsScratch scr, DevCounters *ctr,
                                                        mlp::SeedProposal pr, int pass, TrialRule rule) {
    constexpr bool kRough = (kVar & 1) != 0, kTwo = (kVar & 2) != 0, kNM = (kVar & 4) != 0;
    const int cap = cfg.max_trials > 0 ? cfg.max_trials : kTrialHardLimit;
    TrialStream ts(*(volatile unsigned *)&ctr->trial_count, cap, pass, 32, rule);
    if (ts.total == 0) return;
    if (kTree) tree_smem_fill(sc);
    __shared__ TrialBuffer bufs[4];
    TrialBuffer &buf = bufs[threadIdx.x >> 5];
    constexpr uint32_t kStride = (kLearned ? 3u : 2u) + (kTwo ? 2u : 0u);   // numbers per walk
    LaneStats st;
    uint32_t err = 0;
    const int caster = sc.casters_ss[c];
    while (true) {
        uint32_t qi;
        int t;
        const bool have = ts.next(buf, scr.list, count, ctr, pass, cfg.queue_chunk, ts.plan.lanes, (int)(threadIdx.x & 31),
                                  qi, t);
        if (!__any_sync(0xffffffffu, have)) break;
        if (have) {
            const Query Q = load_query(qs, n, qi);
            Pcg32 rng = query_rng(seed, query_stream(cfg, stream_off, qi), 0);
            Light L;
            sample_emitter(sc, sc.emitters_ss, sc.n_emitters_ss, rng, Q.x, L);   // rng sits at position 3
            const uint32_t pos = scr.pos[qi];
            f3 no = mk(0.f, 0.f, 1.f);
            if (kRough) {
                // the offset normal drawn before the first walk
                Pcg32 r0 = rng;
                r0.advance((uint64_t)(pos - 3u - kStride - 2u));
                float p_off;
                no = caster_offset(sc.shapes[caster], r0, p_off);
            }
            rng.advance((uint64_t)(pos - 3u) + kStride * (uint64_t)(t - 1));
            f3 sp;
            if constexpr (kLearned) {
                const float us = rng.next_f32(), sx = rng.next_f32(), sy = rng.next_f32();
                sp = mlp::proposal_seed(sc, pr, sc.shapes[caster], pr.gmm + qi, n, us, sx, sy);
            } else {
                const float sx = rng.next_f32(), sy = rng.next_f32();
                sp = sample_position(sc, sc.shapes[caster], sx, sy);
            }
            float g0 = 0.f, g1 = 0.f;
            if (kTwo) { g0 = rng.next_f32(); g1 = rng.next_f32(); }
            Vtx v;
            int it;
            bool succ = ss_walk<kRough, kTwo, kNM, kTree>(sc, cfg, caster, Q.x, L.p, sp, v, it, err, st, nullptr, no,
                                                          g0, g1);
            if (succ) {
                const f3 dir0 = mk(scr.dir0[qi], scr.dir0[(size_t)n + qi], scr.dir0[2 * (size_t)n + qi]);
                succ = fabsf(dot(dir0, normalize(v.p - Q.x)) - 1.f) < cfg.uniqueness_threshold;
            }
            trial_end(count, ctr, qi, t, succ, it, st);
        }
    }
    flush_stats(st, ctr, err, kPhaseSsTrials);
}

// ------------------------------------------------- per-variant launchers
template <int kVar>
cudaError_t ss_biased_launch(const DevScene &sc, const SolverCfg &cfg, const float *q, uint32_t n, uint64_t seed,
                             uint64_t stream_off, float *value, int *count, int *walks, DevCounters *ctr,
                             int num_sms, int bps, PhaseTimer *tm, cudaStream_t s) {
    const int G = cfg.max_trials <= 16 ? 16 : 32;
    const uint32_t groups_per_block = 128 / G;
    uint32_t blocks_needed = (n + groups_per_block - 1) / groups_per_block;
    uint32_t blocks = std::min<uint32_t>(blocks_needed, (uint32_t)(num_sms * bps));
    phase_begin(tm, kPhaseSsBiased, s);
    constexpr int kMany = ss_biased_blocks(kVar);
    const bool many = kMany > 4 && blocks_needed > ss_biased_large(kVar) * (uint32_t)num_sms;
    auto biased = G == 16 ? (many ? ss_biased_kernel<16, kVar, kMany> : ss_biased_kernel<16, kVar, 4>)
                          : (many ? ss_biased_kernel<32, kVar, kMany> : ss_biased_kernel<32, kVar, 4>);
    biased<<<blocks, 128, 0, s>>>(sc, cfg, q, n, seed, stream_off, value, count, walks, ctr);
    phase_end(tm, s);
    return cudaGetLastError();
}

// First walks and Bernoulli trials of caster c (kLearnedOk: a learned
// proposal may seed it).
template <int kVar, bool kLearnedOk>
cudaError_t ss_caster_launch(const DevScene &sc, const SolverCfg &cfg, int c, const float *q, uint32_t n,
                             uint64_t seed, uint64_t stream_off, float *value, int *count, int *walks,
                             DevCounters *ctr, const SsScratch &scr, int num_sms, int bps, PhaseTimer *tm,
                             cudaStream_t s, const mlp::SeedProposal *prop, uint32_t treelet = 0) {
    const bool learned = kLearnedOk && prop && prop->shape == sc.casters_ss[c];
    // the trial kernel holds the top `treelet` node records in shared memory
    // (plain and rough casters)
    DevScene st = sc;
    st.n_tnodes = (kVar & 4) ? 0u : std::min<uint32_t>(treelet, sc.n_nodes);
    const size_t tsmem = (size_t)st.n_tnodes * 4 * sizeof(float4);
    const mlp::SeedProposal pr = learned ? *prop : mlp::SeedProposal{};
    phase_begin(tm, kPhaseSsFirst, s);
    cudaError_t e = cudaSuccess;
    const int lanes = first_walk_lanes(n, num_sms);
    const uint32_t fblocks = first_walk_blocks(n, lanes);
    if constexpr (kLearnedOk) {
        if (learned) {
            e = launch_ss_proposal(sc, cfg, q, n, seed, stream_off, pr, num_sms, s);
            if (e != cudaSuccess) return e;
            ss_first_kernel<true, kVar><<<fblocks, 128, 0, s>>>(sc, cfg, c, q, n, seed, stream_off, value, count,
                                                                walks, scr, ctr, pr, lanes);
        }
    }
    if (!learned)
        ss_first_kernel<false, kVar><<<fblocks, 128, 0, s>>>(sc, cfg, c, q, n, seed, stream_off, value, count, walks,
                                                             scr, ctr, pr, lanes);
    phase_end(tm, s);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    phase_begin(tm, kPhaseSsTrials, s);
    auto trials = ss_trials_kernel<false, kVar>;
    if constexpr ((kVar & 4) == 0) {   // the treelet serves the plain and rough casters
        if (st.n_tnodes) trials = ss_trials_kernel<false, kVar, true>;
    }
    if constexpr (kLearnedOk) {
        if (learned) trials = ss_trials_kernel<true, kVar>;
        if constexpr ((kVar & 4) == 0) {
            if (learned && st.n_tnodes) trials = ss_trials_kernel<true, kVar, true>;
        }
    }
    const int tblocks = num_sms * (bps > 0 ? bps : ss_walk_blocks(kVar));
    const int cap = cfg.max_trials > 0 ? cfg.max_trials : kTrialHardLimit;
    TrialRule rule;
    // (the two-stage solver draws a slope for every walk: not deterministic)
    rule.split = (kVar & 2) ? kSplitLong : cfg.mnee_init ? kSplitAlways : kSplitNever;
    rule.claim_by_row = true;
    rule.warps = sc.n_tris <= kSmallTree ? kSmallTreeWarps * num_sms : 0;
    rule.even_end = true;
    for (int pass = trial_split_possible(rule, n, cap, tblocks) ? 0 : 1; pass < 2; ++pass)
        trials<<<tblocks, 128, tsmem, s>>>(st, cfg, c, q, n, seed, stream_off, count, scr, ctr, pr, pass, rule);
    const uint32_t stride = (learned ? 3u : 2u) + ((kVar & 2) ? 2u : 0u);
    trials_finish_kernel<<<finish_blocks(n, num_sms), 128, 0, s>>>(n, value, count, walks, scr, nullptr, cap,
                                                                   cfg.max_trials <= 0, stride, kPhaseSsTrials, ctr);
    phase_end(tm, s);
    return cudaGetLastError();
}

}  // namespace sms
