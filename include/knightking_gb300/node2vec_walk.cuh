/*
 * node2vec walks over the edge set (src/apps/node2vec.hpp:108-197): the draws,
 * decisions and paths of walk_trial() with the node2vec hooks, laid out for
 * the wait that bounds them.
 *
 * A trial reads a bucket (or neighbour), then for about half the trials the
 * edge set (whether the candidate is a neighbour of the previous vertex), and
 * a step with the return-edge outlier reads that edge's slot first: two or
 * three dependent waits of DRAM latency (2.0 us a step for one warp on a graph
 * of 32 M edges with no question asked), and a warp pays each of them whenever
 * one of its lanes needs it.  Here a pass of the loop has one wait: every lane
 * issues the edge-set read its pending question needs and the pick its next
 * trial needs, then both are used.  With q > 1 a lane with a question pending
 * issues the pick of the trial that follows if the answer is no, which is what
 * most answers are then; with q <= 1 an answer seldom rejects, and nothing is
 * read that may not be used.  A step whose bound is still to be read issues
 * its pick beside it, at the draw the pick has when the bound is positive.
 * The previous vertex's row of the edge set is kept with it, so a question is
 * one read.  Against walk_trial()'s loop over a table of (u, v) keys in 64 B
 * buckets (same box): R-MAT 16, 65,536 walkers, p 2, q 0.5 353 -> 250 us;
 * R-MAT 19, 300,007 walkers, p 0.25, q 3 1558 -> 1330 us; R-MAT 22, 2.4 M
 * walkers, p 2, q 0.5 8.42 -> 7.45 ms; 20 jobs on 32 M edges 2.73 -> 2.30 ms.
 */
#pragma once

#include "apps.cuh"

namespace kk
{

/* A job's constants (Node2vecConstants, and min(1, 1/q) below which a dart is
 * accepted whatever the adjacency). */
struct N2vParams
{
    float upperbound, lowerbound, overflow, inv_p, inv_q, sure_below;
    step_t walk_length;
};

/* What every walk of the launch reads. */
template <typename Bucket>
struct N2vTables
{
    const Bucket *alias; /* weighted */
    const float *sum;    /* the alias tables' sums */
    const float *ra;     /* regular_area per vertex, or nullptr */
    EdgeSetView set;
};

/* Walks run (just begun: start vertex, path slot) to its end. */
template <bool Weighted, bool Outlier, typename Bucket>
__device__ __forceinline__ void n2v_walk(const GraphView &g, const N2vTables<Bucket> &t, const N2vParams &P,
                                         const WalkLaunch &L, unsigned team,
                                         WalkerRun<apps::Node2vecState> &run, Sampler &rng)
{
    const uint32_t id = run.w.id;
    uint32_t step = 0, prev = 0, v = run.v, trials = 0;
    Pos pos = pos_from_offsets(g, v);
    float rav = 0.0f; /* regular_area of v */
    /* the step's outlier area, once its return edge is known (find: not yet),
     * and that edge: its weight, and its index unless it leads to prev */
    bool find = false;
    float ob = 0.0f, back_w = 0.0f;
    uint32_t back_i = kNone;
    /* prev's row of the edge set, and the sector to read next, in it (query)
     * or in v's (find) */
    uint64_t prow = 0;
    uint32_t pn = 1, sec = 0;
    /* the pending question: is cand a neighbour of prev, and its dart */
    bool query = false;
    Cand cand{kNone, 0, 0, false};
    float dart = 0.0f;
    /* q > 1: most candidates are no neighbours, and a no rejects */
    const bool ahead = P.inv_q < 1.0f;
    auto begin_step = [&]() {
        rng.enter(id, step, 0);
        trials = 0;
        if constexpr (Outlier)
        {
            const bool on = P.overflow > 0.0f;
            find = Weighted && on;
            ob = Weighted ? 0.0f : P.overflow;
            back_i = kNone;
            sec = kNone; /* find's first sector follows from the position */
            if (on)
            {
                if (t.ra != nullptr)
                    rav = gather(t.ra + v);
                else if constexpr (Weighted)
                    rav = gather(t.sum + v);
            }
        }
    };
    begin_step();
    /* one way through the loop, and the warp's lanes (team) meet at its top:
     * they share the instructions of every pass */
    bool alive = P.walk_length > 0;
    while (__any_sync(team, alive))
    {
        if (alive)
        {
            /* the question's edge-set read; while it is on its way, the next
             * trial's words, then (the position of a step just begun is there by
             * now) the return edge's read and the pick's.  A previous vertex 0 is
             * at or below every neighbour: position 0, no lookup. */
            const bool asked = query;
            const bool look = asked || (Outlier && find && prev != 0);
            uint4 k0, k1, w0, w1;
            if (asked)
            {
                const uint4 *b = reinterpret_cast<const uint4 *>(t.set.keys + (prow + sec) * kEdgeSetSlots);
                k0 = __ldg(b);
                k1 = __ldg(b + 1);
            }
            uint4 nxt = make_uint4(0u, 0u, 0u, 0u), wd = nxt, lo = nxt, hi = nxt;
            bool app = false, trial = !asked || ahead;
            auto load = [&](uint32_t at) {
                if constexpr (Weighted)
                {
                    const uint4 *b = reinterpret_cast<const uint4 *>(t.alias + pos.e0 + at);
                    lo = gather(b);
                    if constexpr (!Bucket::compact)
                        hi = gather(b + 1);
                }
                else if (g.adjc != nullptr)
                {
                    lo = gather(g.adjc + pos.e0 + at);
                }
                else
                {
                    lo.x = gather(g.nbr + pos.e0 + at);
                }
            };
            if (trial)
            {
                wd = rng.quad(nxt);
                alive = pos.deg != 0; /* a vertex without edges ends the walk as its step begins */
                trial = alive;
                app = Outlier && (find || ob > 0.0f);
                if (alive)
                {
                    if (Outlier && Weighted && look && !asked)
                    {
                        if (sec == kNone)
                            sec = edge_set_sector(prev, edge_set_sectors(pos.deg));
                        const uint64_t at = (edge_set_row(pos.e0, v) + sec) * kEdgeSetSlots;
                        const uint4 *b = reinterpret_cast<const uint4 *>(t.set.keys + at);
                        const uint4 *bw = reinterpret_cast<const uint4 *>(t.set.w + at);
                        k0 = __ldg(b);
                        k1 = __ldg(b + 1);
                        w0 = __ldg(bw);
                        w1 = __ldg(bw + 1);
                    }
                    load(map_gen(app ? wd.y : wd.x, pos.deg));
                }
            }
            bool taken = false;
            if (look && alive)
            {
                const uint32_t m = edge_set_match(k0, k1, asked ? cand.nbr : prev);
                if (m == 9)
                {
                    /* undecided: the next sector, next time */
                    sec = sec + 1 == (asked ? pn : edge_set_sectors(pos.deg)) ? 0 : sec + 1;
                    trial = false;
                }
                else if (asked)
                {
                    query = false;
                    taken = dart <= (m < 8 ? 1.0f : P.inv_q);
                    trial = trial && !taken;
                }
                else if constexpr (Outlier && Weighted)
                {
                    const float wl = m & 1 ? (m & 2 ? __uint_as_float(w0.w) : __uint_as_float(w0.y))
                                           : (m & 2 ? __uint_as_float(w0.z) : __uint_as_float(w0.x));
                    const float wh = m & 1 ? (m & 2 ? __uint_as_float(w1.w) : __uint_as_float(w1.y))
                                           : (m & 2 ? __uint_as_float(w1.z) : __uint_as_float(w1.x));
                    back_w = m & 4 ? wh : wl;
                    bool edge = m < 8;
                    if (!edge)
                    {
                        /* directed graphs: std::lower_bound's edge, if any */
                        back_i = apps::lower_bound_adj(g.nbr, (edge_id_t)pos.e0, pos.deg, prev);
                        edge = back_i < pos.deg;
                        if (edge)
                            back_w = gather(g.w + pos.e0 + back_i);
                    }
                    ob = edge ? fmul(back_w, P.overflow) : 0.0f;
                    find = false;
                }
            }
            else if (Outlier && find && alive)
            {
                back_i = 0;
                back_w = gather(g.w + pos.e0);
                ob = fmul(back_w, P.overflow);
                find = false;
            }
            if (trial)
            {
                bool in_app = false, some = true;
                uint32_t drawn = 0;
                if constexpr (Outlier)
                {
                    if (ob > 0.0f)
                    {
                        float area = rav;
                        if (t.ra == nullptr)
                            area = fmul(Weighted ? rav : u2f(pos.deg), P.upperbound);
                        const float r = fsub(map_gen_float(wd.x, fadd(fmul(ob, u2f(1u)), area)), area);
                        wd = make_uint4(wd.y, wd.z, wd.w, 0u);
                        drawn = 1;
                        if (r > 0.0f)
                        {
                            /* the appendix: the return edge (src/apps/node2vec.hpp:85-102) */
                            in_app = true;
                            uint32_t oi = (uint32_t)fdiv(r, ob);
                            if (oi + 1 > 1)
                                oi = 0;
                            float sc = 1.0f;
                            uint32_t at = back_i;
                            if constexpr (Weighted)
                            {
                                sc = back_w; /* a positive area comes with its edge */
                            }
                            else
                            {
                                at = prev == 0 ? 0 : apps::lower_bound_adj(g.nbr, (edge_id_t)pos.e0, pos.deg, prev);
                                some = at < pos.deg; /* none: the retry within the superstep */
                            }
                            cand = Cand{kNone, Weighted && at == kNone ? prev : some ? gather(g.nbr + pos.e0 + at) : 0, 0,
                                        false, 0};
                            dart = fadd(fdiv(fsub(r, fmul(u2f(oi), ob)), sc), P.upperbound);
                        }
                    }
                }
                if (!in_app)
                {
                    if (Outlier && app != (drawn != 0))
                        load(map_gen(wd.x, pos.deg)); /* the bound came out the other way */
                    if constexpr (Weighted)
                    {
                        const bool coin = lo.z != kNone;
                        const bool first = !coin || map_gen_float(wd.y, 1.0f) < __uint_as_float(lo.x);
                        if constexpr (Bucket::compact)
                            cand = Cand{kNone, first ? lo.y : lo.z, 0, false, 0};
                        else if constexpr (Bucket::cursor)
                            cand = Cand{kNone, first ? lo.y : lo.z,
                                        first ? ((uint64_t)hi.y << 32) | hi.x : ((uint64_t)hi.w << 32) | hi.z, true, 0};
                        else
                            cand = Cand{kNone, first ? hi.x : hi.y, 0, false, 0};
                        dart = map_gen_float(coin ? wd.z : wd.y, P.upperbound);
                        drawn += coin ? 3u : 2u;
                    }
                    else
                    {
                        cand = Cand{kNone, lo.x, g.adjc != nullptr ? ((uint64_t)lo.w << 32) | lo.z : 0, g.adjc != nullptr,
                                    0};
                        dart = map_gen_float(wd.y, P.upperbound);
                        drawn += 2u;
                    }
                    taken = dart <= P.lowerbound;
                }
                rng.take(drawn, nxt);
                const bool back = prev == cand.nbr;
                if (!taken && some && step != 0 && !back && !(dart <= P.sure_below))
                {
                    query = true;
                    run.queries++;
                    sec = edge_set_sector(cand.nbr, pn);
                }
                else if (!taken && some)
                {
                    taken = dart <= (step == 0 ? P.upperbound : back ? P.inv_p : P.inv_q);
                }
                if (++trials > L.trial_limit)
                {
                    /* this trial was one too many */
                    atomicOr(L.status, KK_STATUS_TRIAL_LIMIT);
                    run.trials += trials;
                    alive = taken = false;
                }
            }
            if (taken)
            {
                run.trials += trials;
                step++;
                prow = edge_set_row(pos.e0, v);
                pn = edge_set_sectors(pos.deg);
                prev = v;
                v = cand.nbr;
                if (run.out != nullptr)
                    run.out[step] = v;
                pos = cand.has_cur ? pos_from_cursor(g, v, cand.cur) : pos_from_offsets(g, v);
                begin_step();
                alive = step < P.walk_length;
            }
        }
    }
    run.len = step + 1;
}

/* One thread per walker for its whole walk. */
template <bool Weighted, bool Outlier, typename Bucket>
__global__ void __launch_bounds__(256, 4) n2v_walk_kernel(GraphView g, N2vTables<Bucket> t, N2vParams P, WalkLaunch L)
{
    unsigned long long my_steps = 0;
    WalkCounts counts;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned team = __ballot_sync(kFullMask, i < L.walker_num);
    if (i < L.walker_num)
    {
        Sampler rng;
        rng.init(L.seed);
        WalkerRun<apps::Node2vecState> run;
        WalkerConfig<apps::Node2vecState> wc;
        walk_begin<apps::Node2vecState>(g, wc, L, i, run, rng);
        n2v_walk<Weighted, Outlier, Bucket>(g, t, P, L, team, run, rng);
        walk_finish<apps::Node2vecState>(L, i, run, my_steps, counts);
    }
    flush_steps(L.total_steps, my_steps);
    counts.flush(L.stats);
}

/* Whether a transition is node2vec's, with its outlier or without. */
template <typename TC, typename = void>
struct is_node2vec
{
    static constexpr bool value = false;
};
template <typename TC>
struct is_node2vec<TC, std::enable_if_t<std::is_same<decltype(TC::dynamic_comp), apps::Node2vecDyn>::value>>
{
    static constexpr bool value = true;
};

template <typename TC>
N2vParams n2v_params(const TC &tc)
{
    N2vParams P;
    P.upperbound = tc.dcomp_upperbound.value;
    P.lowerbound = tc.dcomp_lowerbound.value;
    P.overflow = 0.0f;
    if constexpr (TC::has_outlier)
        P.overflow = tc.outlier_upperbound.overflow;
    P.inv_p = tc.dynamic_comp.inv_p;
    P.inv_q = tc.dynamic_comp.inv_q;
    P.sure_below = tc.post_query.sure_below;
    P.walk_length = tc.extension_comp.walk_length;
    return P;
}

/* The batch kernel (walk_batch_kernel) of node2vec jobs over the edge set.  A
 * warp may hold walkers of several jobs: the lanes of its last pass over the
 * walkers are its team. */
template <bool Weighted, typename Bucket>
__global__ void __launch_bounds__(256, KK_BATCH_MINB)
    n2v_batch_kernel(GraphView g, apps::Node2vecBatch<Weighted> app, N2vTables<Bucket> t, const BatchJob *jobs,
                     uint32_t njobs, uint32_t total, uint32_t *path, uint32_t *length,
                     unsigned long long *total_steps, int *status, uint32_t trial_limit, unsigned long long *stats,
                     const uint32_t *hdr, BatchNotify nt)
{
    __shared__ uint32_t s_first[2 * kMaxBatchJobs];
    if (hdr != nullptr)
    {
        /* counts from device memory: one captured launch serves every batch */
        njobs = hdr[0];
        total = hdr[1];
    }
    for (uint32_t j = threadIdx.x; j < njobs; j += blockDim.x)
    {
        s_first[j] = jobs[j].launch_first;
        s_first[kMaxBatchJobs + j] = jobs[j].launch_job;
    }
    __syncthreads();
    unsigned long long my_steps = 0;
    WalkCounts counts;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += stride)
    {
        const unsigned team = __activemask();
        typename apps::Node2vecBatch<Weighted>::WC wc;
        typename apps::Node2vecBatch<Weighted>::TC tc;
        WalkLaunch L;
        WalkerRun<apps::Node2vecState> run;
        Sampler rng;
        const uint32_t i = batch_walker_begin<apps::Node2vecState>(g, app, jobs, s_first, njobs, (uint32_t)at, t.sum,
                                                                  path, length, total_steps, status, trial_limit, wc,
                                                                  tc, L, run, rng, nt);
        N2vParams P;
        P.upperbound = tc.dcomp_upperbound.value;
        P.lowerbound = tc.dcomp_lowerbound.value;
        P.overflow = tc.outlier_upperbound.overflow;
        P.inv_p = tc.dynamic_comp.inv_p;
        P.inv_q = tc.dynamic_comp.inv_q;
        P.sure_below = tc.post_query.sure_below;
        P.walk_length = tc.extension_comp.walk_length;
        n2v_walk<Weighted, true, Bucket>(g, t, P, L, team, run, rng);
        L.length[i] = run.len;
        segment_done(L, i);
        my_steps += run.len - 1;
        counts.add(run);
    }
    flush_steps(total_steps, my_steps);
    counts.flush(stats);
}

} // namespace kk
