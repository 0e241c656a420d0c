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
 * buckets (same box): R-MAT 16, 65,536 walkers, p 2, q 0.5 355 -> 263 us;
 * R-MAT 19, 300,007 walkers, p 0.25, q 3 1550 -> 1170 us; R-MAT 22, 2.4 M
 * walkers, p 2, q 0.5 8.36 -> 7.85 ms; 20 jobs on 32 M edges 2.73 -> 1.55 ms.
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

/* Walks walker id from v to its end (the 32-bit offsets at hand), its path to
 * out (vertex 0 on, with room for cap vertices; or nullptr); the path's length
 * in len.  team: the warp's lanes that call this together.  Returns status
 * flags: a step passed the trial limit, or the path's room.  The start's slot
 * need not fit the walk (one vertex for a start outside the graph, whose walker
 * stands on vertex 0 until the host refuses the call). */
template <bool Weighted, bool Outlier, typename Bucket>
__device__ __forceinline__ int n2v_walk(const GraphView &g, const N2vTables<Bucket> &t, const N2vParams &P,
                                        walker_id_t id, vertex_id_t v, uint32_t *out, uint32_t cap,
                                        uint32_t trial_limit, unsigned long long *stats, unsigned team, Sampler &rng,
                                        uint32_t &len)
{
    uint32_t step = 0, prev = 0, trials = 0;
    int status = KK_STATUS_OK;
    /* v's adjacency as read, its first edge and the one past its last: what
     * follows from them is computed where it is used, or the walk would wait
     * for them here */
    uint32_t pb = gather(g.off32 + v), pe = gather(g.off32 + v + 1);
    float rav = 0.0f; /* regular_area of v */
    /* the step's outlier area, once its return edge is known (find: not yet),
     * and that edge: its weight, and its index unless it leads to prev */
    bool find = false;
    float ob = 0.0f, back_w = 0.0f;
    uint32_t back_i = kNone;
    /* prev's row of the edge set, and the sector to read next, in it (query)
     * or in v's (find) */
    uint32_t prow = 0, pn = 1, sec = 0;
    /* the pending question: is cand a neighbour of prev, and its dart */
    bool query = false;
    vertex_id_t cand = 0;
    uint64_t cand_cur = 0;
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
    const step_t last = path_steps(out, cap, P.walk_length);
    /* one way through the loop, and the warp's lanes (team) meet at its top:
     * they share the instructions of every pass */
    bool alive = last > 0;
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
            uint4 k0, k1; /* a sector: ids, and more ids or weights */
            if (asked)
            {
                const uint4 *b =
                    reinterpret_cast<const uint4 *>(t.set.keys + (uint64_t)(prow + sec) * kEdgeSectorWords);
                k0 = __ldg(b);
                if (!Weighted)
                    k1 = __ldg(b + 1);
            }
            uint4 nxt = make_uint4(0u, 0u, 0u, 0u), wd = nxt, lo = nxt, hi = nxt;
            bool app = false, trial = !asked || ahead;
            auto load = [&](uint32_t at) {
                if constexpr (Weighted)
                {
                    const uint4 *b = reinterpret_cast<const uint4 *>(t.alias + pb + at);
                    lo = gather(b);
                    if constexpr (!Bucket::compact)
                        hi = gather(b + 1);
                }
                else if (g.adjc != nullptr)
                {
                    lo = gather(g.adjc + pb + at);
                }
                else
                {
                    lo.x = gather(g.nbr + pb + at);
                }
            };
            if (trial)
            {
                wd = rng.quad(nxt);
                alive = pe != pb; /* a vertex without edges ends the walk as its step begins */
                trial = alive;
                app = Outlier && (find || ob > 0.0f);
                if (alive)
                {
                    if (Outlier && Weighted && look && !asked)
                    {
                        if (sec == kNone)
                            sec = edge_set_sector(prev, edge_set_sectors(pe - pb, t.set.shift));
                        const uint4 *b = reinterpret_cast<const uint4 *>(
                            t.set.keys + (edge_set_row(pb, v, t.set.shift) + sec) * kEdgeSectorWords);
                        k0 = __ldg(b);
                        k1 = __ldg(b + 1);
                    }
                    load(map_gen(app ? wd.y : wd.x, pe - pb));
                }
            }
            bool taken = false;
            if (look && alive)
            {
                const vertex_id_t x = asked ? cand : prev;
                /* a weighted walk's set is weighted; an unweighted walk's may be too */
                const uint32_t m = Weighted ? edge_set_match(k0, x) : edge_set_match(t.set, k0, k1, x);
                if (m == 9)
                {
                    /* undecided: the next sector, next time */
                    sec = sec + 1 == (asked ? pn : edge_set_sectors(pe - pb, t.set.shift)) ? 0 : sec + 1;
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
                    back_w = __uint_as_float(word_of(k1, m));
                    bool edge = m < 8;
                    if (!edge)
                    {
                        /* directed graphs: std::lower_bound's edge, if any */
                        back_i = apps::lower_bound_adj(g.nbr, pb, pe - pb, prev);
                        edge = back_i < pe - pb;
                        if (edge)
                            back_w = gather(g.w + pb + back_i);
                    }
                    ob = edge ? fmul(back_w, P.overflow) : 0.0f;
                    find = false;
                }
            }
            else if (Outlier && find && alive)
            {
                back_i = 0;
                back_w = gather(g.w + pb);
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
                            area = fmul(Weighted ? rav : u2f(pe - pb), P.upperbound);
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
                                at = prev == 0 ? 0 : apps::lower_bound_adj(g.nbr, pb, pe - pb, prev);
                                some = at < pe - pb; /* none: the retry within the superstep */
                            }
                            cand = Weighted && at == kNone ? prev : some ? gather(g.nbr + pb + at) : 0;
                            cand_cur = ~0ull;
                            dart = fadd(fdiv(fsub(r, fmul(u2f(oi), ob)), sc), P.upperbound);
                        }
                    }
                }
                if (!in_app)
                {
                    if (Outlier && app != (drawn != 0))
                        load(map_gen(wd.x, pe - pb)); /* the bound came out the other way */
                    if constexpr (Weighted)
                    {
                        const bool coin = lo.z != kNone;
                        const bool first = !coin || map_gen_float(wd.y, 1.0f) < __uint_as_float(lo.x);
                        if constexpr (Bucket::compact || Bucket::cursor)
                            cand = first ? lo.y : lo.z;
                        else
                            cand = first ? hi.x : hi.y;
                        if constexpr (Bucket::cursor)
                            cand_cur = first ? ((uint64_t)hi.y << 32) | hi.x : ((uint64_t)hi.w << 32) | hi.z;
                        dart = map_gen_float(coin ? wd.z : wd.y, P.upperbound);
                        drawn += coin ? 3u : 2u;
                    }
                    else
                    {
                        cand = lo.x;
                        if (g.adjc != nullptr)
                            cand_cur = ((uint64_t)lo.w << 32) | lo.z;
                        dart = map_gen_float(wd.y, P.upperbound);
                        drawn += 2u;
                    }
                    taken = dart <= P.lowerbound;
                }
                rng.take(drawn, nxt);
                const bool back = prev == cand;
                if (!taken && some && step != 0 && !back && !(dart <= P.sure_below))
                {
                    query = true;
                    if (stats != nullptr)
                        atomicAdd(stats + 1, 1ull);
                    sec = edge_set_sector(cand, pn);
                }
                else if (!taken && some)
                {
                    taken = dart <= (step == 0 ? P.upperbound : back ? P.inv_p : P.inv_q);
                }
                if (stats != nullptr)
                    atomicAdd(stats, 1ull);
                if (++trials > trial_limit)
                {
                    /* this trial was one too many */
                    alive = taken = false;
                    status = KK_STATUS_TRIAL_LIMIT;
                }
            }
            if (taken)
            {
                step++;
                prow = (uint32_t)edge_set_row(pb, v, t.set.shift);
                pn = edge_set_sectors(pe - pb, t.set.shift);
                prev = v;
                v = cand;
                if (out != nullptr)
                    out[step] = v;
                bool cursor = false;
                if constexpr (Weighted)
                    cursor = Bucket::cursor && cand_cur != ~0ull;
                else
                    cursor = g.adjc != nullptr && cand_cur != ~0ull;
                if (cursor)
                {
                    const Pos np = pos_from_cursor(g, v, cand_cur);
                    pb = (uint32_t)np.e0;
                    pe = pb + np.deg;
                }
                else
                {
                    pb = gather(g.off32 + v);
                    pe = gather(g.off32 + v + 1);
                }
                begin_step();
                alive = step < last;
            }
        }
    }
    len = step + 1;
    if (step == last && last < P.walk_length && pe != pb && status == KK_STATUS_OK)
        status = KK_STATUS_PATH_CAPACITY; /* another step was due */
    return status;
}

/* One thread per walker for its whole walk. */
template <bool Weighted, bool Outlier, typename Bucket>
__global__ void __launch_bounds__(256, 4) n2v_walk_kernel(GraphView g, N2vTables<Bucket> t, N2vParams P, WalkLaunch L)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned team = __ballot_sync(kFullMask, i < L.walker_num);
    unsigned long long my_steps = 0;
    if (i < L.walker_num)
    {
        Sampler rng;
        rng.init(L.seed);
        WalkerRun<apps::Node2vecState> run;
        WalkerConfig<apps::Node2vecState> wc;
        walk_begin<apps::Node2vecState>(g, wc, L, i, run, rng);
        uint32_t len;
        const int status = n2v_walk<Weighted, Outlier, Bucket>(g, t, P, run.w.id, run.v, run.out, run.cap,
                                                               L.trial_limit, L.stats, team, rng, len);
        if (status != KK_STATUS_OK)
            atomicOr(L.status, status);
        L.length[i] = len;
        segment_done(L, i);
        my_steps = len - 1;
    }
    flush_steps(L.total_steps, my_steps);
}

/* Whether a walk's hooks are node2vec's own, every one of them (apps.cuh),
 * weighted or not, with its outlier or without: the kernels here restate them,
 * so a walk with another hook among them, or another walker config, is the
 * general kernels'. */
template <typename WC, typename TC>
constexpr bool is_node2vec()
{
    if constexpr (TC::order == 2)
    {
        using namespace apps;
        constexpr bool weighted = TC::has_static, outlier = TC::has_outlier;
        typedef SecondOrderTransitionConfig<
            Node2vecState, vertex_id_t, bool, FixedLengthExt<Node2vecState>,
            typename std::conditional<weighted, WeightStatic, NoHook>::type, Node2vecPostQuery, Node2vecRespond,
            Node2vecDyn, ConstBound, ConstBound,
            typename std::conditional<outlier, Node2vecOutlierUB<weighted>, NoHook>::type,
            typename std::conditional<outlier, Node2vecOutlierSearch, NoHook>::type>
            Plain;
        return std::is_same<TC, Plain>::value &&
               std::is_same<WC, WalkerConfig<Node2vecState, NoHook, NoHook, Node2vecUpdate>>::value;
    }
    return false;
}

/* Whether the kernels here can walk g over the set: they find positions in the
 * 32-bit offsets and count sectors in 32 bits. */
inline bool n2v_over_edge_set(const GraphView &g, const EdgeSetView &set)
{
    return set.keys != nullptr && g.off32 != nullptr && edge_set_in_32_bits(g.E, g.V, set.shift);
}

/* Whether the hooks read what the kernels here do: the graph's arrays, the
 * edge set and the 32-bit offsets, and at step 0 the bound that is the dart's. */
template <typename TC>
bool n2v_reads_graph(const GraphView &g, const TC &tc)
{
    bool same = n2v_over_edge_set(g, tc.respond_query.set) && tc.respond_query.nbr == g.nbr &&
                tc.dynamic_comp.upperbound == tc.dcomp_upperbound.value;
    if constexpr (TC::has_static)
        same = same && tc.static_comp.w == g.w;
    if constexpr (TC::has_outlier)
        same = same && tc.outlier_upperbound.set.keys == tc.respond_query.set.keys &&
               tc.outlier_search.nbr == g.nbr &&
               (!TC::has_static || (tc.outlier_upperbound.w == g.w && tc.outlier_upperbound.nbr == g.nbr));
    return same;
}

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
 * warp may hold walkers of several jobs: the lanes that take a walker in a pass
 * over the batch are its team. */
template <bool Weighted, typename Bucket, int MinBlocks>
__global__ void __launch_bounds__(256, MinBlocks)
    n2v_batch_kernel(GraphView g, N2vTables<Bucket> t, const BatchJob *jobs, uint32_t njobs, uint32_t total,
                     uint32_t *path, uint32_t *length, unsigned long long *total_steps, int *status,
                     uint32_t trial_limit, unsigned long long *stats, const uint32_t *hdr, BatchNotify nt)
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
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint64_t at = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; at < total; at += stride)
    {
        const unsigned team = __activemask();
        /* the walker's job, by its position in the launch order */
        uint32_t k = 0, hi = njobs;
        while (hi - k > 1)
        {
            const uint32_t mid = (k + hi) >> 1;
            if (s_first[mid] <= (uint32_t)at)
                k = mid;
            else
                hi = mid;
        }
        const BatchJob *job = jobs + s_first[kMaxBatchJobs + k];
        const uint32_t i = (uint32_t)at - s_first[k], cap = job->cap;
        Sampler rng;
        rng.init(job->seed);
        const walker_id_t id = job->walker_begin + i;
        const vertex_id_t v = id % g.V;
        uint32_t *out = path != nullptr ? path + job->path_base + (uint64_t)i * cap : nullptr;
        if (out != nullptr)
            out[0] = v;
        uint32_t len;
        const N2vParams P{job->c[0], job->c[1], job->c[2], job->c[3], job->c[4], fminf(job->c[4], 1.0f),
                          job->walk_length};
        const int failed =
            n2v_walk<Weighted, true, Bucket>(g, t, P, id, v, out, cap, trial_limit, stats, team, rng, len);
        const uint32_t j = (uint32_t)(job - jobs);
        if (failed != KK_STATUS_OK)
            atomicOr(nt.count != nullptr ? nt.status + j : status, failed);
        length[job->first_task + i] = len;
        my_steps += len - 1;
        WalkLaunch L;
        if (nt.count != nullptr)
        {
            /* the job is one segment of its own */
            L.walker_num = job->walker_num;
            L.seg_count = nt.count + j;
            L.seg_flag = nt.flag + j;
            L.seg_shift = 31;
            L.seg_status = nt.status + j;
        }
        segment_done(L, i);
    }
    flush_steps(total_steps, my_steps);
}

} // namespace kk
