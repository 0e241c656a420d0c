/*
 * node2vec's functors (apps.cuh) with one of them replaced by a program's own,
 * or with other values in them.  general: the dynamic component under another
 * name, which the kernel for node2vec does not know.
 */
#include "knightking_gb300/engine.cuh"

using namespace kk;
using namespace kk::apps;

namespace
{
struct OwnDyn : Node2vecDyn
{
};
struct OwnStart
{
    uint32_t v_num;
    __device__ vertex_id_t operator()(walker_id_t id, Sampler &rng) const
    {
        return (id * 7u + rng.gen(3)) % v_num;
    }
};
struct OwnExtension
{
    step_t walk_length;
    __device__ real_t operator()(const Walker<Node2vecState> &w, vertex_id_t v) const
    {
        return w.step >= walk_length || v % 5 == 0 ? 0.0f : 1.0f;
    }
};
struct OwnUpdate
{
    uint32_t v_num;
    __device__ void operator()(Walker<Node2vecState> &w, vertex_id_t cur, const AdjUnit &) const
    {
        w.data.previous_vertex = (cur * 3u + 1u) % v_num;
    }
};
struct OwnResponse
{
    __device__ void operator()(vertex_id_t, const vertex_id_t &query, const AdjList &, bool &resp) const
    {
        resp = query & 1;
    }
};
struct OwnQuery : Node2vecPostQuery
{
    __device__ bool operator()(const Walker<Node2vecState> &w, vertex_id_t cur, const AdjUnit &cand,
                               vertex_id_t &target, vertex_id_t &query) const
    {
        target = cur;
        query = cand.neighbour + 1;
        return w.step != 0;
    }
};
struct OwnLowerBound
{
    real_t value;
    __device__ real_t operator()(vertex_id_t v, const AdjList &) const { return v & 1 ? value : 0.0f; }
};

struct Call
{
    kk_engine *e;
    const kk_walk_opts *opts;
    kk_paths **out;
    EdgeSetView set;
    Node2vecConstants c;
};

template <typename Dyn, typename Static, typename OutUB, typename OutSearch, typename WC, typename Ext, typename PQ,
          typename Resp, typename LB>
kk_status walk(const Call &k, WC wc, Static st, Ext ext, PQ pq, Resp resp, float ub, LB lb, OutUB out_ub,
               OutSearch out_search)
{
    SecondOrderTransitionConfig<Node2vecState, vertex_id_t, bool, Ext, Static, PQ, Resp, Dyn, ConstBound, LB, OutUB,
                                OutSearch>
        tc;
    tc.extension_comp = ext;
    tc.static_comp = st;
    tc.post_query = pq;
    tc.respond_query = resp;
    static_cast<Node2vecDyn &>(tc.dynamic_comp) = Node2vecDyn{k.c.upperbound, k.c.inv_p, k.c.inv_q};
    tc.dcomp_upperbound = ConstBound{ub};
    tc.dcomp_lowerbound = lb;
    tc.outlier_upperbound = out_ub;
    tc.outlier_search = out_search;
    wc.walker_num = k.opts->walker_num;
    return random_walk<Node2vecState>(k.e, wc, tc, *k.opts, k.out);
}

template <typename Dyn>
kk_status variant(const Call &k, int which, const float *own_w)
{
    const uint32_t length = k.opts->walk_length;
    WalkerConfig<Node2vecState, NoHook, NoHook, Node2vecUpdate> wc{};
    const FixedLengthExt<Node2vecState> ext{length};
    const Node2vecPostQuery pq{k.c.inv_q < 1.0f ? k.c.inv_q : 1.0f};
    const Node2vecRespond resp{k.e->d_nbr, k.set};
    const ConstBound lb{k.c.lowerbound};
    const float ub = k.c.upperbound;
    const NoHook none{};
    switch (which)
    {
    case 0:
        return walk<Dyn>(k, wc, none, ext, pq, resp, ub, lb, none, none);
    case 1:
    {
        WalkerConfig<Node2vecState, OwnStart, NoHook, Node2vecUpdate> own{};
        own.walker_init_dist = OwnStart{k.e->V};
        return walk<Dyn>(k, own, none, ext, pq, resp, ub, lb, none, none);
    }
    case 2:
        return walk<Dyn>(k, wc, none, OwnExtension{length}, pq, resp, ub, lb, none, none);
    case 3:
    {
        WalkerConfig<Node2vecState, NoHook, NoHook, OwnUpdate> own{};
        own.walker_update_state = OwnUpdate{k.e->V};
        return walk<Dyn>(k, own, none, ext, pq, resp, ub, lb, none, none);
    }
    case 4:
        return walk<Dyn>(k, wc, none, ext, pq, OwnResponse{}, ub, lb, none, none);
    case 5:
        return walk<Dyn>(k, wc, none, ext, pq, resp, ub, OwnLowerBound{k.c.lowerbound}, none, none);
    case 6:
    {
        OwnQuery own;
        own.sure_below = 0.0f;
        return walk<Dyn>(k, wc, none, ext, own, resp, ub, lb, none, none);
    }
    case 7: /* a looser bound: step 0 is not always accepted */
        return walk<Dyn>(k, wc, none, ext, pq, resp, 2.0f * ub, lb, none, none);
    case 8: /* weights of the program's own, the return edge's among them */
        return walk<Dyn>(k, wc, WeightStatic{own_w}, ext, pq, resp, ub, lb,
                         Node2vecOutlierUB<true>{k.e->d_nbr, own_w, k.c.overflow, EdgeSetView{}},
                         Node2vecOutlierSearch{k.e->d_nbr});
    default:
        return KK_ERR_INVALID_CONFIG;
    }
}
} // namespace

extern "C" kk_status kk_node2vec_own_hooks(kk_engine *e, const kk_walk_opts *opts, int which, int general,
                                           const float *h_w, kk_paths **out)
{
    *out = nullptr;
    Call k{e, opts, out, EdgeSetView{}, Node2vecConstants::make(opts->p, opts->q)};
    float *d_w = nullptr;
    kk_status s = guard(e, [&] {
        graph_sort_adjacency(e);
        k.set = node2vec_edge_set(e);
        KK_CUDA_CHECK(cudaMalloc((void **)&d_w, e->E * 4 + 4));
        KK_CUDA_CHECK(cudaMemcpy(d_w, h_w, e->E * 4, cudaMemcpyHostToDevice));
    });
    if (s == KK_OK)
        s = general ? variant<OwnDyn>(k, which, d_w) : variant<Node2vecDyn>(k, which, d_w);
    cudaFree(d_w);
    return s;
}
