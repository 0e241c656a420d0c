/*
 * node2vec from its functors (apps.cuh) through kk::random_walk, as a program
 * with hooks of its own would run it.  kk_node2vec_hooks walks with the
 * extension's length `length` and the path room of opts->walk_length.
 */
#include "knightking_gb300/engine.cuh"

using namespace kk;
using namespace kk::apps;

extern "C" kk_status kk_node2vec_hooks(kk_engine *e, const kk_walk_opts *opts, uint32_t length, kk_paths **out)
{
    *out = nullptr;
    SecondOrderTransitionConfig<Node2vecState, vertex_id_t, bool, FixedLengthExt<Node2vecState>, NoHook,
                                Node2vecPostQuery, Node2vecRespond, Node2vecDyn, ConstBound, ConstBound>
        tc;
    const kk_status s = guard(e, [&] {
        graph_sort_adjacency(e);
        const EdgeSetView set = node2vec_edge_set(e);
        const Node2vecConstants c = Node2vecConstants::make(opts->p, opts->q);
        tc.extension_comp = FixedLengthExt<Node2vecState>{length};
        tc.post_query = Node2vecPostQuery{c.inv_q < 1.0f ? c.inv_q : 1.0f};
        tc.respond_query = Node2vecRespond{e->d_nbr, set};
        tc.dynamic_comp = Node2vecDyn{c.upperbound, c.inv_p, c.inv_q};
        tc.dcomp_upperbound = ConstBound{c.upperbound};
        tc.dcomp_lowerbound = ConstBound{c.lowerbound};
    });
    if (s != KK_OK)
        return s;
    WalkerConfig<Node2vecState, NoHook, NoHook, Node2vecUpdate> wc;
    wc.walker_num = opts->walker_num;
    return random_walk<Node2vecState>(e, wc, tc, *opts, out);
}
