/* Which walk goes to the kernel for node2vec, asked on the host: prints a line
 * "V E shift keys off32 yes|no" per line "V E shift keys off32" read. */
#include <stdint.h>
#include <stdio.h>

#include "knightking_gb300/node2vec_walk.cuh"

using namespace kk;
using namespace kk::apps;

int main()
{
    unsigned long long V, E;
    unsigned shift, keys, off32;
    while (scanf("%llu %llu %u %u %u", &V, &E, &shift, &keys, &off32) == 5)
    {
        static uint32_t word[4]; /* an address for arrays that are there; nothing reads them */
        GraphView g{(vertex_id_t)V, E, nullptr, word, nullptr, nullptr};
        g.off32 = off32 ? word : nullptr;
        SecondOrderTransitionConfig<Node2vecState, vertex_id_t, bool, FixedLengthExt<Node2vecState>, NoHook,
                                    Node2vecPostQuery, Node2vecRespond, Node2vecDyn, ConstBound, ConstBound>
            tc;
        tc.dynamic_comp = Node2vecDyn{1.0f, 1.0f, 1.0f};
        tc.dcomp_upperbound = ConstBound{1.0f};
        tc.respond_query = Node2vecRespond{word, EdgeSetView{keys ? word : nullptr, false, nullptr, shift}};
        printf("%llu %llu %u %u %u %s\n", V, E, shift, keys, off32, n2v_reads_graph(g, tc) ? "yes" : "no");
    }
    return 0;
}
