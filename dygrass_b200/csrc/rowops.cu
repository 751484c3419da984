// rowops.cu -- workspace of the row operations (rowops.cuh).
#include "rowops.cuh"

namespace dyg {

dyg_status rowops_ensure(dyg_graph *G, uint64_t m, cudaStream_t st) {
    Workspace &ws = G->ws;
    DYG_TRY(ensure(ws.nxt, sizeof(uint32_t) * (size_t)(m ? m : 1)));
    DYG_TRY(ensure(ws.rowlist, sizeof(uint32_t) * (size_t)(m ? m : 1)));
    DYG_TRY(ensure(ws.runs, sizeof(uint32_t) * (size_t)(m ? m : 1)));
    DYG_TRY(ensure(ws.blk, sizeof(uint32_t) * kOpBlocksMax * 2));
    if (!ws.rowcnt.p || !ws.rowhead.p) {
        const size_t bytes = sizeof(uint32_t) * (size_t)(G->g.n ? G->g.n : 1);
        DYG_TRY(ensure(ws.rowcnt, bytes));
        DYG_TRY(ensure(ws.rowhead, bytes));
        DYG_CUDA(cudaMemsetAsync(ws.rowcnt.p, 0, ws.rowcnt.bytes, st));
        DYG_CUDA(cudaMemsetAsync(ws.rowhead.p, 0, ws.rowhead.bytes, st));
    }
    return DYG_OK;
}

GridBar grid_bar(dyg_graph *G, unsigned long long *halt) {
    unsigned long long *sc = ptr<unsigned long long>(G->ws.scalars);
    uint32_t *words = reinterpret_cast<uint32_t *>(sc + S_BAR);
    return GridBar{words, words + 1, sc + S_ERR, halt, G->bar_limit, false};
}

AppSide append_side(dyg_graph *G, const uint32_t *src, const uint32_t *dst, const float *w) {
    Workspace &ws = G->ws;
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    return AppSide{G->g,
                   Chains{ptr<uint32_t>(ws.rowcnt), ptr<uint32_t>(ws.rowhead), ptr<uint32_t>(ws.nxt),
                          ptr<uint32_t>(ws.rowlist), sc + S_ITEMS, ptr<uint32_t>(ws.runs), sc + S_RUNS},
                   EdgeList{src, dst, w}, G->slack, sc};
}

}  // namespace dyg
