// stream.cu -- one file of the mixed insert/delete edge stream
// (dynamic_update/main.cu:96-126: preprocessStreamEdges, then walks in
// chunks with the sparsifier updated after each chunk).
//
// Insert file (gpu_graph.cuh:373-396, 620-643), all on the device:
//   probe    every edge's slot positions in G and H (rows scanned by groups
//            of 8 lanes, the shorter row first); the occurrences of one edge
//            chained under its (min, max) key in a hash table;
//   merge    one thread per edge: its occurrences in file order; an edge
//            already in G adds every
//            occurrence's weight to G (and H) in file order; a new edge's
//            first occurrence enters G with the later occurrences' weights
//            folded in, and is listed for walking (edges repeated more than 32
//            times are folded by warps and blocks, as the append's first phase);
//   append   the new edges to G in file order (row order as the reference's
//            edgeInsertion produces);
//   chunks   of the walk list: walk H, then append the accepted edges to H
//            with their stream weight before the next chunk walks.
// Delete file (gpu_graph.cuh:398-431, 645-700): the whole file is deleted
// from G and H, then the walk list is walked on G and recovered in chunks.
// One host synchronize per file; a reservation that does not fit halts every
// later kernel and the file resumes at the halted stage after the arena or
// record buffers grew (nothing changed after the halt; the weight merges
// come before any reservation and are not repeated).
#include "dyg_internal.cuh"
#include "gridsync.cuh"
#include "rowops.cuh"

namespace dyg {

namespace {

constexpr uint32_t kProbeLanes = 8;

inline int blocks(uint64_t n, int th) { return (int)((n + th - 1) / th); }

#define HALTED(h) ((h) && *(h))

// Arena index of the first slot of row x holding y, or ~0u.  Called by the
// kProbeLanes lanes of one group together (`gmask` = the group's lanes).
__device__ __forceinline__ uint32_t group_find(const DevGraph &g, uint32_t x, uint32_t y,
                                               uint32_t lane, uint32_t gbase, uint32_t gmask) {
    const uint2 d = g.desc[x];
    constexpr uint32_t U = 4;   // a group's tile: U loads per lane issued before any compare
    for (uint32_t t0 = 0; t0 < d.y; t0 += U * kProbeLanes) {
        uint32_t cv[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t j = t0 + u * kProbeLanes + lane;
            cv[u] = j < d.y ? g.slots[d.x + j].x : ~0u;   // vertex ids are never ~0u
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t bits =
                (__ballot_sync(gmask, cv[u] == y) >> gbase) & ((1u << kProbeLanes) - 1u);
            if (bits) return d.x + t0 + u * kProbeLanes + (uint32_t)(__ffs(bits) - 1);
        }
    }
    return ~0u;
}

// Slots of edge {a, b} in g: .x in row a, .y in row b (~0u when absent).
__device__ __forceinline__ uint2 group_edge(const DevGraph &g, uint32_t a, uint32_t b,
                                            uint32_t lane, uint32_t gbase, uint32_t gmask) {
    const bool a_short = g.desc[a].y <= g.desc[b].y;
    const uint32_t s = a_short ? a : b, l = a_short ? b : a;
    const uint32_t ps = group_find(g, s, l, lane, gbase, gmask);
    if (ps == ~0u) return make_uint2(~0u, ~0u);
    const uint32_t pl = group_find(g, l, s, lane, gbase, gmask);
    return a_short ? make_uint2(ps, pl) : make_uint2(pl, ps);
}

__device__ __forceinline__ bool long_rows(const DevGraph &g, uint32_t a, uint32_t b) {
    return g.desc[a].y > kBigRow || g.desc[b].y > kBigRow;
}

// group_edge for an edge with a row longer than kBigRow: the group searches
// the shorter row when it has at most kBigRow slots, which settles an absent
// edge; *open is set when a search of a long row remains (the edge is in the
// short row, whose slot is returned, or both rows are long).
__device__ __forceinline__ uint2 group_edge_short(const DevGraph &g, uint32_t a, uint32_t b,
                                                  uint32_t lane, uint32_t gbase, uint32_t gmask,
                                                  bool *open) {
    const uint2 da = g.desc[a], db = g.desc[b];
    const bool a_short = da.y <= db.y;
    *open = false;
    if ((a_short ? db.y : da.y) <= kBigRow) return group_edge(g, a, b, lane, gbase, gmask);
    if ((a_short ? da.y : db.y) > kBigRow) {
        *open = true;
        return make_uint2(~0u, ~0u);
    }
    const uint32_t ps = group_find(g, a_short ? a : b, a_short ? b : a, lane, gbase, gmask);
    *open = ps != ~0u;
    return a_short ? make_uint2(ps, ~0u) : make_uint2(~0u, ps);
}

// The file's edges by (min, max) key: an open-addressing table of T >= 2n slots
// (empty between files: key ~0, no occurrences) with a chain of occurrences
// per key.
struct EdgeTable {
    unsigned long long *key;
    uint32_t *cnt, *head;     // per slot: occurrences, last occurrence + 1
    uint32_t mask;
    uint32_t *nxt, *slot;     // per edge: previous occurrence + 1 (0: leader, ~0u: not in the
                              // table); its slot
};

__device__ __forceinline__ unsigned long long pair_key(uint32_t a, uint32_t b) {
    return ((unsigned long long)a << 32) | b;   // a < b
}

__device__ __forceinline__ void table_link(const EdgeTable &t, uint32_t i, unsigned long long k) {
    unsigned long long h = k * 0x9E3779B97F4A7C15ull;
    h ^= h >> 32;
    uint32_t s = (uint32_t)h & t.mask;
    while (true) {
        const unsigned long long prev = atomicCAS(t.key + s, ~0ull, k);
        if (prev == ~0ull || prev == k) break;
        s = (s + 1u) & t.mask;
    }
    t.slot[i] = s;
    t.nxt[i] = atomicExch(t.head + s, i + 1u);
    atomicAdd(t.cnt + s, 1u);
}

// One group of kProbeLanes lanes per edge: slot positions in G and H, and the
// edge's entry in the table; self-loops and invalid endpoints stay out of it
// (never merged or walked).  An edge with a row longer
// than kBigRow in G or H has its short rows searched here
// (group_edge_short); if a long row remains to be searched it goes to the big
// list for k_st_probe_big, with bit 0 (G) and bit 1 (H) of .w naming the
// graphs whose search is open.
__global__ void k_st_probe(const unsigned long long *halt, DevGraph G, DevGraph H,
                           const uint32_t *src, const uint32_t *dst, uint32_t n, EdgeTable tab,
                           uint4 *pos, uint32_t *nflag,
                           int32_t *status, float *cond, uint4 *big, unsigned long long *nbig,
                           bool big_ok, unsigned long long *fold, unsigned long long *err) {
    if (HALTED(halt)) return;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0u) *fold = 0ull;
    const uint32_t i = t / kProbeLanes;
    const uint32_t lane = t % kProbeLanes;
    const uint32_t gbase = (threadIdx.x & 31u) & ~(kProbeLanes - 1u);
    const uint32_t gmask = ((1u << kProbeLanes) - 1u) << gbase;
    if (i >= n) return;   // whole groups leave together (n is per group)
    uint32_t a = src[i], b = dst[i];
    if (a > b) {
        const uint32_t x = a;
        a = b;
        b = x;
    }
    if (a == b || b >= G.n) {
        if (lane == 0) {
            if (b >= G.n) atomicOr(err, (unsigned long long)kErrVertex);
            tab.nxt[i] = ~0u;
            pos[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
            nflag[i] = 0;
            status[i] = DYG_INS_SELF_LOOP;
            cond[i] = 0.f;
        }
        return;
    }
    if (lane == 0) {
        table_link(tab, i, pair_key(a, b));
        nflag[i] = 0;
    }
    if (big_ok && (long_rows(G, a, b) || long_rows(H, a, b))) {
        bool og, oh;
        const uint2 pg = group_edge_short(G, a, b, lane, gbase, gmask, &og);
        const uint2 ph = group_edge_short(H, a, b, lane, gbase, gmask, &oh);
        if (lane == 0) {
            pos[i] = make_uint4(pg.x, pg.y, ph.x, ph.y);
            if (og || oh)
                big[atomicAdd(nbig, 1ull)] = make_uint4(i, a, b, (og ? 1u : 0u) | (oh ? 2u : 0u));
        }
        return;
    }
    const uint2 pg = group_edge(G, a, b, lane, gbase, gmask);
    const uint2 ph = group_edge(H, a, b, lane, gbase, gmask);
    if (lane == 0) pos[i] = make_uint4(pg.x, pg.y, ph.x, ph.y);
}

// Finishes group_edge_short's search of edge {a, b} in g by block-wide
// scans: `part` is its result (the short row's slot when only the long row
// remains).
__device__ uint2 block_edge(const DevGraph &g, uint32_t a, uint32_t b, uint2 part,
                            uint32_t *s_best) {
    const uint2 da = g.desc[a], db = g.desc[b];
    const bool a_short = da.y <= db.y;
    const uint2 ds = a_short ? da : db, dl = a_short ? db : da;
    const uint32_t s = a_short ? a : b, l = a_short ? b : a;
    uint32_t ps = a_short ? part.x : part.y;
    if (ds.y > kBigRow) {
        const uint32_t js = block_find(g.slots, ds.x, ds.y, l, s_best);
        if (js == ~0u) return make_uint2(~0u, ~0u);
        ps = ds.x + js;
    }
    const uint32_t jl = block_find(g.slots, dl.x, dl.y, s, s_best);
    const uint32_t pl = jl == ~0u ? ~0u : dl.x + jl;
    return a_short ? make_uint2(ps, pl) : make_uint2(pl, ps);
}

// One block per edge on the big list: the long-row searches k_st_probe left.
__global__ void k_st_probe_big(const unsigned long long *halt, DevGraph G, DevGraph H,
                               const uint4 *big, const unsigned long long *nbig, uint4 *pos) {
    __shared__ uint32_t s_best;
    if (HALTED(halt)) return;
    const uint32_t nbl = (uint32_t)*nbig;
    for (uint32_t q = blockIdx.x; q < nbl; q += gridDim.x) {
        const uint4 e = big[q];
        uint4 p = pos[e.x];
        if (e.w & 1u) {
            const uint2 pg = block_edge(G, e.y, e.z, make_uint2(p.x, p.y), &s_best);
            p.x = pg.x;
            p.y = pg.y;
        }
        if (e.w & 2u) {
            const uint2 ph = block_edge(H, e.y, e.z, make_uint2(p.z, p.w), &s_best);
            p.z = ph.x;
            p.w = ph.y;
        }
        if (threadIdx.x == 0) pos[e.x] = p;   // each edge is on the list once
    }
}

__device__ __forceinline__ void set_weight(const DevGraph &g, uint32_t slot, float w) {
    g.wts[slot] = w;
    g.slots[slot].y = __float_as_uint(__frcp_rn(w));
}

// One edge's occurrences folded in file order, one float add each
// (dynamic_update/gpu_graph.cuh:373-396, 452-465).
struct Fold {
    uint4 p;       // the first occurrence's slots
    uint32_t i0;
    bool first;
    float ga, gb, ha, hb, wa;
};
struct MergeArgs {
    DevGraph G, H;
    const uint32_t *src, *dst;
    const float *w;
    uint32_t n;
    EdgeTable tab;
    const uint4 *pos;
    uint32_t *nflag;
    float *wapp;
    int32_t *status;
    float *cond;
    uint4 *often;               // edges repeated more than kFoldChain times: slot, count, start of run
    uint32_t *runs;             // their occurrences
    unsigned long long *fold;   // S_FOLD
};

__device__ __forceinline__ void fold_add(const MergeArgs &a, Fold &f, uint32_t i) {
    const float wi = a.w[i];
    if (f.first) {
        f.first = false;
        f.i0 = i;
        f.p = a.pos[i];
        f.ga = f.p.x != ~0u ? a.G.wts[f.p.x] : 0.f;
        f.gb = f.p.y != ~0u ? a.G.wts[f.p.y] : 0.f;
        f.ha = f.p.z != ~0u ? a.H.wts[f.p.z] : 0.f;
        f.hb = (f.p.z != ~0u && f.p.w != ~0u) ? a.H.wts[f.p.w] : 0.f;
        if (f.p.x == ~0u) {
            // new: the first occurrence enters G and is walked; the later ones
            // add their weights to its G copy (and to H's, if H has the edge)
            f.wa = wi;
            return;
        }
    }
    // already in G: every occurrence adds its weight to G and (if there) H
    f.wa = __fadd_rn(f.wa, wi);
    f.ga = __fadd_rn(f.ga, wi);
    f.gb = __fadd_rn(f.gb, wi);
    f.ha = __fadd_rn(f.ha, wi);
    f.hb = __fadd_rn(f.hb, wi);
    a.status[i] = DYG_INS_MERGED;
    a.cond[i] = 0.f;
}

__device__ __forceinline__ void fold_end(const MergeArgs &a, const Fold &f) {
    if (f.p.x != ~0u) {
        set_weight(a.G, f.p.x, f.ga);
        if (f.p.y != ~0u) set_weight(a.G, f.p.y, f.gb);
    } else {
        a.nflag[f.i0] = 1u;
        a.wapp[f.i0] = f.wa;
    }
    if (f.p.z != ~0u) {
        set_weight(a.H, f.p.z, f.ha);
        if (f.p.w != ~0u) set_weight(a.H, f.p.w, f.hb);
    }
}

// One thread per edge: the leader of each key's chain empties its table slot
// and folds its occurrences.  A chain of up to kFoldChain is followed and put
// in file order, in a local array of 128 bytes; a longer one is left to fold_often.
constexpr uint32_t kFoldChain = 32;
constexpr uint32_t kFoldThreads = 256;
__global__ void __launch_bounds__(kFoldThreads) k_st_merge(const unsigned long long *halt, MergeArgs a) {
    if (HALTED(halt)) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || a.tab.nxt[i] != 0u) return;
    const uint32_t s = a.tab.slot[i], c = a.tab.cnt[s];
    uint32_t k = a.tab.head[s];
    if (c > kFoldChain) {
        const unsigned long long at = atomicAdd(a.fold, (1ull << 32) + c);
        a.often[at >> 32] = make_uint4(s, c, (uint32_t)at, 0u);
        a.tab.head[s] = (uint32_t)at;
        return;
    }
    a.tab.key[s] = ~0ull;
    a.tab.cnt[s] = 0u;
    a.tab.head[s] = 0u;
    Fold f{};
    f.first = true;
    if (c == 1u) {
        fold_add(a, f, i);
    } else {
        uint32_t idx[kFoldChain];
        for (uint32_t u = 0; u < c; ++u) {   // insertion by file index
            const uint32_t v = k - 1u;
            k = a.tab.nxt[v];
            uint32_t b = u;
            while (b > 0u && idx[b - 1u] > v) {
                idx[b] = idx[b - 1u];
                --b;
            }
            idx[b] = v;
        }
        for (uint32_t u = 0; u < c; ++u) fold_add(a, f, idx[u]);
    }
    fold_end(a, f);
}

// A warp folds the c occurrences run[0, c), in file order: 32 weights at a time
// are loaded together and added one after the other, as fold_add does.
__device__ __forceinline__ void warp_fold(const MergeArgs &a, const uint32_t *run, uint32_t c, uint32_t lane) {
    Fold f{};
    f.i0 = run[0];
    f.p = a.pos[f.i0];
    f.ga = f.p.x != ~0u ? a.G.wts[f.p.x] : 0.f;
    f.gb = f.p.y != ~0u ? a.G.wts[f.p.y] : 0.f;
    f.ha = f.p.z != ~0u ? a.H.wts[f.p.z] : 0.f;
    f.hb = (f.p.z != ~0u && f.p.w != ~0u) ? a.H.wts[f.p.w] : 0.f;
    const bool is_new = f.p.x == ~0u;
    for (uint32_t g0 = 0; g0 < c; g0 += 32u) {
        const uint32_t gc = min(32u, c - g0);
        float w = 0.f;
        if (lane < gc) {
            const uint32_t i = run[g0 + lane];
            w = a.w[i];
            if (!is_new || g0 + lane > 0u) {
                a.status[i] = DYG_INS_MERGED;
                a.cond[i] = 0.f;
            }
        }
        for (uint32_t u = 0; u < gc; ++u) {
            const float x = __shfl_sync(kFull, w, u);
            if (is_new && g0 + u == 0u) {   // enters G; the later ones are added
                f.wa = x;
                continue;
            }
            f.wa = __fadd_rn(f.wa, x);
            f.ga = __fadd_rn(f.ga, x);
            f.gb = __fadd_rn(f.gb, x);
            f.ha = __fadd_rn(f.ha, x);
            f.hb = __fadd_rn(f.hb, x);
        }
    }
    __syncwarp();   // every lane has read the weights
    if (lane == 0u) fold_end(a, f);
}

// The edges repeated more than kFoldChain times.  Their occurrences put
// themselves into runs, which a warp (up to kWarpRun) or a block (kSortMax) puts
// in file order; for more occurrences the block scans the file.  Files of a
// million edges, 33 / 100 / 1,000 times each: 0.96, 0.83, 0.87 ms; with a scan of
// the file for each such edge, whose finds one thread folded, 705, 662, 169 ms
// (4,096 edges, 64 times each: 0.10 and 0.33).
static __device__ __noinline__ bool fold_often(const MergeArgs &a, const GridBar &bar, RowShared &s) {
    const uint32_t n_often = (uint32_t)(__ldcg(a.fold) >> 32);
    const uint2 rg = block_range(a.n);
    for (uint32_t i = rg.x + threadIdx.x; i < rg.y; i += blockDim.x) {
        if (a.tab.nxt[i] == ~0u) continue;
        const uint32_t t = a.tab.slot[i], c = a.tab.cnt[t];   // 0: folded
        if (c > kFoldChain && c <= kSortMax) a.runs[atomicAdd(a.tab.head + t, 1u)] = i;
    }
    if (!grid_sync(bar)) return false;
    const uint32_t lane = threadIdx.x & 31u, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; q < n_often; q += warps) {
        const uint4 e = a.often[q];
        if (e.y > kWarpRun) continue;
        warp_sort_run(a.runs + e.z, e.y, lane);
        warp_fold(a, a.runs + e.z, e.y, lane);
    }
    for (uint32_t q = blockIdx.x; q < n_often; q += gridDim.x) {
        const uint4 e = a.often[q];
        if (e.y <= kWarpRun) continue;
        uint32_t *run = a.runs + e.z;
        if (e.y <= kSortMax) {
            block_load_sorted(run, e.y, s.sort);
            for (uint32_t k = threadIdx.x; k < e.y; k += blockDim.x) run[k] = s.sort[k];
        } else {
            scan_entries(
                a.n, e.y, s, [&](uint32_t i) { return a.tab.nxt[i] != ~0u && a.tab.slot[i] == e.x ? 1u : 0u; },
                [&](uint32_t k, uint32_t j) { run[k] = j >> 1; });
        }
        __syncthreads();
        if (threadIdx.x < 32u) warp_fold(a, run, e.y, lane);
        __syncthreads();
    }
    // every block is done with the counts before the slots are emptied
    if (!grid_sync(bar, [&] { *a.fold = 0ull; })) return false;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n_often; q += gridDim.x * blockDim.x) {
        const uint32_t t = a.often[q].x;
        a.tab.key[t] = ~0ull;
        a.tab.cnt[t] = 0u;
        a.tab.head[t] = 0u;
    }
    return true;
}

// New edges in file order: G's half-edges (src gets dst, dst gets src; merged
// weight) and the walk list (file orientation, stream weight).
struct NewEdgeOp {
    static constexpr bool kList = true, kPrep = true;
    MergeArgs merge;
    const uint32_t *nflag, *src, *dst;
    const float *w;
    uint32_t n;
    unsigned long long uid0;
    uint32_t *f_src, *f_dst;
    float *f_w;
    unsigned long long *f_uid;
    uint32_t *f_idx, *counts;
    unsigned long long *hkeys;   // zeroed for the first chunk's walks
    uint32_t nkeys;
    __device__ bool pending() const { return __ldcg(merge.fold) != 0ull; }
    __device__ bool prep(const GridBar &bar, RowShared &s) const { return fold_often(merge, bar, s); }
    __device__ uint32_t count() const { return n; }
    __device__ uint32_t take(uint32_t i) const {
        if (i < nkeys) hkeys[i] = 0ull;
        return nflag[i];
    }
    __device__ bool listed(uint32_t i) const { return nflag[i] != 0u; }
    __device__ void list(uint32_t i, uint32_t q) const {
        f_src[q] = src[i];
        f_dst[q] = dst[i];
        f_w[q] = w[i];
        f_uid[q] = uid0 + i;
        f_idx[q] = i;
    }
    __device__ void total(uint32_t n_new) const { counts[C_WALKLIST] = n_new; }
};

// Chunk results: found_at / conductance by file index, and the accepted
// edges (no walker connected them) to H in chunk order.  Keys are zeroed
// behind the decode for the next chunk's walks.
struct StAcceptOp {
    static constexpr bool kList = false, kPrep = false;
    WalkJob job;
    unsigned long long *keys;
    const uint32_t *f_idx;
    int32_t *status;
    float *cond;
    __device__ uint32_t count() const { return job_count(job); }
    __device__ uint32_t take(uint32_t f) const {
        const unsigned long long k = keys[f];
        if (k) keys[f] = 0ull;
        const uint32_t i = f_idx[f];
        status[i] = key_found(k);
        cond[i] = k ? __uint_as_float((uint32_t)(k >> 32)) : 0.f;
        return k ? 0u : 1u;
    }
};

uint64_t table_slots(uint32_t n) {
    uint64_t T = 1024;
    while (T < 2ull * n) T <<= 1;
    return T;
}

dyg_status table_ensure(dyg_graph *G, uint32_t n, cudaStream_t st) {
    Workspace &ws = G->ws;
    const uint64_t T = table_slots(n);
    if (ws.st_key.bytes < sizeof(unsigned long long) * T || ws.st_cnt.bytes < 2 * sizeof(uint32_t) * T) {
        // empty when allocated, and left empty by every file
        DYG_TRY(ensure(ws.st_key, sizeof(unsigned long long) * T));
        DYG_TRY(ensure(ws.st_cnt, 2 * sizeof(uint32_t) * T));
        DYG_CUDA(cudaMemsetAsync(ws.st_key.p, 0xFF, ws.st_key.bytes, st));
        DYG_CUDA(cudaMemsetAsync(ws.st_cnt.p, 0, ws.st_cnt.bytes, st));
    }
    return DYG_OK;
}

MergeArgs merge_args(dyg_graph *G, dyg_graph *H, const uint32_t *src, const uint32_t *dst, const float *w,
                     uint32_t n, int32_t *status, float *cond) {
    Workspace &ws = G->ws;
    // counts and heads: the halves of one allocation
    uint32_t *cnt = ptr<uint32_t>(ws.st_cnt), *head = cnt + ws.st_cnt.bytes / (2 * sizeof(uint32_t));
    uint32_t *nxt = ptr<uint32_t>(ws.st_val), *slot = nxt + n;
    const EdgeTable tab{ptr<unsigned long long>(ws.st_key), cnt, head, (uint32_t)(table_slots(n) - 1), nxt, slot};
    return MergeArgs{G->g, H->g, src, dst, w, n, tab, ptr<uint4>(ws.st_pos), ptr<uint32_t>(ws.flags),
                     ptr<float>(ws.st_wapp), status, cond, ptr<uint4>(ws.big), ptr<uint32_t>(ws.runs),
                     ptr<unsigned long long>(ws.scalars) + S_FOLD};
}

// Probe and merge an insert file (no reservation: never halts).
dyg_status insert_prep_enqueue(dyg_graph *G, dyg_graph *H, const MergeArgs &a, unsigned long long *halt,
                               cudaStream_t st) {
    Workspace &ws = G->ws;
    const uint32_t n = a.n;
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    const bool big_ok = G->long_rows || H->long_rows;
    if (big_ok) DYG_CUDA(cudaMemsetAsync(sc + S_NBIG, 0, sizeof(unsigned long long), st));
    k_st_probe<<<blocks((uint64_t)n * kProbeLanes, 256), 256, 0, st>>>(
        halt, G->g, H->g, a.src, a.dst, n, a.tab, ptr<uint4>(ws.st_pos), a.nflag, a.status, a.cond,
        ptr<uint4>(ws.big), sc + S_NBIG, big_ok, a.fold, sc + S_ERR);
    count_launch();
    if (big_ok) {
        k_st_probe_big<<<num_sms() * 4, kBigThreads, 0, st>>>(halt, G->g, H->g, ptr<uint4>(ws.big),
                                                              sc + S_NBIG, ptr<uint4>(ws.st_pos));
        count_launch();
    }
    k_st_merge<<<blocks(n, kFoldThreads), kFoldThreads, 0, st>>>(halt, a);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

dyg_status insert_gappend_enqueue(dyg_graph *G, dyg_graph *H, const MergeArgs &a, uint64_t uid0,
                                  uint32_t nkeys, unsigned long long *halt, cudaStream_t st) {
    Workspace &ws = G->ws;
    const uint32_t n = a.n;
    const NewEdgeOp op{a, a.nflag, a.src, a.dst, a.w, n, (unsigned long long)uid0,
                       ptr<uint32_t>(ws.f_src), ptr<uint32_t>(ws.f_dst), ptr<float>(ws.f_w),
                       ptr<unsigned long long>(ws.f_uid), ptr<uint32_t>(ws.f_idx),
                       ptr<uint32_t>(ws.counts), ptr<unsigned long long>(H->ws.keys), nkeys};
    return append_enqueue(op, n, G, EdgeList{a.src, a.dst, a.wapp}, nullptr, EdgeList{},
                          ptr<unsigned long long>(H->ws.scalars) + S_WORK, halt, halt_code(0, (uint32_t)kHaltArena, 1), st);
}

// Walks chunk c (walk-list entries [c*chunk, c*chunk + nc)) on H and appends
// its accepted edges to H.  walk_ready: the launch before left H's keys and
// chunk counter zero.
dyg_status insert_chunk_enqueue(dyg_graph *G, dyg_graph *H, uint32_t c, uint32_t chunk,
                                uint32_t nc, const dyg_walk_params &p, unsigned long long *halt,
                                int32_t *status, float *cond, bool walk_ready, WalkScratch &scratch,
                                cudaStream_t st) {
    Workspace &wg = G->ws, &wh = H->ws;
    const uint32_t f0 = c * chunk;
    const uint32_t *fsrc = ptr<uint32_t>(wg.f_src) + f0, *fdst = ptr<uint32_t>(wg.f_dst) + f0;
    const float *fw = ptr<float>(wg.f_w) + f0;
    unsigned long long *keys = ptr<unsigned long long>(wh.keys);
    if (!walk_ready) DYG_CUDA(cudaMemsetAsync(keys, 0, sizeof(unsigned long long) * nc, st));
    const WalkJob job{halt, fsrc, fdst, fw, ptr<unsigned long long>(wg.f_uid) + f0, 0ull,
                      ptr<uint32_t>(wg.counts) + C_WALKLIST, nc, kDomainIncr, f0};
    RowIndex ix{};
    DYG_TRY(index_enqueue(H, nc, p, true, halt, scratch, &ix, st));
    DYG_TRY(launch_walk(H, job, p, true, keys, ix, st, walk_ready));
    const StAcceptOp op{job, keys, ptr<uint32_t>(wg.f_idx) + f0, status, cond};
    return append_enqueue(op, nc, H, EdgeList{fsrc, fdst, fw}, nullptr, EdgeList{},
                          ptr<unsigned long long>(wh.scalars) + S_WORK, halt,
                          halt_code(c + 1, (uint32_t)kHaltArena, 0), st);
}

struct HaltInfo {
    uint32_t batch, kind, phase;
};

HaltInfo decode_halt(unsigned long long h) {
    return HaltInfo{(uint32_t)(h >> 8) - 1u, (uint32_t)((h >> 4) & 0xF), (uint32_t)(h & 0xF)};
}

dyg_status clear_halt(dyg_graph *D, cudaStream_t st) {
    DYG_CUDA(cudaMemsetAsync(ptr<unsigned long long>(D->ws.scalars) + S_HALT, 0,
                             sizeof(unsigned long long), st));
    return DYG_OK;
}

dyg_status insert_file_run(dyg_graph *G, dyg_graph *H, const uint32_t *src, const uint32_t *dst,
                           const float *w, uint32_t n, uint64_t uid0, uint32_t chunk,
                           const dyg_walk_params &p, int32_t *status, float *cond,
                           cudaStream_t st, bool check_inputs,
                           const std::function<dyg_status()> *fetch) {
    Workspace &wg = G->ws, &wh = H->ws;
    const uint32_t nc_max = n < chunk ? n : chunk;
    // every buffer at its final size before anything is enqueued: a resumed
    // stage finds the earlier stages' lists where they were left
    DYG_TRY(ensure(wg.st_val, sizeof(uint32_t) * (size_t)n * 2));
    DYG_TRY(ensure(wg.st_pos, sizeof(uint4) * (size_t)n));
    DYG_TRY(ensure(wg.st_wapp, sizeof(float) * (size_t)n));
    DYG_TRY(ensure(wg.big, sizeof(uint4) * (size_t)n));
    DYG_TRY(ensure(wg.flags, sizeof(uint32_t) * (size_t)n));
    DYG_TRY(ensure(wg.f_src, sizeof(uint32_t) * (size_t)n));
    DYG_TRY(ensure(wg.f_dst, sizeof(uint32_t) * (size_t)n));
    DYG_TRY(ensure(wg.f_w, sizeof(float) * (size_t)n));
    DYG_TRY(ensure(wg.f_uid, sizeof(unsigned long long) * (size_t)n));
    DYG_TRY(ensure(wg.f_idx, sizeof(uint32_t) * (size_t)n));
    DYG_TRY(ensure(wh.keys, sizeof(unsigned long long) * (size_t)nc_max));
    DYG_TRY(rowops_ensure(G, 2ull * n, st));
    DYG_TRY(rowops_ensure(H, 2ull * nc_max, st));
    DYG_TRY(table_ensure(G, n, st));
    WalkScratch scratch(st);
    unsigned long long *halt = ptr<unsigned long long>(wg.scalars) + S_HALT;
    DYG_TRY(clear_halt(G, st));
    if (check_inputs)
        DYG_TRY(validate_enqueue(halt, ptr<unsigned long long>(wg.scalars) + S_ERR, src, dst, w, n,
                                 G->g.n, st));
    DYG_TRY(insert_prep_enqueue(G, H, merge_args(G, H, src, dst, w, n, status, cond), halt, st));
    const uint32_t nchunks = (uint32_t)(((uint64_t)n + chunk - 1) / chunk);
    uint32_t start = 0;   // 0 = G append, c + 1 = chunk c
    for (int round = 0; round < 64; ++round) {
        if (start == 0)   // G's arena may have grown: its arrays as they are now
            DYG_TRY(insert_gappend_enqueue(G, H, merge_args(G, H, src, dst, w, n, status, cond), uid0, nc_max, halt, st));
        const uint32_t c0 = start ? start - 1 : 0;
        for (uint32_t c = c0; c < nchunks; ++c) {
            const uint32_t f0 = c * chunk;
            const uint32_t nc = n - f0 < chunk ? n - f0 : chunk;
            DYG_TRY(insert_chunk_enqueue(G, H, c, chunk, nc, p, halt, status, cond, start == 0 || c > c0, scratch, st));
        }
        if (fetch) DYG_TRY((*fetch)());
        DYG_TRY(read_scalars2(G, H, st));
        const unsigned long long h = wg.host_scalars[S_HALT];
        if (!h) return DYG_OK;
        const HaltInfo hi = decode_halt(h);
        if (hi.kind == kHaltInvalid) return rejected_inputs(G, st);
        dyg_graph *grow = hi.batch == 0 ? G : H;
        DYG_TRY(scratch.with_room([&] { return grow_arena(grow, grow->g.arena_cap * 2, st); }));
        DYG_TRY(clear_halt(G, st));
        start = hi.batch;
    }
    set_error("insert file: too many arena regrowths");
    return DYG_ENOMEM;
}

dyg_status delete_file_run(dyg_graph *G, dyg_graph *H, const uint32_t *src, const uint32_t *dst,
                           uint32_t n, uint64_t uid0, uint32_t chunk, const dyg_walk_params &p,
                           int32_t *status, float *cond, uint64_t *n_rec, cudaStream_t st,
                           bool check_inputs, const std::function<dyg_status()> *fetch) {
    Workspace &ws = G->ws;
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    unsigned long long *halt = sc + S_HALT;
    const uint64_t want = (uint64_t)n * 4 + 1024;
    DYG_TRY(ensure(ws.rx2, sizeof(uint32_t) * want));
    DYG_TRY(ensure(ws.ry2, sizeof(uint32_t) * want));
    DYG_TRY(ensure(ws.rk2, want));
    uint64_t cap = ws.rx2.bytes / 4;
    if (ws.ry2.bytes / 4 < cap) cap = ws.ry2.bytes / 4;
    if (ws.rk2.bytes < cap) cap = ws.rk2.bytes;
    unsigned long long init[2] = {0ull, cap};   // S_RECCNT, S_RECCAP
    DYG_CUDA(cudaMemcpyAsync(sc + S_RECCNT, init, sizeof(init), cudaMemcpyHostToDevice, st));
    DYG_TRY(clear_halt(G, st));
    if (check_inputs)
        DYG_TRY(validate_enqueue(halt, sc + S_ERR, src, dst, nullptr, n, G->g.n, st));
    DYG_TRY(decr_delete_ensure(G, H, n, st));
    DYG_TRY(decr_walk_ensure(G, H, n < chunk ? n : chunk, p, st));
    WalkScratch scratch(st);
    scratch.open_paths(G, n, p);
    DYG_TRY(decr_delete_enqueue(G, H, src, dst, n, uid0, nullptr, true, halt, status, cond, st));
    const uint32_t nchunks = (uint32_t)(((uint64_t)n + chunk - 1) / chunk);
    uint32_t c_start = 0, ph_start = 0;
    for (int round = 0; round < 64; ++round) {
        for (uint32_t c = c_start; c < nchunks; ++c) {
            const uint32_t f0 = c * chunk;
            const uint32_t nc = n - f0 < chunk ? n - f0 : chunk;
            DYG_TRY(decr_walk_enqueue(G, H, f0, nc, ptr<uint32_t>(ws.counts) + C_FILTERED, p, halt,
                                      c, c == c_start ? ph_start : 0, status, cond, st, true, scratch));
        }
        if (fetch) DYG_TRY((*fetch)());
        DYG_TRY(read_scalars2(G, H, st));
        const unsigned long long h = ws.host_scalars[S_HALT];
        if (!h) {
            *n_rec = ws.host_scalars[S_RECCNT];
            return DYG_OK;
        }
        const HaltInfo hi = decode_halt(h);
        if (hi.kind == kHaltInvalid) return rejected_inputs(G, st);
        if (hi.kind == kHaltRecords) {
            const uint64_t used = ws.host_scalars[S_RECCNT];
            const uint64_t ncap = cap * 2;
            DYG_TRY(scratch.with_room([&] {
                DYG_TRY(grow_keep(ws.rx2, sizeof(uint32_t) * ncap, sizeof(uint32_t) * used, st));
                DYG_TRY(grow_keep(ws.ry2, sizeof(uint32_t) * ncap, sizeof(uint32_t) * used, st));
                return grow_keep(ws.rk2, ncap, used, st);
            }));
            cap = ncap;
            DYG_CUDA(cudaMemcpyAsync(sc + S_RECCAP, &cap, sizeof(cap), cudaMemcpyHostToDevice, st));
            DYG_CUDA(cudaStreamSynchronize(st));
        } else if (hi.kind == kHaltPaths) {
            scratch.grow_paths(G);
        } else {
            DYG_TRY(scratch.with_room([&] { return grow_arena(H, H->g.arena_cap * 2, st); }));
        }
        DYG_TRY(clear_halt(G, st));
        c_start = hi.batch;
        ph_start = hi.phase;
    }
    set_error("delete file: too many buffer regrowths");
    return DYG_ENOMEM;
}

}  // namespace

uint32_t stream_default_chunk(uint32_t n_vertices) {
    const uint32_t c = (uint32_t)((double)n_vertices * 0.05);
    return c < 10000u ? 10000u : c;
}

dyg_status stream_file_run(dyg_graph *G, dyg_graph *H, uint32_t op, const uint32_t *src,
                           const uint32_t *dst, const float *w, uint32_t n, uint64_t uid0,
                           uint32_t chunk, const dyg_walk_params &p, int32_t *status, float *cond,
                           uint64_t *n_rec, cudaStream_t st, bool check_inputs,
                           const std::function<dyg_status()> *fetch) {
    *n_rec = 0;
    DYG_TRY(check_usable(G, H));
    if (chunk == 0) chunk = stream_default_chunk(G->g.n);
    if (op == DYG_STREAM_INSERT)
        return insert_file_run(G, H, src, dst, w, n, uid0, chunk, p, status, cond, st,
                               check_inputs, fetch);
    return delete_file_run(G, H, src, dst, n, uid0, chunk, p, status, cond, n_rec, st,
                           check_inputs, fetch);
}

}  // namespace dyg
