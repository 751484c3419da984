// rowops.cuh -- device-driven row updates of the dynamic CSR, as phases of a
// cooperative launch (gridsync.cuh).
//
// A list of edges e < n has half-edges i = 2e (the source's row gets the
// target) and i = 2e + 1 (the target's row gets the source).  Both operations
// apply the half-edges of a row in list order without sorting the list:
//   link:    each half-edge pushes itself on its row's chain (one exchange on
//            rowhead, one add on rowcnt); the one that found the chain empty
//            is the row's leader.
//   append:  leaders size their rows and the block that arrives last reserves
//            the arena space of all moves, all or nothing (halting the stream
//            when it does not fit); then each leader moves its row if it
//            overflows, gathers its chain, puts it in list order and writes
//            the tail.  Row order is therefore exactly the order the
//            reference's host loop produces
//            (random_walk_incremental/gpu_graph.cuh:297-329).
//   delete:  each leader gathers its chain, puts it in list order and removes
//            the entries one by one with swap-with-last
//            (random_walk_decremental/gpu_graph.cuh:359-399).
// The work of a row is done by its leader's lane, by a warp, or -- hub rows
// and long chains -- by a block.  Leaders put the rows that are not for their
// lane on a list, which the warps and blocks of the whole grid share out: the
// leaders of hub rows are whichever blocks linked first, so a block keeping
// its own leaders' rows could get most of them (725 us instead of 134 for the
// recoveries of a 4,096-edge R-MAT file).  A chain of more than 32 entries is
// not followed (each link is a dependent load).  Its row gets a run of words:
// the entries of the whole list put themselves into their rows' runs (one more
// pass over the list, and one barrier, where there are such rows), and a warp
// or a block puts the run in order.  Only for chains that do not fit the block's
// shared memory, or in a list of two tiles, does the block scan the list for the
// row's entries, which meets them in order: the scan is of the whole list for
// each row, and with it alone a batch of a million edges of 25,000 rows took
// 273 ms to insert and 159 to delete (with runs 1.29 and 1.98), one of 20,000
// edges of 500 rows 0.66 and 0.69 (0.14 and 0.20).
// Nothing here needs a host-visible count, so a whole update stream is
// enqueued with a single synchronize at its end.
#pragma once

#include "dyg_internal.cuh"
#include "gridsync.cuh"

namespace dyg {

constexpr uint32_t kLaneRow = 32;     // rows up to this length are edited by one lane
constexpr uint32_t kLaneChain = 4;    // ... with up to this many entries
constexpr uint32_t kWarpChain = 32;   // entries of a chain that is followed
constexpr uint32_t kWarpRun = 256;    // entries of a run that a warp puts in order
constexpr uint32_t kSortMax = 4096;   // ... that a block does
constexpr uint32_t kWarpSearch = 4096;   // slots a warp looks at for one row's deletions
constexpr uint32_t kTrackMax = 128;   // deletions of a hub row found in one pass over it

// The chains of one graph's rows.
struct Chains {
    uint32_t *rowcnt, *rowhead;   // per row: entries, last entry + 1 (zero between operations)
    uint32_t *nxt;                // per half-edge: previous entry + 1; ~0u not in the list; a leader:
                                  // 0, or kItem with bits for the graphs whose row is on a list
    uint32_t *list;               // leaders of rows for a block (from the front) and a warp (back)
    unsigned long long *items;    // their numbers: low word, high word
    uint32_t *runs;               // entries of the rows with long chains
    unsigned long long *cursor;   // its next free word (low word), runs to be filled (high word)
};
constexpr uint32_t kItem = 0xFFFFFFF0u;

__device__ __forceinline__ bool is_leader(uint32_t nx) { return nx == 0u || (nx >= kItem && nx != ~0u); }

__device__ __forceinline__ void list_row(uint32_t *list, unsigned long long *items, uint32_t m,
                                         uint32_t i, bool warp) {
    if (warp) list[m - 1u - (uint32_t)(atomicAdd(items, 1ull << 32) >> 32)] = i;
    else list[(uint32_t)atomicAdd(items, 1ull)] = i;
}

// A list of up to this many half-edges is two tiles of scan_entries: cheaper for
// a block than to sort.
constexpr uint32_t kScanHalves = 2u * 2u * 8u * kOpThreads;
// Whether the entries of a row with a long chain put themselves into its run.
__device__ __forceinline__ bool run_filled(uint32_t cnt, uint32_t m) {
    return cnt > kWarpChain && cnt <= kSortMax && (cnt <= kWarpRun || m > kScanHalves);
}
// Room for a long chain; rowhead, whose chain is not followed, gets its start
// (and is its end once the entries are in).
__device__ __forceinline__ void open_run(const Chains &c, uint32_t x, uint32_t cnt, uint32_t m) {
    if (cnt <= kWarpChain) return;
    c.rowhead[x] =
        (uint32_t)atomicAdd(c.cursor, ((unsigned long long)(run_filled(cnt, m) ? 1u : 0u) << 32) + cnt);
}
// Every thread of the grid: its share of the entries into the runs.
template <class Row>
__device__ __forceinline__ void fill_runs(const Chains &c, uint32_t m, Row row) {
    const uint2 rg = block_range(m);
    for (uint32_t i = rg.x + threadIdx.x; i < rg.y; i += blockDim.x) {
        if (c.nxt[i] == ~0u) continue;
        const uint32_t x = row(i);
        if (run_filled(c.rowcnt[x], m)) c.runs[atomicAdd(c.rowhead + x, 1u)] = i;
    }
}
// After that: where the run of a row starts, rowhead being `head`.
__device__ __forceinline__ uint32_t run_start(uint32_t head, uint32_t cnt, uint32_t m) {
    return run_filled(cnt, m) ? head - cnt : head;
}

// Sorts s[0, N) ascending, N a power of two; every thread of the block calls it.
__device__ __forceinline__ void block_sort(uint32_t *s, uint32_t N) {
    for (uint32_t k = 2u; k <= N; k <<= 1)
        for (uint32_t h = k >> 1; h > 0u; h >>= 1) {
            __syncthreads();
            for (uint32_t p = threadIdx.x; p < N / 2u; p += blockDim.x) {
                const uint32_t i = 2u * p - (p & (h - 1u)), o = i + h;
                const uint32_t a = s[i], b = s[o];
                if ((a > b) == ((i & k) == 0u)) {
                    s[i] = b;
                    s[o] = a;
                }
            }
        }
    __syncthreads();
}
// Loads run[0, cnt) (at most kSortMax, distinct) into s and sorts it.
__device__ __forceinline__ void block_load_sorted(const uint32_t *run, uint32_t cnt, uint32_t *s) {
    uint32_t N = 64u;
    while (N < cnt) N <<= 1;
    for (uint32_t j = threadIdx.x; j < N; j += blockDim.x) s[j] = j < cnt ? __ldcg(run + j) : ~0u;
    block_sort(s, N);
}

// A warp's run of up to kWarpRun distinct entries: v[k] is entry 32 k + lane of
// it (~0u past its end), r[k] its rank among all.
struct WarpRun {
    static constexpr uint32_t K = kWarpRun / 32u;
    uint32_t v[K], r[K];
};
__device__ __forceinline__ void warp_rank_run(const uint32_t *run, uint32_t cnt, uint32_t lane, WarpRun &w) {
#pragma unroll
    for (uint32_t k = 0; k < WarpRun::K; ++k) {
        w.v[k] = 32u * k + lane < cnt ? __ldcg(run + 32u * k + lane) : ~0u;
        w.r[k] = 0u;
    }
#pragma unroll
    for (uint32_t g = 0; g < WarpRun::K; ++g) {
        if (32u * g >= cnt) break;
#pragma unroll 8
        for (uint32_t u = 0; u < 32u; ++u) {
            const uint32_t o = __shfl_sync(kFull, w.v[g], u);
#pragma unroll
            for (uint32_t k = 0; k < WarpRun::K; ++k) w.r[k] += o < w.v[k] ? 1u : 0u;
        }
    }
}
// Puts it in order where it is.
__device__ __forceinline__ void warp_sort_run(uint32_t *run, uint32_t cnt, uint32_t lane) {
    WarpRun w;
    warp_rank_run(run, cnt, lane, w);
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < WarpRun::K; ++k)
        if (w.v[k] != ~0u) run[w.r[k]] = w.v[k];
    __syncwarp();
}

struct EdgeList {
    const uint32_t *src, *dst;
    const float *w;
};

struct AppSide {
    DevGraph g;
    Chains c;
    EdgeList E;
    uint32_t slack;
    unsigned long long *sc;   // the graph's scalars
};
struct AppSides {
    AppSide s[2];
    uint32_t n;   // sides used
};

struct RowItem {
    uint32_t x, cnt, head, old_off, deg, off;
};

// Edges each thread looks at per tile of scan_entries.
constexpr uint32_t kScanEdges = 8;
static_assert(kScanHalves == 2u * 2u * kScanEdges * kOpThreads, "two tiles");

// Shared memory of the row phases.
struct RowShared {
    union {
        RowItem item[kOpThreads];   // candidates whose rows the block searches (k_recover)
        uint32_t sort[kSortMax];    // a run being put in order
    };
    uint32_t nbig;
    uint32_t warp[kOpThreads / 32 + 1];
    uint32_t tile[kScanEdges * kOpThreads / 32 + 1];
    RowItem row;                    // the block's item
    uint32_t chain[kWarpChain];     // its entries in list order, if it has no run
    // hub-row deletions
    uint32_t best, ok, nlive;
    uint32_t y[kTrackMax], pos[kTrackMax], occ[kTrackMax];
    unsigned long long key[kTrackMax];
};

__device__ __forceinline__ void link_entry(const Chains &c, uint32_t i, uint32_t x, bool on) {
    uint32_t nx = ~0u;
    if (on) {
        nx = atomicExch(c.rowhead + x, i + 1u);
        atomicAdd(c.rowcnt + x, 1u);
    }
    c.nxt[i] = nx;
}

__device__ __forceinline__ uint32_t entry_row(const EdgeList &E, uint32_t i) {
    return (i & 1u) ? E.dst[i >> 1] : E.src[i >> 1];
}
__device__ __forceinline__ uint32_t entry_col(const EdgeList &E, uint32_t i) {
    return (i & 1u) ? E.src[i >> 1] : E.dst[i >> 1];
}

// Arena slots row x needs to take cnt more entries; 0 if they fit where it is.
__device__ __forceinline__ uint32_t move_need(uint32_t deg, uint32_t cnt, uint32_t cap,
                                              uint32_t slack) {
    const uint32_t nd = deg + cnt;
    if (nd <= cap) return 0u;
    const uint32_t need = max(2u * nd, nd + slack);
    return (need + 1u) & ~1u;
}

// ------------------------------------------------------------------ append

// Leaders add up the arena slots their rows' moves need and list the rows
// that are not for their lane.
__device__ __forceinline__ void app_need(const AppSide &a, uint32_t m,
                                         unsigned long long *s_need) {
    const uint2 r = block_range(m);
    unsigned long long mine = 0ull;
    for (uint32_t i = r.x + threadIdx.x; i < r.y; i += blockDim.x) {
        if (a.c.nxt[i] != 0u) continue;
        const uint32_t x = entry_row(a.E, i);
        const uint32_t deg = a.g.desc[x].y, cnt = a.c.rowcnt[x];
        const uint32_t need = move_need(deg, cnt, a.g.cap[x], a.slack);
        mine += need;
        if (cnt > kLaneChain || (need && deg > kLaneRow)) {
            a.c.nxt[i] = kItem;
            open_run(a.c, x, cnt, m);
            list_row(a.c.list, a.c.items, m, i, cnt <= kWarpRun && (!need || deg <= kBigRow));
        }
    }
    if (threadIdx.x == 0) *s_need = 0ull;
    __syncthreads();
    if (mine) atomicAdd(s_need, mine);
    __syncthreads();
    if (threadIdx.x == 0 && *s_need) atomicAdd(a.sc + S_NEED, *s_need);
}

// Reserves the moves of all sides, all or nothing, or halts.  One thread.
__device__ __forceinline__ bool reserve_moves(const AppSides &A, unsigned long long *halt,
                                              unsigned long long code) {
    bool ok = true;
    for (uint32_t k = 0; k < A.n; ++k)
        ok &= *A.s[k].g.top + __ldcg(A.s[k].sc + S_NEED) <= A.s[k].g.arena_cap;
    for (uint32_t k = 0; k < A.n; ++k) {
        unsigned long long *sc = A.s[k].sc;
        const unsigned long long need = __ldcg(sc + S_NEED);
        if (ok) {
            sc[S_CURSOR] = *A.s[k].g.top;
            *A.s[k].g.top += need;
        }
        sc[S_NEED] = 0ull;
    }
    if (!ok) *halt = code;
    return ok;
}

// Slots [from, from + deg) to [to, to + deg) by `nt` threads of rank t.  The
// ranges never overlap (a row moves to fresh arena space), so U slots per
// thread are loaded before they are stored.
template <uint32_t U>
__device__ __forceinline__ void copy_row(const DevGraph &g, uint32_t from, uint32_t to,
                                         uint32_t deg, uint32_t t, uint32_t nt) {
    for (uint32_t j0 = 0; j0 < deg; j0 += U * nt) {
        uint2 sv[U];
        float wv[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t j = j0 + u * nt + t;
            if (j < deg) {
                sv[u] = g.slots[from + j];
                wv[u] = g.wts[from + j];
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t j = j0 + u * nt + t;
            if (j < deg) {
                g.slots[to + j] = sv[u];
                g.wts[to + j] = wv[u];
            }
        }
    }
}

__device__ __forceinline__ void put_slot(const DevGraph &g, uint32_t at, uint32_t y, float w) {
    g.slots[at] = make_uint2(y, __float_as_uint(__frcp_rn(w)));
    g.wts[at] = w;
}

__device__ __forceinline__ void publish_row(const AppSide &a, uint32_t x, uint32_t off,
                                            uint32_t deg, uint32_t cnt, uint32_t need) {
    a.g.desc[x] = make_uint2(off, deg + cnt);
    if (need) a.g.cap[x] = need;
    if (deg + cnt > kBigRow && deg <= kBigRow) a.sc[S_LONG] = 1ull;
}

// The whole block calls back(k, i) for the k-th of cnt half-edges i, in list
// order, that hits(e) names: bit 0 for edge e's first half-edge, bit 1 for its
// second.  The n edges are read kScanEdges per thread at a time, all loads
// issued together (a 20,000-edge list: five tiles).
template <class Hits, class Back>
__device__ __forceinline__ void scan_entries(uint32_t n, uint32_t cnt, RowShared &s, Hits hits, Back back) {
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t nw = blockDim.x >> 5;
    uint32_t run = 0;
    for (uint32_t t0 = 0; t0 < n && run < cnt; t0 += kScanEdges * blockDim.x) {
        uint32_t on = 0u;   // bits 2u, 2u + 1: the half-edges of edge u
#pragma unroll
        for (uint32_t u = 0; u < kScanEdges; ++u) {
            const uint32_t e = t0 + u * blockDim.x + threadIdx.x;
            if (e < n) on |= hits(e) << (2u * u);
        }
        uint32_t before[kScanEdges];   // of this edge row, in this warp's earlier lanes
#pragma unroll
        for (uint32_t u = 0; u < kScanEdges; ++u) {
            const uint32_t m0 = __ballot_sync(kFull, (on >> (2u * u)) & 1u);
            const uint32_t m1 = __ballot_sync(kFull, (on >> (2u * u + 1u)) & 1u);
            const uint32_t lt = (1u << lane) - 1u;
            before[u] = __popc(m0 & lt) + __popc(m1 & lt);
            if (lane == 0u) s.tile[u * nw + wid] = __popc(m0) + __popc(m1);
        }
        __syncthreads();
        if (wid == 0u) {   // exclusive scan of the kScanEdges * nw counts
            uint32_t carry = 0u;
            for (uint32_t q = 0; q < kScanEdges * nw; q += 32u) {
                const uint32_t v = q + lane < kScanEdges * nw ? s.tile[q + lane] : 0u;
                uint32_t incl = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(kFull, incl, o);
                    if (lane >= (uint32_t)o) incl += t;
                }
                if (q + lane < kScanEdges * nw) s.tile[q + lane] = carry + incl - v;
                carry += __shfl_sync(kFull, incl, 31);
            }
            if (lane == 0u) s.tile[kScanEdges * nw] = carry;
        }
        __syncthreads();
        if (on) {
#pragma unroll
            for (uint32_t u = 0; u < kScanEdges; ++u) {
                const uint32_t e = t0 + u * blockDim.x + threadIdx.x;
                uint32_t k = run + s.tile[u * nw + wid] + before[u];
                if ((on >> (2u * u)) & 1u) back(k++, 2u * e);
                if ((on >> (2u * u + 1u)) & 1u) back(k, 2u * e + 1u);
            }
        }
        run += s.tile[kScanEdges * nw];
        __syncthreads();   // s.tile is written again by the next tile
    }
}

// The half-edges of row x in a list whose edges' rows are rows(e).
template <class Rows, class Back>
__device__ __forceinline__ void scan_row(const Chains &c, uint32_t m, uint32_t x, uint32_t cnt, RowShared &s,
                                         Rows rows, Back back) {
    scan_entries(
        m >> 1, cnt, s,
        [&](uint32_t e) {
            const uint2 nx = reinterpret_cast<const uint2 *>(c.nxt)[e];
            const uint2 v = rows(e);
            return ((nx.x != ~0u && v.x == x) ? 1u : 0u) | ((nx.y != ~0u && v.y == x) ? 2u : 0u);
        },
        back);
}

// A chain of up to kWarpChain entries followed by warp 0 of the block; each
// lane's entry goes to its rank in `out`.
__device__ __forceinline__ void block_order_chain(const uint32_t *nxt, uint32_t head, uint32_t cnt, uint32_t *out) {
    if (threadIdx.x < 32u) {
        uint32_t mine = ~0u, k = head;
        for (uint32_t u = 0; u < cnt; ++u) {
            if (threadIdx.x == u) mine = k - 1u;
            k = nxt[k - 1u];
        }
        uint32_t r = 0;
        for (uint32_t u = 0; u < cnt; ++u) r += __shfl_sync(kFull, mine, u) < mine ? 1u : 0u;
        if (threadIdx.x < cnt) out[r] = mine;
    }
    __syncthreads();
}

// Row of leader i with its chain taken off, its space allocated.
__device__ __forceinline__ RowItem app_take(const AppSide &a, uint32_t i, uint32_t *need) {
    RowItem it{};
    it.x = entry_row(a.E, i);
    it.cnt = a.c.rowcnt[it.x];
    it.head = a.c.rowhead[it.x];
    const uint2 d = a.g.desc[it.x];
    *need = move_need(d.y, it.cnt, a.g.cap[it.x], a.slack);
    it.old_off = d.x;
    it.deg = d.y;
    it.off = *need ? (uint32_t)atomicAdd(a.sc + S_CURSOR, (unsigned long long)*need) : d.x;
    a.c.rowcnt[it.x] = 0u;
    a.c.rowhead[it.x] = 0u;
    return it;
}

// After a halt: the chains taken off.  Every thread of the grid calls it.
__device__ __forceinline__ void app_clear(const AppSide &a, uint32_t m) {
    const uint2 rg = block_range(m);
    for (uint32_t i = rg.x + threadIdx.x; i < rg.y; i += blockDim.x)
        if (is_leader(a.c.nxt[i])) {
            const uint32_t x = entry_row(a.E, i);
            a.c.rowcnt[x] = 0u;
            a.c.rowhead[x] = 0u;
        }
}

// Moves, fills and publishes the rows that are for their leader's lane.  Every
// thread of the grid calls it.
__device__ __forceinline__ void app_lane_rows(const AppSide &a, uint32_t m) {
    const uint2 rg = block_range(m);
    for (uint32_t i = rg.x + threadIdx.x; i < rg.y; i += blockDim.x) {
        if (a.c.nxt[i] != 0u) continue;
        uint32_t need;
        const RowItem it = app_take(a, i, &need);
        if (need) copy_row<4>(a.g, it.old_off, it.off, it.deg, 0u, 1u);
        // the chain at once, then each entry to its rank among the (distinct)
        // list indices
        uint32_t idx[kLaneChain], y[kLaneChain];
        float w[kLaneChain];
        uint32_t k = it.head;
#pragma unroll
        for (uint32_t u = 0; u < kLaneChain; ++u)
            if (u < it.cnt) {
                idx[u] = k - 1u;
                k = a.c.nxt[k - 1u];
            }
#pragma unroll
        for (uint32_t u = 0; u < kLaneChain; ++u)
            if (u < it.cnt) {
                y[u] = entry_col(a.E, idx[u]);
                w[u] = a.E.w[idx[u] >> 1];
            }
#pragma unroll
        for (uint32_t u = 0; u < kLaneChain; ++u)
            if (u < it.cnt) {
                uint32_t r = 0;
#pragma unroll
                for (uint32_t v = 0; v < kLaneChain; ++v)
                    if (v < it.cnt) r += idx[v] < idx[u] ? 1u : 0u;
                put_slot(a.g, it.off + it.deg + r, y[u], w[u]);
            }
        publish_row(a, it.x, it.off, it.deg, it.cnt, need);
    }
}

// The listed rows, shared out over the grid's warps and blocks (runs filled).
// Not inlined: a batch that has no such rows is a few microseconds, some of them
// the fetch of its instructions.
static __device__ __noinline__ void app_listed_rows(const AppSide &a, unsigned long long items, uint32_t m, RowShared &s) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n_block = (uint32_t)items, n_warp = (uint32_t)(items >> 32);
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    // warp q of block 0, then of block 1, ...: a short list still spreads
    for (uint32_t q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; q < n_warp; q += warps) {
        uint32_t need = 0u;
        RowItem it{};
        if (lane == 0u) it = app_take(a, a.c.list[m - 1u - q], &need);
        it.x = __shfl_sync(kFull, it.x, 0);
        it.cnt = __shfl_sync(kFull, it.cnt, 0);
        it.old_off = __shfl_sync(kFull, it.old_off, 0);
        it.deg = __shfl_sync(kFull, it.deg, 0);
        it.off = __shfl_sync(kFull, it.off, 0);
        it.head = __shfl_sync(kFull, it.head, 0);
        if (it.off != it.old_off) copy_row<4>(a.g, it.old_off, it.off, it.deg, lane, 32u);
        if (it.cnt <= kWarpChain) {
            uint32_t mine = ~0u, k = it.head;
            for (uint32_t u = 0; u < it.cnt; ++u) {   // the chain: one load for the whole warp each
                if (lane == u) mine = k - 1u;
                k = a.c.nxt[k - 1u];
            }
            uint32_t r = 0;
            for (uint32_t u = 0; u < it.cnt; ++u) r += __shfl_sync(kFull, mine, u) < mine ? 1u : 0u;
            if (lane < it.cnt)
                put_slot(a.g, it.off + it.deg + r, entry_col(a.E, mine), a.E.w[mine >> 1]);
        } else {
            WarpRun w;
            warp_rank_run(a.c.runs + run_start(it.head, it.cnt, m), it.cnt, lane, w);
#pragma unroll
            for (uint32_t k = 0; k < WarpRun::K; ++k)
                if (w.v[k] != ~0u)
                    put_slot(a.g, it.off + it.deg + w.r[k], entry_col(a.E, w.v[k]), a.E.w[w.v[k] >> 1]);
        }
        if (lane == 0u) publish_row(a, it.x, it.off, it.deg, it.cnt, need);
    }
    for (uint32_t q = blockIdx.x; q < n_block; q += gridDim.x) {
        __syncthreads();   // the item before is done with s.row
        uint32_t need = 0u;
        if (threadIdx.x == 0) s.row = app_take(a, a.c.list[q], &need);
        __syncthreads();
        const RowItem it = s.row;
        if (it.off != it.old_off) copy_row<4>(a.g, it.old_off, it.off, it.deg, threadIdx.x, blockDim.x);
        const uint32_t to = it.off + it.deg;
        // a link costs a fifth of a tile of the list
        if (it.cnt <= kWarpChain && it.cnt * (uint64_t)kScanHalves < 10ull * m) {
            block_order_chain(a.c.nxt, it.head, it.cnt, s.chain);
            if (threadIdx.x < it.cnt) {
                const uint32_t j = s.chain[threadIdx.x];
                put_slot(a.g, to + threadIdx.x, entry_col(a.E, j), a.E.w[j >> 1]);
            }
        } else if (run_filled(it.cnt, m)) {
            block_load_sorted(a.c.runs + run_start(it.head, it.cnt, m), it.cnt, s.sort);
            for (uint32_t k = threadIdx.x; k < it.cnt; k += blockDim.x) {
                const uint32_t j = s.sort[k];
                put_slot(a.g, to + k, entry_col(a.E, j), a.E.w[j >> 1]);
            }
        } else {
            scan_row(
                a.c, m, it.x, it.cnt, s, [&](uint32_t e) { return make_uint2(a.E.src[e], a.E.dst[e]); },
                [&](uint32_t k, uint32_t j) { put_slot(a.g, to + k, entry_col(a.E, j), a.E.w[j >> 1]); });
        }
        if (threadIdx.x == 0) publish_row(a, it.x, it.off, it.deg, it.cnt, need);
    }
}

// Sizing, reservation and rows of an append whose m half-edges are linked and
// whose row lists are empty.  on_reserve runs in one thread once the space is
// reserved.  False: the barrier gave up.
template <class F>
__device__ __forceinline__ bool app_commit(const AppSides &A, uint32_t m, const GridBar &bar,
                                           unsigned long long *halt, unsigned long long code,
                                           RowShared &s, F on_reserve) {
    __shared__ unsigned long long s_need;
    for (uint32_t k = 0; k < A.n; ++k) {
        app_need(A.s[k], m, &s_need);
        __syncthreads();
    }
    if (!grid_sync(bar, [&] {
            if (reserve_moves(A, halt, code)) on_reserve();
        }))
        return false;
    // read beside the halt word, not after it and after the lanes' rows
    unsigned long long items[2], filled[2];
#pragma unroll
    for (uint32_t k = 0; k < 2u; ++k) {
        items[k] = k < A.n ? __ldcg(A.s[k].c.items) : 0ull;
        filled[k] = k < A.n ? __ldcg(A.s[k].c.cursor) >> 32 : 0ull;
    }
    if (*(volatile unsigned long long *)halt == code) {
        for (uint32_t k = 0; k < A.n; ++k) app_clear(A.s[k], m);
        return true;
    }
    for (uint32_t k = 0; k < A.n; ++k) app_lane_rows(A.s[k], m);
    if (filled[0] | filled[1]) {
#pragma unroll
        for (uint32_t k = 0; k < 2u; ++k)
            if (filled[k]) {
                const AppSide &a = A.s[k];
                fill_runs(a.c, m, [&](uint32_t i) { return entry_row(a.E, i); });
            }
        if (!grid_sync(bar)) return false;
    }
#pragma unroll
    for (uint32_t k = 0; k < 2u; ++k)
        if (items[k]) app_listed_rows(A.s[k], items[k], m, s);
    return true;
}

// ------------------------------------------------------------------ delete

// Endpoints of deletion e: min -> max (random_walk_decremental/gpu_graph.cuh:340-343).
__device__ __forceinline__ uint2 del_ends(const uint32_t *src, const uint32_t *dst, uint32_t e) {
    const uint32_t a = src[e], b = dst[e];
    return make_uint2(min(a, b), max(a, b));
}

struct DelList {
    Chains c;
    const uint32_t *src, *dst;   // as given
    uint32_t *list_h;            // listed rows of H (c.list, c.items: of G)
    unsigned long long *items_h;
};

__device__ __forceinline__ uint32_t del_row(const DelList &D, uint32_t i) {
    const uint2 v = del_ends(D.src, D.dst, i >> 1);
    return (i & 1u) ? v.y : v.x;
}
__device__ __forceinline__ uint32_t del_col(const DelList &D, uint32_t i) {
    const uint2 v = del_ends(D.src, D.dst, i >> 1);
    return (i & 1u) ? v.x : v.y;
}

// Whether entry k is to be applied: with a mask, only if its edge was found
// on both sides of it.
__device__ __forceinline__ bool del_on(const uint8_t *mask, uint32_t k) {
    return !mask || (mask[k & ~1u] && mask[k | 1u]);
}

// The row's last slot into the hole at `pos`.
__device__ __forceinline__ void del_swap(const DevGraph &g, uint32_t off, uint32_t pos,
                                         uint32_t deg) {
    g.slots[off + pos] = g.slots[off + deg - 1u];
    g.wts[off + pos] = g.wts[off + deg - 1u];
}

// One block removes a hub row's entries (or a long chain's).  They are put in
// list order (a long chain's in its run, once for both graphs: `in_order`), then
// taken kTrackMax at a time: when a group's columns
// are distinct and each occurs at most once in the row, one pass over the row
// finds every target's slot and one thread applies the swaps in order,
// following the single slot each swap moves (the row's last); otherwise every
// deletion of the group is a block-wide search.  Both give what removing them
// one by one gives.
__device__ inline void block_del_row(const DevGraph &g, const DelList &D, uint32_t m, uint32_t x,
                              uint32_t cnt, uint32_t head, bool in_order, const uint8_t *mask,
                              uint8_t *found, RowShared &s) {
    const uint32_t *sorted = s.chain;
    if (cnt <= kWarpChain) {
        block_order_chain(D.c.nxt, head, cnt, s.chain);
    } else {
        uint32_t *run = D.c.runs + run_start(head, cnt, m);
        sorted = run;
        if (!in_order && run_filled(cnt, m)) {
            block_load_sorted(run, cnt, s.sort);
            for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) run[k] = s.sort[k];
        } else if (!in_order) {
            scan_row(
                D.c, m, x, cnt, s, [&](uint32_t e) { return del_ends(D.src, D.dst, e); },
                [&](uint32_t k, uint32_t j) { run[k] = j; });
        }
    }
    __syncthreads();
    const uint2 d = g.desc[x];
    uint32_t deg = d.y;
    for (uint32_t g0 = 0; g0 < cnt; g0 += kTrackMax) {
        const uint32_t gc = min(kTrackMax, cnt - g0);
        const uint32_t *grp = sorted + g0;
        if (threadIdx.x == 0) {
            s.ok = 1u;
            s.nlive = 0u;
        }
        __syncthreads();
        for (uint32_t a = threadIdx.x; a < gc; a += blockDim.x) {
            const bool on = del_on(mask, grp[a]);
            s.y[a] = on ? del_col(D, grp[a]) : ~0u;
            s.pos[a] = ~0u;
            s.occ[a] = 0u;
            if (on) atomicAdd(&s.nlive, 1u);
        }
        __syncthreads();
        const uint32_t nlive = s.nlive;   // masked-off entries (column ~0u) sort last
        // the group's columns sorted (rank by count, ties by index), so each
        // slot of the row finds its deletion by binary search
        for (uint32_t a = threadIdx.x; a < gc; a += blockDim.x) {
            const unsigned long long ka = ((unsigned long long)s.y[a] << 8) | a;
            uint32_t r = 0;
            for (uint32_t c = 0; c < gc; ++c) {
                const unsigned long long kc = ((unsigned long long)s.y[c] << 8) | c;
                r += kc < ka;
                if (c < a && s.y[a] != ~0u && s.y[c] == s.y[a]) s.ok = 0u;
            }
            s.key[r] = ka;
        }
        __syncthreads();
        const uint32_t *cols = reinterpret_cast<const uint32_t *>(g.slots + d.x);
        if (s.ok && nlive) {
            for (uint32_t base = 0; base < deg; base += kFindUnroll * blockDim.x) {
                uint32_t v[kFindUnroll];   // a tile's loads are issued before any search
#pragma unroll
                for (uint32_t u = 0; u < kFindUnroll; ++u) {
                    const uint32_t j = base + u * blockDim.x + threadIdx.x;
                    v[u] = j < deg ? cols[2u * j] : ~0u;
                }
#pragma unroll
                for (uint32_t u = 0; u < kFindUnroll; ++u) {
                    const uint32_t col = v[u];
                    if (col == ~0u) continue;
                    uint32_t lo = 0, hi = nlive;
                    while (lo < hi) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if ((uint32_t)(s.key[mid] >> 8) < col) lo = mid + 1u;
                        else hi = mid;
                    }
                    if (lo < nlive && (uint32_t)(s.key[lo] >> 8) == col) {
                        const uint32_t a = (uint32_t)(s.key[lo] & 0xFFu);
                        atomicMin(&s.pos[a], base + u * blockDim.x + threadIdx.x);
                        atomicAdd(&s.occ[a], 1u);
                    }
                }
            }
        }
        __syncthreads();
        for (uint32_t a = threadIdx.x; a < gc; a += blockDim.x)
            if (s.occ[a] > 1u) s.ok = 0u;
        __syncthreads();
        if (s.ok) {
            if (threadIdx.x == 0) {
                for (uint32_t a = 0; a < gc; ++a) {
                    const uint32_t p = s.pos[a];
                    if (s.y[a] == ~0u || p == ~0u) continue;
                    const uint32_t last = deg - 1u;
                    del_swap(g, d.x, p, deg);
                    --deg;
                    found[grp[a]] = 1;
                    if (p != last)   // the slot from `last` now sits at p
                        for (uint32_t c = a + 1; c < gc; ++c)
                            if (s.pos[c] == last) s.pos[c] = p;
                }
                s.best = deg;
            }
            __syncthreads();
            deg = s.best;
            __syncthreads();   // block_find and the next group write s.best
        } else {
            for (uint32_t a = 0; a < gc; ++a) {
                if (s.y[a] == ~0u) continue;
                const uint32_t j = block_find(g.slots, d.x, deg, s.y[a], &s.best);
                if (j != ~0u) {
                    if (threadIdx.x == 0) {
                        del_swap(g, d.x, j, deg);
                        found[grp[a]] = 1;
                    }
                    --deg;
                    __syncthreads();   // the moved slot is visible to the next search
                }
            }
        }
        __syncthreads();   // every thread is done with the group's shared words
    }
    if (threadIdx.x == 0) g.desc[x] = make_uint2(d.x, deg);
    __syncthreads();
}

// One warp removes a row's entries (at most kWarpRun), searching the row once per
// deletion, 256 slots at a time.
__device__ __forceinline__ void warp_del_row(const DevGraph &g, const DelList &D, uint32_t m, const RowItem &it,
                                             bool in_order, const uint8_t *mask, uint8_t *found, uint32_t lane) {
    uint32_t *run = nullptr;
    uint32_t mine = ~0u;   // the lane's entry of 32 in list order
    if (it.cnt > kWarpChain) {
        run = D.c.runs + run_start(it.head, it.cnt, m);
        if (!in_order) warp_sort_run(run, it.cnt, lane);
    } else {
        uint32_t k = it.head, own = ~0u;
        for (uint32_t u = 0; u < it.cnt; ++u) {
            if (lane == u) own = k - 1u;
            k = D.c.nxt[k - 1u];
        }
        uint32_t rank = 0;
        for (uint32_t u = 0; u < it.cnt; ++u) rank += __shfl_sync(kFull, own, u) < own ? 1u : 0u;
        for (uint32_t u = 0; u < it.cnt; ++u) {
            const uint32_t v = __shfl_sync(kFull, own, u);
            if (__shfl_sync(kFull, rank, u) == lane) mine = v;
        }
    }
    const uint32_t off = it.old_off;
    uint32_t deg = it.deg;
    for (uint32_t g0 = 0; g0 < it.cnt; g0 += 32u) {
        const uint32_t gc = min(32u, it.cnt - g0);
        if (run) mine = lane < gc ? run[g0 + lane] : ~0u;
        const uint32_t my_y = lane < gc ? del_col(D, mine) : 0u;
        const bool my_on = lane < gc && del_on(mask, mine);
        for (uint32_t a = 0; a < gc; ++a) {
            if (!__shfl_sync(kFull, my_on ? 1u : 0u, a)) continue;
            const uint32_t y = __shfl_sync(kFull, my_y, a);
            uint32_t pos = ~0u;
            for (uint32_t j0 = 0; j0 < deg && pos == ~0u; j0 += 256u) {
                uint32_t cv[8];
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u) {
                    const uint32_t j = j0 + 32u * u + lane;
                    cv[u] = j < deg ? g.slots[off + j].x : ~0u;   // vertex ids are never ~0u
                }
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u) {
                    const unsigned hit = __ballot_sync(kFull, cv[u] == y);
                    if (hit && pos == ~0u) pos = j0 + 32u * u + (uint32_t)(__ffs(hit) - 1);
                }
            }
            if (pos != ~0u) {
                if (lane == a) {
                    del_swap(g, off, pos, deg);
                    found[mine] = 1;
                }
                --deg;
                __syncwarp();   // the moved slot is visible to the next search
            }
        }
    }
    if (lane == 0u && deg != it.deg) g.desc[it.x] = make_uint2(off, deg);
    __syncwarp();
}

// How a row's cnt deletions are done.  A warp searches the row once per
// deletion, 256 slots at a time: for one row that is worth it up to kWarpSearch
// slots looked at in all, in a list that may have hundreds of such rows up to
// kWarpRun searches (a million deletions of 10,000 rows 6.28 -> 2.00 ms, 20,000
// of 200 rows 0.57 -> 0.26).
__device__ __forceinline__ bool del_by_lane(uint32_t deg, uint32_t cnt) {
    return cnt <= kLaneChain && deg <= kLaneRow;
}
__device__ __forceinline__ bool del_by_warp(uint32_t deg, uint32_t cnt, uint32_t m) {
    return cnt <= kWarpRun && ((uint64_t)deg * cnt <= kWarpSearch ||
                               (m > kScanHalves && (uint64_t)((deg + 255u) >> 8) * cnt <= kWarpRun));
}

// Leaders list the rows of G (bit 1 of the mark) and of H (bit 2) that are
// not for their lane.
__device__ __forceinline__ void del_list(const DevGraph &G, const DevGraph &H, const DelList &D,
                                         uint32_t m) {
    const uint2 rg = block_range(m);
    for (uint32_t i = rg.x + threadIdx.x; i < rg.y; i += blockDim.x) {
        if (D.c.nxt[i] != 0u) continue;
        const uint32_t x = del_row(D, i), cnt = D.c.rowcnt[x];
        const uint32_t dg = G.desc[x].y, dh = H.desc[x].y;
        uint32_t mark = 0u;
        if (!del_by_lane(dg, cnt)) {
            mark |= 1u;
            list_row(D.c.list, D.c.items, m, i, del_by_warp(dg, cnt, m));
        }
        if (!del_by_lane(dh, cnt)) {
            mark |= 2u;
            list_row(D.list_h, D.items_h, m, i, del_by_warp(dh, cnt, m));
        }
        if (!mark) continue;
        D.c.nxt[i] = kItem | mark;
        open_run(D.c, x, cnt, m);   // a long chain's row is on both lists
    }
}

// The rows of g that are for their leader's lane: entries removed in list
// order (mask as in del_on); found[i] = 1 for each entry that was there.
// `bit`: the graph's mark.
__device__ __forceinline__ void del_lane_rows(const DevGraph &g, const DelList &D, uint32_t m,
                                              uint32_t bit, const uint8_t *mask, uint8_t *found,
                                              bool clear) {
    const uint2 rg = block_range(m);
    for (uint32_t i = rg.x + threadIdx.x; i < rg.y; i += blockDim.x) {
        const uint32_t nx = D.c.nxt[i];
        if (!is_leader(nx) || (nx & bit)) continue;
        const uint32_t x = del_row(D, i), cnt = D.c.rowcnt[x], head = D.c.rowhead[x];
        const uint2 d = g.desc[x];
        uint32_t idx[kLaneChain];
        uint32_t k = head;
#pragma unroll
        for (uint32_t u = 0; u < kLaneChain; ++u) {
            idx[u] = ~0u;
            if (u < cnt) {
                idx[u] = k - 1u;
                k = D.c.nxt[k - 1u];
            }
        }
        uint32_t deg = d.y, from = 0u;
        for (uint32_t a = 0; a < cnt; ++a) {
            k = ~0u;   // the next entry in list order
#pragma unroll
            for (uint32_t u = 0; u < kLaneChain; ++u)
                if (idx[u] >= from) k = min(k, idx[u]);
            from = k + 1u;
            if (!del_on(mask, k)) continue;
            const uint32_t y = del_col(D, k);
            // first slot holding y, eight columns loaded before they are
            // compared (vertex ids are never ~0u)
            uint32_t pos = ~0u;
            for (uint32_t j0 = 0; j0 < deg && pos == ~0u; j0 += 8u) {
                uint32_t cv[8];
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u)
                    cv[u] = j0 + u < deg ? g.slots[d.x + j0 + u].x : ~0u;
#pragma unroll
                for (uint32_t u = 0; u < 8u; ++u)
                    if (pos == ~0u && cv[u] == y) pos = j0 + u;
            }
            if (pos != ~0u) {
                del_swap(g, d.x, pos, deg);
                --deg;
                found[k] = 1;
            }
        }
        if (deg != d.y) g.desc[x] = make_uint2(d.x, deg);
        if (clear) {
            D.c.rowcnt[x] = 0u;
            D.c.rowhead[x] = 0u;
        }
    }
}

// The listed rows of g, shared out over the grid's warps and blocks.
__device__ __forceinline__ void del_listed_rows(const DevGraph &g, const DelList &D,
                                                const uint32_t *list, unsigned long long items,
                                                uint32_t m, bool in_order, const uint8_t *mask,
                                                uint8_t *found, bool clear, RowShared &s) {
    const uint32_t n_block = (uint32_t)items, n_warp = (uint32_t)(items >> 32);
    const uint32_t lane = threadIdx.x & 31u, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; q < n_warp; q += warps) {
        const uint32_t x = del_row(D, list[m - 1u - q]);
        const uint2 d = g.desc[x];
        const RowItem it{x, D.c.rowcnt[x], D.c.rowhead[x], d.x, d.y, 0u};
        __syncwarp();
        if (lane == 0u && clear) {
            D.c.rowcnt[x] = 0u;
            D.c.rowhead[x] = 0u;
        }
        warp_del_row(g, D, m, it, in_order, mask, found, lane);
    }
    for (uint32_t q = blockIdx.x; q < n_block; q += gridDim.x) {
        const uint32_t x = del_row(D, list[q]);
        const uint32_t cnt = D.c.rowcnt[x], head = D.c.rowhead[x];
        __syncthreads();
        if (threadIdx.x == 0 && clear) {
            D.c.rowcnt[x] = 0u;
            D.c.rowhead[x] = 0u;
        }
        block_del_row(g, D, m, x, cnt, head, in_order, mask, found, s);
    }
}

// ------------------------------------------------------------- append kernel

// One launch per commit: op.take(e) decides edge e (and writes its results),
// bit k of its value appending the edge to side k; edges whose op.listed(e)
// holds go to op.list(e, q) in list order, op.total(n) getting their number.
//   uint32_t count()                  edges (device or host count)
//   uint32_t take(uint32_t e)
//   static constexpr bool kList       whether take's bit 0 also lists the edge
//   static constexpr bool kPrep       whether something may come before all this:
//   bool pending()                    what, read beside the halt word; if so
//   bool prep(bar, s)                 every thread of the grid does it (false: the
//                                     barrier gave up)
template <class Op>
__global__ void __launch_bounds__(kOpThreads, 2)
k_append(const __grid_constant__ Op op, const __grid_constant__ AppSides A, uint32_t *blk, unsigned long long *work,
         unsigned long long *halt, unsigned long long code, GridBar bar) {
    __shared__ RowShared s;
    bool pending = false;
    if constexpr (Op::kPrep) pending = op.pending();
    if (*halt) return;
    if constexpr (Op::kPrep)
        if (pending && !op.prep(bar, s)) return;
    const uint32_t n = op.count();
    const uint2 rg = block_range(n);
    uint32_t mine = 0u;
    for (uint32_t e = rg.x + threadIdx.x; e < rg.y; e += blockDim.x) {
        const uint32_t take = op.take(e);
        mine += take & 1u;
        for (uint32_t k = 0; k < A.n; ++k) {
            const AppSide &a = A.s[k];
            const uint32_t u = a.E.src[e], v = a.E.dst[e];
            const bool on = (take >> k) & 1u;
            link_entry(a.c, 2u * e, u, on && u < a.g.n);
            link_entry(a.c, 2u * e + 1u, v, on && v < a.g.n);
        }
    }
    if (work && blockIdx.x == 0 && threadIdx.x == 0) *work = 0ull;   // the next walk's chunk counter
    if constexpr (Op::kList) {
        const uint32_t sum = block_sum(mine, s.warp);
        if (threadIdx.x == 0) blk[blockIdx.x] = sum;
    }
    if (!grid_sync(bar, [&] {
            for (uint32_t k = 0; k < A.n; ++k) *A.s[k].c.items = *A.s[k].c.cursor = 0ull;
        }))
        return;
    if constexpr (Op::kList) {
        uint32_t base = blocks_before(blk, s.warp).x;
        for (uint32_t t = rg.x; t < rg.y; t += blockDim.x) {
            const uint32_t e = t + threadIdx.x;
            const uint32_t v = e < rg.y && op.listed(e) ? 1u : 0u;
            uint32_t total;
            const uint32_t q = base + block_excl(v, s.warp, &total);
            if (v) op.list(e, q);
            base += total;
        }
        if (blockIdx.x == gridDim.x - 1u && threadIdx.x == 0) op.total(base);
    }
    app_commit(A, 2u * n, bar, halt, code, s, [] {});
}

// Workspace of a row operation on up to m half-edges (cleared on st).
dyg_status rowops_ensure(dyg_graph *G, uint64_t m, cudaStream_t st);
GridBar grid_bar(dyg_graph *G, unsigned long long *halt);
AppSide append_side(dyg_graph *G, const uint32_t *src, const uint32_t *dst, const float *w);

template <class Op>
dyg_status append_enqueue(const Op &op, uint32_t n_host, dyg_graph *GA, const EdgeList &EA,
                          dyg_graph *GB, const EdgeList &EB, unsigned long long *work,
                          unsigned long long *halt, unsigned long long code, cudaStream_t st) {
    if (n_host == 0) return DYG_OK;
    DYG_TRY(rowops_ensure(GA, 2ull * n_host, st));
    AppSides A{};
    A.s[0] = append_side(GA, EA.src, EA.dst, EA.w);
    A.n = 1;
    if (GB) {
        DYG_TRY(rowops_ensure(GB, 2ull * n_host, st));
        A.s[1] = append_side(GB, EB.src, EB.dst, EB.w);
        A.n = 2;
    }
    const bool hubs = GA->long_rows || (GB && GB->long_rows);
    return launch_phases<k_append<Op>>(op_blocks(2ull * n_host, hubs), st, grid_bar(GA, halt), op, A,
                                       ptr<uint32_t>(GA->ws.blk), work, halt, code);
}

}  // namespace dyg
