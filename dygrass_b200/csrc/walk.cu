// walk.cu -- sm_100a random-walk kernels of the dyGRASS update path.
//
// One walker = one non-backtracking random walk from an edge's source towards
// its target (random_walk_incremental/main.cu:70-211 and
// random_walk_decremental/main.cu:77-220 restated).  Walk lengths differ by
// two orders of magnitude between walkers (dead ends after one step, full
// max_steps walks), so instead of the reference's one-block-per-edge with a
// 512-thread barrier tree, each warp of a persistent grid keeps its 32 lanes
// busy: a lane whose walker ends takes the next walker of the warp's current
// chunk, and the warp pulls a new chunk (16, 32 or 64 walkers of an edge, see
// chunk_for) from a global counter when that is handed out.  The per-edge winner (max 1/R, lowest
// walker id) is a 64-bit key reduced with atomicMax, so no barrier and no
// global scratch arrays are needed.  Lanes refill in step with one another
// (every four moves), so the random-number blocks are drawn by whole warps.
//
// Draw d of walker k of update u is word d&3 of
// Philox4x32-10({d>>2, k, u_lo, u_hi | domain<<24}, seed).  The decremental
// winner's path comes from the record its walker left (PathRec) or, in the
// batches that keep none, from a replay of that walker: any walker can be
// replayed.  Neither needs the reference's per-thread path[100] arrays.
#include <stdlib.h>

#include <mutex>
#include <vector>

#include <atomic>

#include "dyg_internal.cuh"
#include "gridsync.cuh"
#include "rowops.cuh"

namespace dyg {

// ------------------------------------------------------------- profiling
namespace {
struct ProfEvent {
    cudaEvent_t a, b;
    int kind;  // 0 incremental walk, 1 decremental walk, 2 replay/fallback
};
std::mutex g_prof_mu;
bool g_prof_on = false;
std::vector<ProfEvent> g_prof_events;
dyg_profile g_prof_acc{};

void prof_flush_locked() {
    for (ProfEvent &e : g_prof_events) {
        float ms = 0.f;
        if (cudaEventSynchronize(e.b) == cudaSuccess && cudaEventElapsedTime(&ms, e.a, e.b) == cudaSuccess) {
            if (e.kind == 0) { g_prof_acc.incr_walk_ms += ms; g_prof_acc.incr_walk_launches++; }
            else if (e.kind == 1) { g_prof_acc.decr_walk_ms += ms; g_prof_acc.decr_walk_launches++; }
            else { g_prof_acc.other_walk_ms += ms; g_prof_acc.other_walk_launches++; }
        }
        cudaGetLastError();
        cudaEventDestroy(e.a);
        cudaEventDestroy(e.b);
    }
    g_prof_events.clear();
}

struct ProfScope {
    bool on = false;
    ProfEvent ev{};
    cudaStream_t st;
    ProfScope(int kind, cudaStream_t s) : st(s) {
        std::lock_guard<std::mutex> lk(g_prof_mu);
        if (!g_prof_on) return;
        ev.kind = kind;
        if (cudaEventCreate(&ev.a) != cudaSuccess || cudaEventCreate(&ev.b) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        cudaEventRecord(ev.a, st);
        on = true;
    }
    ~ProfScope() {
        if (!on) return;
        cudaEventRecord(ev.b, st);
        std::lock_guard<std::mutex> lk(g_prof_mu);
        g_prof_events.push_back(ev);
        if (g_prof_events.size() > 4096) prof_flush_locked();
    }
};
}  // namespace

constexpr int kWalkThreads = 256;

struct WalkArgs {
    DevGraph g;
    WalkJob job;
    RowIndex ix;      // weighted walks
    PathRec rec;      // decremental walks
    uint32_t walkers, max_steps;
    uint32_t prune;
    uint32_t prune_every;   // iterations between reads of the edge's best (a power of two)
    uint32_t chunk;   // walkers handed to a warp at a time
    float threshold;
    uint2 key;
    unsigned long long *keys;
    unsigned long long *scalars;
};

struct Walker {
    uint32_t cur, prev, step, tgt, walker, c2, c3, rblk;
    uint4 rbuf;
    float R, we;
};

enum : int { kContinue = 0, kFail = 1, kFound = 2 };

// Draw for the walker's current step: word (step-1)&3 of the Philox block
// (step-1)>>2, computed once per block of four draws.
__device__ __forceinline__ uint32_t draw_next(Walker &s, uint2 key) {
    const uint32_t di = s.step - 1u, b = di >> 2;
    if (b != s.rblk) {
        s.rbuf = philox4x32_10(make_uint4(b, s.walker, s.c2, s.c3), key);
        s.rblk = b;
    }
    return pick4(s.rbuf, di & 3u);
}

// The move's common end: R += 1/w; distortion test (incremental only, from
// step 2 on), then the target test; the walk ends when the step counter
// reaches max_steps (main.cu:116, 139-157).
template <bool INCR>
__device__ __forceinline__ int finish_move(Walker &s, uint2 sl, uint32_t at, bool first,
                                           uint32_t max_steps, float thr, bool *moved,
                                           uint2 *taken, uint32_t *taken_at) {
    *moved = true;
    *taken = sl;
    *taken_at = at;
    // the slot holds the correctly rounded 1/w: one add per move, as R += 1/w
    s.R = __fadd_rn(s.R, __uint_as_float(sl.y));
    if (INCR && !first && __fmul_rn(s.R, s.we) >= thr) return kFail;
    if (sl.x == s.tgt) return kFound;
    s.prev = s.cur;
    s.cur = sl.x;
    s.step += 1u;
    if (s.step >= max_steps) return kFail;
    return kContinue;
}

// Weight-proportional choice in row [lo, lo + deg) by one thread: the first
// slot, in row order, among those whose column is not `ex` (when has_ex),
// whose inclusive prefix of fixed-point weights wq(w) exceeds
// floor(r * total / 2^32).  ~0u when total is 0; *picked receives the chosen
// slot.  The row is read kPickGroup slots at a time with the group's loads
// issued together.  A row of one group (every lattice row) is read once, its
// weights staying in registers for the choice; a longer row is read from its last
// group back to its first, which is in registers then, and forward again only if
// the choice is not in that one.
// (8,000 insertions and 12,000 deletions on a 40^3 mesh: 8.99 -> 7.68 ms with
// this and wq in integers, against groups of four read twice and wq in FP64.  A
// random geometric graph of 400,000 vertices, rows of 5 to 25 slots, 40,000
// deletions and insertions with 512 walkers: 3.78 and 7.41 ms with those, 3.93 and
// 6.58 with groups of eight read twice, 3.55 and 5.97 read back and forth.)
constexpr uint32_t kPickGroup = 8;
constexpr uint32_t kPickShort = 4;   // rows of a sparsifier: half the work of a group

template <uint32_t U>
struct PickGroup {
    uint2 c[U];
    unsigned long long p[U];   // inclusive prefixes over the group
};
template <uint32_t U>
__device__ __forceinline__ void pick_load(PickGroup<U> &g, const uint2 *__restrict__ slots,
                                          const float *__restrict__ wts, uint32_t lo,
                                          uint32_t left, uint32_t ex, bool has_ex) {
    float w[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
        g.c[u] = u < left ? __ldg(slots + lo + u) : make_uint2(0u, 0u);
        w[u] = u < left ? __ldg(wts + lo + u) : 0.f;
    }
    unsigned long long sum = 0ull;
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
        if (has_ex && g.c[u].x == ex) w[u] = 0.f;   // counts as absent
        sum += wq(w[u]);
        g.p[u] = sum;
    }
}
// The group's first slot whose prefix (after `before`) exceeds target, ~0u if
// none.  A slot that is absent or weighs nothing has its predecessor's prefix,
// so it is never the first, whether or not the sums wrapped past 2^64.
template <uint32_t U>
__device__ __forceinline__ uint32_t pick_in_group(const PickGroup<U> &g, unsigned long long target,
                                                  unsigned long long before, uint2 *picked) {
    uint32_t at = ~0u;
#pragma unroll
    for (int u = (int)U - 1; u >= 0; --u)
        if (before + g.p[u] > target) {
            at = (uint32_t)u;
            *picked = g.c[u];
        }
    return at;
}

// A row of up to U slots.
template <uint32_t U>
__device__ __forceinline__ uint32_t lane_pick_short(const uint2 *__restrict__ slots,
                                                    const float *__restrict__ wts, uint32_t lo,
                                                    uint32_t deg, uint32_t ex, bool has_ex,
                                                    uint32_t r, uint2 *picked) {
    PickGroup<U> g;
    pick_load(g, slots, wts, lo, deg, ex, has_ex);
    const unsigned long long total = g.p[U - 1u];
    if (total == 0ull) return ~0u;
    return lo + pick_in_group(g, mul_hi32(r, total), 0ull, picked);
}

__device__ __forceinline__ uint32_t lane_pick_weighted(const uint2 *__restrict__ slots,
                                                       const float *__restrict__ wts, uint32_t lo,
                                                       uint32_t deg, uint32_t ex, bool has_ex,
                                                       uint32_t r, uint2 *picked) {
    if (deg <= kPickGroup) return lane_pick_short<kPickGroup>(slots, wts, lo, deg, ex, has_ex, r, picked);
    PickGroup<kPickGroup> g;
    unsigned long long total = 0ull;
    // the last group first, so that the first one is in registers at the end
    uint32_t j0 = (deg - 1u) & ~(kPickGroup - 1u);
    while (true) {
        pick_load(g, slots, wts, lo + j0, deg - j0, ex, has_ex);
        total += g.p[kPickGroup - 1u];
        if (j0 == 0u) break;
        j0 -= kPickGroup;
    }
    if (total == 0ull) return ~0u;
    const unsigned long long target = mul_hi32(r, total);
    unsigned long long before = 0ull;
    while (true) {
        const uint32_t u = pick_in_group(g, target, before, picked);
        if (u != ~0u) return lo + j0 + u;
        before += g.p[kPickGroup - 1u];
        j0 += kPickGroup;
        if (j0 >= deg) return ~0u;
        pick_load(g, slots, wts, lo + j0, deg - j0, ex, has_ex);
    }
}

// The uniform move from row d (deg = d.y, past the dead-end test) with draw r.
template <bool INCR>
__device__ __forceinline__ int move_uniform(Walker &s, uint2 d, uint32_t r,
                                            const uint2 *__restrict__ slots, uint32_t max_steps,
                                            float thr, bool *moved, uint2 *taken,
                                            uint32_t *taken_at) {
    const bool first = (s.step == 1u);
    const uint32_t deg = d.y;
    uint32_t at = d.x + (first ? r % deg : r % (deg - 1u));
    uint2 sl = __ldg(slots + at);
    if (!first) {
        // the row's last slot is loaded beside the drawn one, not after it:
        // some lane of a warp lands on its previous vertex in almost every
        // step, and a dependent reload would hold the whole warp
        const uint32_t at_last = d.x + deg - 1u;
        const uint2 sl_last = __ldg(slots + at_last);
        if (sl.x == s.prev) {
            at = at_last;
            sl = sl_last;
        }
    }
    return finish_move<INCR>(s, sl, at, first, max_steps, thr, moved, taken, taken_at);
}

// One uniform move of one walker, mirroring the reference loop body:
//   step 1:  any neighbour, r % deg                    (main.cu:99-106)
//   step >1: dead end if deg == 1; r % (deg - 1) and the last slot when the
//            draw lands on the previous vertex          (main.cu:118-137)
// then finish_move.  *moved is set when a neighbour was drawn; *taken
// receives its slot.
template <bool INCR>
__device__ __forceinline__ int step_uniform(Walker &s, const uint2 *__restrict__ desc,
                                            const uint2 *__restrict__ slots, uint32_t max_steps,
                                            float thr, uint2 key, bool *moved, uint2 *taken,
                                            uint32_t *taken_at) {
    *moved = false;
    const uint2 d = __ldg(desc + s.cur);
    if (s.step == 1u ? (d.y == 0u) : (d.y <= 1u)) return kFail;
    return move_uniform<INCR>(s, d, draw_next(s, key), slots, max_steps, thr, moved, taken, taken_at);
}

// ------------------------------------------------ weighted, warp-cooperative
// Rows longer than kCoopRow slots are searched by the whole warp, one lane's
// row at a time: each lane takes four consecutive slots per pass over 128
// slots (two 128-bit slot loads and one 128-bit weight load for a quad inside
// the row; the quad grid starts at the row start rounded down to four slots,
// so every vector load is 16-byte aligned), a warp reduction gives the sum of
// each 128-slot tile, and the sums of up to kSegs segments of tiles are kept
// in shared memory.  The second pass finds the segment holding the target
// from those sums and scans only its tiles with a warp prefix scan.  The
// choice is the per-thread scan's: prefix sums of the fixed-point weights are
// exact integers, so the order of additions does not matter; only when a sum
// wraps past 2^64 (weights near 2^32) are prefixes not monotone, and then the
// second pass scans the whole row from its start, as the per-thread scan does.
constexpr uint32_t kCoopRow = 32;
constexpr uint32_t kSegs = 64;

__device__ __forceinline__ unsigned long long wq_ex(uint32_t col, float w, uint32_t ex,
                                                    bool has_ex) {
    return (has_ex && col == ex) ? 0ull : wq(w);
}

// Fixed-point weights of slots [j, j + 4) inside row [lo, hi) (0 outside it
// or for the excluded column).
__device__ __forceinline__ void quad_weights(const uint2 *__restrict__ slots,
                                             const float *__restrict__ wts, uint32_t j,
                                             uint32_t lo, uint32_t hi, uint32_t ex, bool has_ex,
                                             unsigned long long q[4]) {
    if (j >= lo && j + 4u <= hi) {
        const uint4 s01 = __ldg(reinterpret_cast<const uint4 *>(slots + j));
        const uint4 s23 = __ldg(reinterpret_cast<const uint4 *>(slots + j + 2u));
        const float4 w4 = __ldg(reinterpret_cast<const float4 *>(wts + j));
        q[0] = wq_ex(s01.x, w4.x, ex, has_ex);
        q[1] = wq_ex(s01.z, w4.y, ex, has_ex);
        q[2] = wq_ex(s23.x, w4.z, ex, has_ex);
        q[3] = wq_ex(s23.z, w4.w, ex, has_ex);
    } else {
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
            const uint32_t k = j + u;
            q[u] = (k >= lo && k < hi) ? wq_ex(__ldg(&slots[k].x), __ldg(wts + k), ex, has_ex) : 0ull;
        }
    }
}

// Sum over the warp with a wrap flag (any addition past 2^64).
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v, bool *wrap) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(kFull, v, o);
        const unsigned long long x = v + t;
        *wrap |= x < v;
        v = x;
    }
    return v;
}

__device__ __forceinline__ unsigned long long warp_incl_scan_u64(unsigned long long v,
                                                                 uint32_t lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, v, o);
        if (lane >= (uint32_t)o) v += t;
    }
    return v;
}

// Every lane of the warp calls this with the same row; returns the chosen
// slot (absolute index) on every lane, or ~0u when the total weight is 0.
__device__ __forceinline__ uint32_t warp_pick_weighted(const uint2 *__restrict__ slots,
                                                    const float *__restrict__ wts, uint32_t lo,
                                                    uint32_t deg, uint32_t ex, bool has_ex,
                                                    uint32_t r, unsigned long long *seg,
                                                    uint32_t lane) {
    const uint32_t hi = lo + deg;
    const uint32_t abase = lo & ~3u;
    const uint32_t ntile = (hi - abase + 127u) >> 7;
    uint32_t G = (ntile + kSegs - 1u) / kSegs;   // tiles per segment
    unsigned long long total = 0ull, segsum = 0ull;
    bool wrap = false;
    for (uint32_t t = 0; t < ntile; ++t) {
        unsigned long long q[4];
        quad_weights(slots, wts, abase + (t << 7) + 4u * lane, lo, hi, ex, has_ex, q);
        unsigned long long v = q[0] + q[1];
        wrap |= v < q[0];
        unsigned long long v2 = q[2] + q[3];
        wrap |= v2 < q[2];
        const unsigned long long v3 = v + v2;
        wrap |= v3 < v;
        v = warp_sum_u64(v3, &wrap);
        const unsigned long long nt = total + v;
        wrap |= nt < total;
        total = nt;
        segsum += v;
        if (t % G == G - 1u || t == ntile - 1u) {
            if (lane == 0u) seg[t / G] = segsum;
            segsum = 0ull;
        }
    }
    wrap = __any_sync(kFull, wrap);
    __syncwarp();
    if (total == 0ull) return ~0u;
    const unsigned long long target = mul_hi32(r, total);
    uint32_t t0 = 0u, t1 = ntile;
    unsigned long long base = 0ull;
    if (!wrap) {
        // the segment holding the target: lane l holds segments 2l and 2l+1
        const uint32_t nseg = (ntile + G - 1u) / G;
        const unsigned long long a = 2u * lane < nseg ? seg[2u * lane] : 0ull;
        const unsigned long long b = 2u * lane + 1u < nseg ? seg[2u * lane + 1u] : 0ull;
        const unsigned long long incl = warp_incl_scan_u64(a + b, lane);
        const unsigned long long excl = incl - (a + b);
        const uint32_t L = __ffs(__ballot_sync(kFull, incl > target)) - 1u;
        const bool in_a = excl + a > target;
        const uint32_t sidx = __shfl_sync(kFull, 2u * lane + (in_a ? 0u : 1u), L);
        base = __shfl_sync(kFull, in_a ? excl : excl + a, L);
        t0 = sidx * G;
        t1 = min(ntile, t0 + G);
    }
    __syncwarp();   // every lane read seg before a later row overwrites it
    for (uint32_t t = t0; t < t1; ++t) {
        const uint32_t j = abase + (t << 7) + 4u * lane;
        unsigned long long q[4];
        quad_weights(slots, wts, j, lo, hi, ex, has_ex, q);
        const unsigned long long v = q[0] + q[1] + q[2] + q[3];
        const unsigned long long incl = warp_incl_scan_u64(v, lane);
        // wrapped prefixes when `wrap`: then every tile is scanned in order
        // and the first slot whose prefix exceeds the target is the
        // per-thread scan's choice
        unsigned long long acc = base + incl - v;
        uint32_t hit = ~0u;
#pragma unroll
        for (uint32_t u = 0; u < 4u; ++u) {
            acc += q[u];
            if (hit == ~0u && j + u >= lo && j + u < hi && acc > target) hit = j + u;
        }
        const unsigned m = __ballot_sync(kFull, hit != ~0u);
        if (m) return __shfl_sync(kFull, hit, __ffs(m) - 1u);
        base += __shfl_sync(kFull, incl, 31);
    }
    return ~0u;
}

// ------------------------------------------------------------ row index
// On a graph with hub rows nearly every weighted move is at one, and a warp
// reading such a row for one lane after another bounds the walk: 9.87 ms for
// the deletion walks of a 1,000-edge R-MAT file (scale 13).  A walker needs
// two things of the row: the position and weight of the column it came from,
// and the first prefix sum above its target.  k_index tabulates both, once per
// launch of walks (the rows do not change while they walk), and each lane then
// chooses by itself: one hash lookup and one search of the prefixes.  Rows with
// a repeated column, or whose sum wraps past 2^64, get no index and are searched
// by the warp as before.
//
// It is built whenever the graph has hub rows (over kBigRow slots), of the rows
// that the warp would search (over kCoopRow): even a single edge's 256 walkers
// scan more than it costs.  Stream files on R-MAT graphs, us a file with the
// index and without (and with the rows read slot by slot as before either):
//   scale 13, 204,000 slots      1 deletion 287, 627 (1,408)    1,000: 1,826, 18,300 (28,600)
//   scale 18, 7.6 M slots        1 deletion 2,021, 13,210 (28,400)  1,000: 5,170, 68,500 (76,200)
//   scale 20, 31 M slots         1 deletion 2,570, 2,290 (4,530)    1,000: 11,200, 137,000 (149,000)
// The rows of kIdxRow + 1 to kCoopRow slots, which a lane can search, are
// indexed as well where that at most doubles the index (the R-MAT graphs: a few
// per cent slower without) or where there are enough walks: their index costs as
// a pass over their slots, and each walk saves some scans of such rows.  On a
// random geometric graph of 200,000 vertices and 3.2 M slots with one hub, us a
// batch with and without them (as before): 1 insertion 889, 557 (878); 32: 959,
// 698 (1,038); 1,000: 2,490, 3,260 (3,540); 4,096 deletions 669, 502 (628),
// 1,000: 513, 301 (377).  The lines lie at 16 slots a walk for insertions, whose
// walks are long, and at one for deletions, most of which walk a few moves.
constexpr uint32_t kIdxRow = kPickGroup;   // longer rows are indexed: the lane reads up to it at once
constexpr uint32_t kIdxInsertSlots = 16;   // slots a walk is worth
constexpr uint32_t kIdxBlockRow = 1024; // ... by a whole block from here on
constexpr uint32_t kIdxTile = 8;        // slots per thread of a block's tile

__device__ __forceinline__ uint32_t idx_bits(uint32_t deg) { return 32u - __clz(2u * deg - 1u); }
__device__ __forceinline__ uint32_t idx_hash(uint32_t col, uint32_t bits) {
    return (col * 0x9E3779B1u) >> (32u - bits);
}

// The choice of lane_pick_weighted from row v's index region.
__device__ __forceinline__ uint32_t index_pick(const uint2 *__restrict__ slots,
                                               const float *__restrict__ wts,
                                               const uint32_t *__restrict__ region, uint32_t lo,
                                               uint32_t deg, uint32_t ex, bool has_ex, uint32_t r) {
    const uint32_t bits = idx_bits(deg);
    const unsigned long long *pre = reinterpret_cast<const unsigned long long *>(region + (1u << bits));
    unsigned long long total = __ldg(pre + deg - 1u), e = 0ull;
    uint32_t pos = deg;
    if (has_ex) {
        uint32_t h = idx_hash(ex, bits);
        for (uint32_t left = 1u << bits; left > 0u; --left) {   // half of the table is empty
            const uint32_t t = __ldg(region + h);
            if (t == 0u) break;
            const uint32_t col = __ldg(&slots[lo + t - 1u].x);
            const float w = __ldg(wts + lo + t - 1u);   // beside the column, not after it
            if (col == ex) {
                pos = t - 1u;
                e = wq(w);
                break;
            }
            h = (h + 1u) & ((1u << bits) - 1u);
        }
    }
    total -= e;
    if (total == 0ull) return ~0u;
    const unsigned long long target = mul_hi32(r, total);
    // first slot whose prefix without `ex` exceeds the target; the slot of
    // `ex` itself leaves that prefix as it was, so it is never the first
    // (seven pivots at a time: each round of loads divides the range by eight)
    uint32_t a = 0u, len = deg;   // the first is in [a, a + len)
    while (len > 1u) {
        const uint32_t step = (len + 7u) >> 3;
        uint32_t below = 0u;   // pivots whose prefix does not exceed the target
#pragma unroll
        for (uint32_t u = 1u; u <= 7u; ++u) {
            const uint32_t j = a + u * step - 1u;   // last slot of the u-th part
            const bool in = u * step < len;
            const unsigned long long v = in ? __ldg(pre + j) - (j >= pos ? e : 0ull) : ~0ull;
            below += v <= target ? 1u : 0u;
        }
        a += below * step;
        len = min(step, len - below * step);
    }
    return lo + a;
}

struct IndexArgs {
    DevGraph g;
    uint32_t *rbase, *list, *words;
    uint32_t cap;                    // words
    unsigned long long *cursor;      // next free word (from 2 on: 0 means no region)
    unsigned long long *counts;      // S_IDXN
    unsigned long long *sums;        // S_IDXSUM
    unsigned long long budget;       // slots of short rows that the walks are worth
    bool all;                        // the budget covers any graph: nothing to count
    const unsigned long long *halt;
};

// Hash insert of slot j's column; true if the column is there already.
__device__ __forceinline__ bool idx_insert(const IndexArgs &a, uint32_t *tab, uint32_t bits,
                                           uint32_t lo, uint32_t j, uint32_t col) {
    uint32_t h = idx_hash(col, bits);
    while (true) {
        const uint32_t old = atomicCAS(tab + h, 0u, j + 1u);
        if (old == 0u) return false;
        if (a.g.slots[lo + old - 1u].x == col) return true;
        h = (h + 1u) & ((1u << bits) - 1u);
    }
}

__global__ void __launch_bounds__(kOpThreads, 2) k_index(const __grid_constant__ IndexArgs a, GridBar bar) {
    __shared__ unsigned long long s_sum[kOpThreads / 32];
    __shared__ uint32_t s_bad;
    if (*a.halt) return;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    uint32_t shortest = kIdxRow;
    if (!a.all) {
        uint32_t mid = 0u, lng = 0u;   // a graph's slots fit 32 bits
        for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.g.n; v += gridDim.x * blockDim.x) {
            const uint32_t deg = a.g.desc[v].y;
            if (deg > kCoopRow) lng += deg;
            else if (deg > kIdxRow) mid += deg;
        }
        __syncwarp();
        mid = __reduce_add_sync(kFull, mid);
        lng = __reduce_add_sync(kFull, lng);
        if (lane == 0u && (mid | lng)) atomicAdd(a.sums, ((unsigned long long)lng << 32) + mid);
        if (!grid_sync(bar)) return;
        const unsigned long long both = __ldcg(a.sums);
        if ((both & 0xFFFFFFFFull) > (both >> 32) + a.budget) shortest = kCoopRow;
    }
    // regions, and the lists of rows: for a warp from the front, for a block
    // from the back
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.g.n; v += gridDim.x * blockDim.x) {
        const uint32_t deg = a.g.desc[v].y;
        uint32_t base = 0u;
        if (deg > shortest) {
            const unsigned long long want = (1ull << idx_bits(deg)) + 2ull * deg;
            const unsigned long long at = atomicAdd(a.cursor, want) + 2ull;
            if (at + want <= a.cap) {
                base = (uint32_t)at;
                if (deg <= kIdxBlockRow) a.list[(uint32_t)atomicAdd(a.counts, 1ull)] = v;
                else a.list[a.g.n - 1u - (uint32_t)(atomicAdd(a.counts, 1ull << 32) >> 32)] = v;
            }
        }
        a.rbase[v] = base;
    }
    if (!grid_sync(bar)) return;
    const unsigned long long both = __ldcg(a.counts);
    const uint32_t n_warp = (uint32_t)both, n_block = (uint32_t)(both >> 32);
    for (uint32_t q = blockIdx.x; q < n_block; q += gridDim.x) {
        const uint32_t v = a.list[a.g.n - 1u - q];
        const uint2 d = a.g.desc[v];
        const uint32_t bits = idx_bits(d.y);
        uint32_t *tab = a.words + a.rbase[v];
        unsigned long long *pre = reinterpret_cast<unsigned long long *>(tab + (1u << bits));
        for (uint32_t h = threadIdx.x; h < (1u << bits); h += blockDim.x) tab[h] = 0u;
        if (threadIdx.x == 0) s_bad = 0u;
        __syncthreads();
        bool bad = false;
        unsigned long long carry = 0ull;
        for (uint32_t t0 = 0; t0 < d.y; t0 += kIdxTile * blockDim.x) {
            const uint32_t j0 = t0 + kIdxTile * threadIdx.x;
            unsigned long long q8[kIdxTile], run = 0ull;
#pragma unroll
            for (uint32_t u = 0; u < kIdxTile; ++u) {
                q8[u] = j0 + u < d.y ? wq(a.g.wts[d.x + j0 + u]) : 0ull;
                if (j0 + u < d.y) bad |= idx_insert(a, tab, bits, d.x, j0 + u, a.g.slots[d.x + j0 + u].x);
            }
#pragma unroll
            for (uint32_t u = 0; u < kIdxTile; ++u) {
                run += q8[u];
                bad |= run < q8[u];
                q8[u] = run;
            }
            unsigned long long incl = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long x = __shfl_up_sync(kFull, incl, o);
                if (lane >= (uint32_t)o) {
                    incl += x;
                    bad |= incl < x;
                }
            }
            if (lane == 31u) s_sum[wid] = incl;
            __syncthreads();
            unsigned long long before = carry, all = carry;
            for (uint32_t k = 0; k < blockDim.x >> 5; ++k) {
                const unsigned long long x = s_sum[k];
                all += x;
                bad |= all < x;
                if (k < wid) before += x;
            }
            before += incl - run;
#pragma unroll
            for (uint32_t u = 0; u < kIdxTile; ++u)
                if (j0 + u < d.y) pre[j0 + u] = before + q8[u];
            carry = all;
            __syncthreads();
        }
        if (bad) s_bad = 1u;
        __syncthreads();
        if (threadIdx.x == 0 && s_bad) a.rbase[v] = 0u;
        __syncthreads();
    }
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; q < n_warp; q += warps) {
        const uint32_t v = a.list[q];
        const uint2 d = a.g.desc[v];
        const uint32_t bits = idx_bits(d.y);
        uint32_t *tab = a.words + a.rbase[v];
        unsigned long long *pre = reinterpret_cast<unsigned long long *>(tab + (1u << bits));
        for (uint32_t h = lane; h < (1u << bits); h += 32u) tab[h] = 0u;
        __syncwarp();
        bool bad = false;
        unsigned long long carry = 0ull;
        for (uint32_t j0 = 0; j0 < d.y; j0 += 32u) {
            const uint32_t j = j0 + lane;
            unsigned long long incl = j < d.y ? wq(a.g.wts[d.x + j]) : 0ull;
            if (j < d.y) bad |= idx_insert(a, tab, bits, d.x, j, a.g.slots[d.x + j].x);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long x = __shfl_up_sync(kFull, incl, o);
                if (lane >= (uint32_t)o) {
                    incl += x;
                    bad |= incl < x;
                }
            }
            const unsigned long long at = carry + incl;
            bad |= at < carry;
            if (j < d.y) pre[j] = at;
            carry = __shfl_sync(kFull, at, 31);
        }
        bad = __any_sync(kFull, bad);
        if (lane == 0u && bad) a.rbase[v] = 0u;
    }
}

// One move of every active lane's walker: in a row with an index through it,
// in another of up to kCoopRow slots by the lane, in a longer one by the whole
// warp (all 32 lanes call this).  Returns the move's result for active lanes.
template <bool INCR>
__device__ __forceinline__ int step_weighted_warp(Walker &s, bool active, const DevGraph &g,
                                                  const RowIndex &ix, uint32_t max_steps, float thr, uint2 key,
                                                  unsigned long long *seg, uint32_t lane,
                                                  bool *moved, uint2 *taken, uint32_t *taken_at) {
    *moved = false;
    uint2 d = make_uint2(0u, 0u);
    bool first = false, pick = false;
    uint32_t r = 0u;
    if (active) {
        d = __ldg(g.desc + s.cur);
        first = (s.step == 1u);
        if (!(first ? (d.y == 0u) : (d.y <= 1u))) {
            r = draw_next(s, key);
            pick = true;
        }
    }
    uint32_t at = ~0u;
    uint2 sl = make_uint2(0u, 0u);
    uint32_t base = 0u;
    if (pick && d.y > kIdxRow && ix.rbase) base = __ldg(ix.rbase + s.cur);
    if (base) at = index_pick(g.slots, g.wts, ix.words + base, d.x, d.y, s.prev, !first, r);
    const bool own_row = pick && !base && d.y <= kCoopRow;   // chosen by this lane, slot in hand
    // insertion walks are on a sparsifier, whose rows are short (their walks on
    // a weighted 40^3 mesh 1.52 -> 1.36 ms); one width for the whole warp: two
    // in turn would cost more than the wider
    if (!INCR || __any_sync(kFull, own_row && d.y > kPickShort)) {
        if (own_row) at = lane_pick_weighted(g.slots, g.wts, d.x, d.y, s.prev, !first, r, &sl);
    } else if (own_row) {
        at = lane_pick_short<kPickShort>(g.slots, g.wts, d.x, d.y, s.prev, !first, r, &sl);
    }
    unsigned coop = __ballot_sync(kFull, pick && !own_row && !base);
    while (coop) {
        const uint32_t L = __ffs(coop) - 1u;
        coop &= coop - 1u;
        const uint32_t lo = __shfl_sync(kFull, d.x, L), dg = __shfl_sync(kFull, d.y, L);
        const uint32_t ex = __shfl_sync(kFull, s.prev, L), rr = __shfl_sync(kFull, r, L);
        const bool hx = __shfl_sync(kFull, first ? 0u : 1u, L) != 0u;
        const uint32_t j = warp_pick_weighted(g.slots, g.wts, lo, dg, ex, hx, rr, seg, lane);
        if (lane == L) at = j;
    }
    if (!pick || at == ~0u) return kFail;
    if (!own_row) sl = __ldg(g.slots + at);
    return finish_move<INCR>(s, sl, at, first, max_steps, thr, moved, taken, taken_at);
}

// RN(1/R) < c for positive finite R, c, decided by one product where it can
// be: p = RN(R*c) is within 2^-24 of R*c, so p > 1 + 2^-21 gives
// 1/R < c (1 - 7 * 2^-24), below c by more than half an ulp of c, hence
// RN(1/R) < c; p < 1 - 2^-21 gives RN(1/R) > c the same way.  Only products
// inside that band take the correctly rounded reciprocal.
__device__ __forceinline__ bool below_best(float R, float c) {
    const float p = __fmul_rn(R, c);
    if (p > 1.0000004768371582f) return true;    // 1 + 2^-21
    if (p < 0.9999995231628418f) return false;   // 1 - 2^-21
    return __frcp_rn(R) < c;
}

// ---------------------------------------------------------- uniform walks
// r mod d for d below kDivTab by a table of floor((2^32 - 1) / d): the high
// word of r times it is the quotient or one less, so one correction makes the
// remainder exact.  A shared-memory lookup and two multiplies take the place
// of the general division's conversions and its reciprocal.
constexpr uint32_t kDivTab = 256;
__device__ __forceinline__ uint32_t rem_small(uint32_t r, uint32_t d, const uint32_t *s_div) {
    if (d >= kDivTab) return r % d;
    const uint32_t m = r - __umulhi(r, s_div[d]) * d;
    return m >= d ? m - d : m;
}

// ------------------------------------------------------- handing out walkers
// Edge of a warp's current chunk of walkers.
struct ChunkEdge {
    uint32_t src, tgt, e;
    float we;
    uint32_t c2, c3;
};
// Warp-uniform: the walkers left of the current chunk.
struct Chunk {
    uint32_t next = 0u, end = 0u;
    bool exhausted = false;
};

// Starts walkers in the warp's free lanes.  One lane takes a chunk from the
// global counter and reads its edge into shared memory, from where the lanes
// that start its walkers take it; it also counts the chunk's walks (a walker
// that started ends before the kernel does).  `start(edge, walker)` runs in
// each lane that takes a walker.
template <bool INCR, class Start>
__device__ __forceinline__ void refill(const WalkArgs &a, unsigned long long n_chunks, Chunk &c,
                                       ChunkEdge *ce, uint32_t lane, uint32_t free_mask,
                                       uint32_t *walks, Start start) {
    while (free_mask != 0u && !c.exhausted) {
        if (c.next >= c.end) {
            __syncwarp();   // the lanes that took the last chunk's walkers have read its edge
            uint32_t first = 0u, have = 0u;
            if (lane == 0u) {
                const uint32_t cpe = a.walkers / a.chunk;   // chunks per edge
                const unsigned long long t = atomicAdd(a.scalars + S_WORK, 1ull);
                if (t < n_chunks) {
                    // chunk t = edge e, part t mod cpe
                    const uint32_t e = (t >> 32) ? (uint32_t)(t / cpe) : (uint32_t)t / cpe;
                    first = (uint32_t)(t - (unsigned long long)e * cpe) * a.chunk;
                    const unsigned long long uid = a.job.uid ? a.job.uid[e] : a.job.uid0 + e;
                    const ChunkEdge x{a.job.src[e], a.job.dst[e], e, INCR ? a.job.w[e] : 0.f,
                                      (uint32_t)uid, ctr3_of(uid, a.job.domain)};
                    *ce = x;
                    *walks += a.chunk;
                    have = 1u;
                    if (x.src >= a.g.n || x.tgt >= a.g.n) {
                        atomicOr(a.scalars + S_ERR, (unsigned long long)kErrVertex);
                        have = 2u;
                    }
                }
            }
            __syncwarp();
            have = __shfl_sync(kFull, have, 0);
            if (have == 0u) {
                c.exhausted = true;
                break;
            }
            if (have == 2u) continue;   // not walked
            c.next = __shfl_sync(kFull, first, 0);
            c.end = c.next + a.chunk;
        }
        const uint32_t take = min((uint32_t)__popc(free_mask), c.end - c.next);
        const uint32_t rank = __popc(free_mask & ((1u << lane) - 1u));
        const bool mine = ((free_mask >> lane) & 1u) && rank < take;
        if (mine) start(*ce, c.next + rank);
        free_mask &= ~__ballot_sync(kFull, mine);
        c.next += take;
    }
}

__device__ __forceinline__ void count_moves(const WalkArgs &a, uint32_t moves, uint32_t walks,
                                            uint32_t lane) {
    const uint32_t wm = __reduce_add_sync(kFull, moves);
    if (lane == 0u) {
        if (wm) atomicAdd(a.scalars + S_MOVES, (unsigned long long)wm);
        if (walks) atomicAdd(a.scalars + S_WALKS, (unsigned long long)walks);
    }
}

// Conductance bits of the best walk an edge has so far.
__device__ __forceinline__ uint32_t best_bits(const WalkArgs &a, uint32_t e) {
    return *(reinterpret_cast<const volatile uint32_t *>(a.keys + e) + 1);
}

// Copies a walker's path of L moves to a record of edge e: its first `kept`
// moves from the history (four = true: four moves to a uint4), the rest from
// `last`.
__device__ __forceinline__ void write_record(const PathRec &rec, uint32_t e, unsigned long long key,
                                             uint32_t L, uint32_t tid, uint32_t nth, bool four,
                                             uint32_t kept, const uint32_t (&last)[4]) {
    const unsigned long long at = atomicAdd(rec.cursor, (unsigned long long)L + 3ull);
    if (at + L + 3ull > rec.cap) return;   // the commit sees the cursor past the end
    uint32_t *w = rec.words + at;
    w[0] = atomicExch(rec.heads + e, (uint32_t)at + 1u);
    w[1] = (uint32_t)key;
    w[2] = (uint32_t)(key >> 32);
    if (four) {
        const uint4 *h = reinterpret_cast<const uint4 *>(rec.hist) + tid;
        for (uint32_t j = 0; j < kept; j += 4u, h += nth) {
            const uint4 q = *h;
            w[3u + j] = q.x;
            w[4u + j] = q.y;
            w[5u + j] = q.z;
            w[6u + j] = q.w;
        }
    } else {
        for (uint32_t j = 0; j < kept; ++j) w[3u + j] = rec.hist[(size_t)j * nth + tid];
    }
#pragma unroll
    for (uint32_t u = 0; u < 4u; ++u)
        if (kept + u < L) w[3u + kept + u] = last[u];
}

// The uniform transition's walks.  Walks are short (5.8 moves on the mesh's
// sparsifier: most end in a leaf), so the cost is shared between the moves and
// what surrounds them; every iteration starts walkers in the free lanes and
// then moves each walker four times, so that a walker enters every iteration
// at a step 1 mod 4 and draws one Philox block for it, and the step counter
// advances once per iteration.  The edge's best is read once per iteration
// and applied after the moves to the walkers still alive: R only grows along a walk and
// 1/R is monotone, so a walker whose 1/R is below it can neither win nor tie,
// and stopping it leaves every result unchanged.
// 40 registers: six blocks (48 warps) per SM; eight blocks spill (insertions
// of the 100^3 mesh 4.43 -> 6.43 ms).  Bound by the L1's gathers on a sparsifier
// (88 % of its throughput, 66 % of issue cycles, 71 % of the warps, third insertion
// batch of a 60^3 mesh) and by gather latency and the last long walks on the dense
// graph (57 %, 29 %, 42 %, its third deletion batch).  Against one lane-private edge read
// and best per walker and the general remainder: insertions of the 100^3 mesh
// 5.27 -> 4.43 ms, 24 random geometric graphs 1.14 -> 0.96 ms, deletions of
// the mesh 2.28 -> 2.25 ms.  With chunks of 64 and the edge's best read before the
// moves (insertions), the two mesh walks take 4.0 and 1.9 ms.
// REC: the walkers keep their paths (see PathRec), at five blocks of 48
// registers, since six would spill.
template <bool INCR, bool REC>
__global__ void __launch_bounds__(kWalkThreads, REC ? 5 : 6) k_walk_uniform(WalkArgs a) {
    __shared__ uint32_t s_div[kDivTab];
    __shared__ ChunkEdge s_edge[kWalkThreads / 32];
    if (a.job.halt && *a.job.halt) return;
    for (uint32_t d = threadIdx.x; d < kDivTab; d += kWalkThreads) s_div[d] = d ? 0xFFFFFFFFu / d : 0u;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    ChunkEdge *ce = s_edge + (threadIdx.x >> 5);
    const unsigned long long n_chunks = (unsigned long long)job_count(a.job) * (a.walkers / a.chunk);
    Chunk chunk;
    bool active = false;
    uint32_t cur = 0u, prev = 0u, step = 0u, tgt = 0u, walker = 0u, c2 = 0u, c3 = 0u, my_e = 0u;
    float R = 0.f, we = 0.f;
    uint32_t moves = 0u, walks = 0u;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;   // REC
    for (uint32_t T = 0u;; ++T) {
        refill<INCR>(a, n_chunks, chunk, ce, lane, __ballot_sync(kFull, !active), &walks,
                     [&](const ChunkEdge &x, uint32_t k) {
                         walker = k;
                         cur = x.src;
                         tgt = x.tgt;
                         my_e = x.e;
                         we = x.we;
                         c2 = x.c2;
                         c3 = x.c3;
                         step = 1u;
                         R = 0.f;
                         active = true;
                     });
        if (!__any_sync(kFull, active)) break;
        if (active) {
            const uint4 blk = philox4x32_10(make_uint4((step - 1u) >> 2, walker, c2, c3), a.key);
            // insertion walks read the edge's best before the moves, whose
            // latency hides it; few of their edges ever have one, so its age
            // matters little (insertion rounds 2-6 % faster; deletion walks
            // prune on the latest)
            const uint32_t early = INCR && a.prune ? best_bits(a, my_e) : 0u;
            const uint32_t left = a.max_steps - step;   // the walk ends when its step reaches max_steps
            uint32_t took[4] = {0u, 0u, 0u, 0u};        // slots of this iteration's moves (decremental)
            uint32_t found = 0u;
#pragma unroll
            for (uint32_t mv = 0; mv < 4u; ++mv) {
                if (!active) break;
                const uint2 d = __ldg(a.g.desc + cur);
                const bool first = mv == 0u && step == 1u;
                // step 1: any neighbour; later: dead end if deg == 1, else
                // r % (deg - 1) and the last slot when the draw lands on the
                // previous vertex (main.cu:99-137)
                const uint32_t deg = first ? d.y : d.y - 1u;
                if ((int)deg <= 0) {
                    active = false;
                    break;
                }
                const uint32_t r = mv == 0u ? blk.x : (mv == 1u ? blk.y : (mv == 2u ? blk.z : blk.w));
                const uint2 *row = a.g.slots + d.x;
                uint32_t at = rem_small(r, deg, s_div);
                uint2 sl = __ldg(row + at);
                if (!first) {
                    // loaded beside the drawn slot: some lane lands on its
                    // previous vertex in almost every move
                    const uint2 last = __ldg(row + deg);
                    if (sl.x == prev) {
                        sl = last;
                        at = deg;
                    }
                }
                if (REC) took[mv] = d.x + at;
                ++moves;
                R = __fadd_rn(R, __uint_as_float(sl.y));
                if (INCR && !first && __fmul_rn(R, we) >= a.threshold) {
                    active = false;
                } else if (sl.x == tgt) {
                    // published at once, so the edge's other walkers can stop early
                    if (REC) found = step + mv;
                    else atomicMax(a.keys + my_e, pack_key(__frcp_rn(R), walker, step + mv));
                    active = false;
                } else if (mv + 1u >= left) {
                    active = false;
                }
                prev = cur;
                cur = sl.x;
            }
            if (REC && found) {
                const unsigned long long key = pack_key(__frcp_rn(R), walker, found);
                const unsigned long long was = atomicMax(a.keys + my_e, key);
                if (key > was) write_record(a.rec, my_e, key, found, tid, nth, true, step - 1u, took);
            }
            if (REC && active)
                reinterpret_cast<uint4 *>(a.rec.hist)[(size_t)((step - 1u) >> 2) * nth + tid] =
                    make_uint4(took[0], took[1], took[2], took[3]);
            step += 4u;
            if (active && a.prune && (T & (a.prune_every - 1u)) == a.prune_every - 1u) {
                const uint32_t known = INCR ? early : best_bits(a, my_e);
                if (known && below_best(R, __uint_as_float(known))) active = false;
            }
        }
    }
    count_moves(a, moves, walks, lane);
}

// The weighted transition's walks: as the uniform ones, but a move costs a
// look at the whole row (or its index), so the bound is applied after every
// move, and read again after every fourth.  Three blocks per SM.
template <bool INCR>
__global__ void __launch_bounds__(kWalkThreads, 3) k_walk_weighted(WalkArgs a) {
    __shared__ unsigned long long s_seg[(kWalkThreads / 32) * kSegs];
    __shared__ ChunkEdge s_edge[kWalkThreads / 32];
    if (a.job.halt && *a.job.halt) return;
    const uint32_t lane = threadIdx.x & 31u;
    ChunkEdge *ce = s_edge + (threadIdx.x >> 5);
    unsigned long long *seg = s_seg + (threadIdx.x >> 5) * kSegs;
    const unsigned long long n_chunks = (unsigned long long)job_count(a.job) * (a.walkers / a.chunk);
    Chunk chunk;
    bool active = false;
    uint32_t my_e = 0u, known = 0u;
    Walker s{};
    uint32_t moves = 0u, walks = 0u;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    for (uint32_t T = 0u;; ++T) {
        refill<INCR>(a, n_chunks, chunk, ce, lane, __ballot_sync(kFull, !active), &walks,
                     [&](const ChunkEdge &x, uint32_t k) {
                         s.walker = k;
                         s.cur = x.src;
                         s.tgt = x.tgt;
                         s.we = x.we;
                         s.c2 = x.c2;
                         s.c3 = x.c3;
                         s.rblk = 0xFFFFFFFFu;
                         s.step = 1u;
                         s.R = 0.f;
                         s.prev = 0u;
                         my_e = x.e;
                         known = a.prune ? best_bits(a, x.e) : 0u;
                         active = true;
                     });
        if (!__any_sync(kFull, active)) break;
#pragma unroll 1
        for (uint32_t mv = 0; mv < 4u; ++mv) {
            bool moved = false;
            uint2 taken;
            uint32_t taken_at;
            const int r = step_weighted_warp<INCR>(s, active, a.g, a.ix, a.max_steps, a.threshold, a.key,
                                                   seg, lane, &moved, &taken, &taken_at);
            if (active) {
                moves += moved ? 1u : 0u;
                if (r == kFound) {
                    const unsigned long long key = pack_key(__frcp_rn(s.R), s.walker, s.step);
                    const unsigned long long was = atomicMax(a.keys + my_e, key);
                    if (!INCR && a.rec.heads && key > was) {
                        const uint32_t took[4] = {taken_at, 0u, 0u, 0u};
                        write_record(a.rec, my_e, key, s.step, tid, nth, false, s.step - 1u, took);
                    }
                } else if (!INCR && a.rec.heads && r == kContinue) {
                    a.rec.hist[(size_t)(s.step - 2u) * nth + tid] = taken_at;   // the move just made
                }
                if (r != kContinue || (known && below_best(s.R, __uint_as_float(known)))) active = false;
            }
            if (!__any_sync(kFull, active)) break;
        }
        if (active && a.prune && (T & (a.prune_every - 1u)) == a.prune_every - 1u) {
            known = best_bits(a, my_e);
            if (known && below_best(s.R, __uint_as_float(known))) active = false;
        }
    }
    count_moves(a, moves, walks, lane);
}

// Replays the winner of each edge of uniform decremental walks and writes its
// path (random_walk_decremental/main.cu:206-217 writes the same vertices from a
// per-thread local array).
__global__ void k_winner_paths(DevGraph g, WalkJob job, uint32_t max_steps, uint2 key,
                               const unsigned long long *keys, uint32_t stride, uint32_t *pv,
                               uint32_t *ps, int32_t *plen, unsigned long long *scalars) {
    if (job.halt && *job.halt) return;
    const uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n = job_count(job);
    if (f >= n) return;
    const unsigned long long k = keys[f];
    if (!k) {
        plen[f] = -1;
        return;
    }
    Walker s;
    s.walker = key_walker(k);
    s.cur = job.src[f];
    s.tgt = job.dst[f];
    s.we = 0.f;
    const unsigned long long uid = job.uid ? job.uid[f] : job.uid0 + f;
    s.c2 = (uint32_t)uid;
    s.c3 = ctr3_of(uid, job.domain);
    s.rblk = 0xFFFFFFFFu;
    s.rbuf = make_uint4(0u, 0u, 0u, 0u);
    s.step = 1u;
    s.R = 0.f;
    s.prev = 0u;
    uint32_t *row_v = pv + (size_t)f * stride;
    uint32_t *row_s = ps + (size_t)f * stride;
    row_v[0] = s.cur;
    int r;
    do {
        const uint32_t at = s.step;
        bool moved;
        uint2 taken;
        uint32_t taken_at;
        r = step_uniform<false>(s, g.desc, g.slots, max_steps, 0.f, key, &moved, &taken, &taken_at);
        if (moved && at < stride) {   // no load: a store waiting on one would stall the chain
            row_v[at] = taken.x;
            row_s[at] = taken_at;
        }
    } while (r == kContinue);
    const int32_t found = (r == kFound) ? (int32_t)s.step : -1;
    plen[f] = found;
    if (found != key_found(k)) atomicOr(scalars + S_ERR, (unsigned long long)kErrPath);
}

// Weighted winner replays, one warp per path: the walker lives in lane 0 and
// rows longer than kCoopRow are searched by the whole warp, as in the walk
// kernel (a replay through a hub row would otherwise scan it one slot at a
// time).
constexpr int kReplayThreads = 128;
__global__ void __launch_bounds__(kReplayThreads)
k_winner_paths_weighted(DevGraph g, WalkJob job, RowIndex ix, uint32_t max_steps, uint2 key,
                        const unsigned long long *keys, uint32_t stride, uint32_t *pv, uint32_t *ps,
                        int32_t *plen, unsigned long long *scalars) {
    __shared__ unsigned long long s_seg[(kReplayThreads / 32) * kSegs];
    if (job.halt && *job.halt) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t f = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n = job_count(job);
    if (f >= n) return;   // whole warps leave together
    const unsigned long long k = keys[f];
    if (!k) {
        if (lane == 0u) plen[f] = -1;
        return;
    }
    Walker s;
    s.walker = key_walker(k);
    s.cur = job.src[f];
    s.tgt = job.dst[f];
    s.we = 0.f;
    const unsigned long long uid = job.uid ? job.uid[f] : job.uid0 + f;
    s.c2 = (uint32_t)uid;
    s.c3 = ctr3_of(uid, job.domain);
    s.rblk = 0xFFFFFFFFu;
    s.rbuf = make_uint4(0u, 0u, 0u, 0u);
    s.step = 1u;
    s.R = 0.f;
    s.prev = 0u;
    uint32_t *row_v = pv + (size_t)f * stride;
    uint32_t *row_s = ps + (size_t)f * stride;
    if (lane == 0u) row_v[0] = s.cur;
    unsigned long long *seg = s_seg + (threadIdx.x >> 5) * kSegs;
    int r;
    do {
        const uint32_t at = s.step;
        bool moved;
        uint2 taken;
        uint32_t taken_at;
        r = step_weighted_warp<false>(s, lane == 0u, g, ix, max_steps, 0.f, key, seg, lane, &moved,
                                      &taken, &taken_at);
        r = __shfl_sync(kFull, r, 0);
        if (lane == 0u && moved && at < stride) {
            row_v[at] = taken.x;
            row_s[at] = taken_at;
        }
    } while (r == kContinue);
    if (lane == 0u) {
        const int32_t found = (r == kFound) ? (int32_t)s.step : -1;
        plen[f] = found;
        if (found != key_found(k)) atomicOr(scalars + S_ERR, (unsigned long long)kErrPath);
    }
}

// Walkers handed to a warp at a time: 32 by default, so that the 512 walks
// of an edge nobody connects spread over 16 warps instead of running as 16
// waves on one; 64 for uniform insertion batches of 2M walkers and more, and
// deletion batches of 4M (a part of which is walked), which fill the device
// many times over, so that half as many chunks are fetched (uniform
// walks with 32 and 64, ms a call: 200,000 insertions of the 100^3 mesh in ten
// batches 4.45 and 4.07, in batches of 5,000 0.68 and 0.63 per 25,000; 297,000
// deletions 2.29 and 1.91; but rounds of 2,400 insertions 0.93 and 1.08, of
// 100 insertions 0.22 and 0.30).  DYG_WALK_CHUNK (a multiple of 32 dividing
// the walker count) overrides it for tuning sweeps.
constexpr uint64_t kBigChunkWalkers = 2u << 20;
// Launch shape of the walk kernel, process-wide (dyg_tune_set); 0 = default.
static std::atomic<uint32_t> g_tune_chunk{0}, g_tune_bpsm{0}, g_tune_prune{0};

// Iterations between reads of an edge's best result for pruning (1, 2 or 4).
static uint32_t prune_every() {
    const uint32_t t = g_tune_prune.load();
    return (t == 2u || t == 4u) ? t : 1u;
}

// Weighted deletion walks take 16 in batches of up to 2M walkers: their walks
// are long-tailed, and a warp with fewer of them waits less for its slowest
// (12,000 deletions of a 40^3 mesh in ten batches 2.47 -> 2.16 ms of walks;
// insertions 1.51 -> 1.59).  Where the batch fills the device many times over,
// fetching twice as many chunks costs more (calls of one batch, 512 walkers, us
// with 16 and 32: random geometric graph of 400,000 vertices, 1,000 deletions 504
// and 503, 4,000 765 and 735, 8,000 1,093 and 1,016, 16,000 1,902 and 1,732; 100^3
// mesh 430 and 494, 847 and 861, 1,378 and 1,359, 2,408 and 2,344).
static uint32_t chunk_for(uint32_t n, uint32_t walkers, bool weighted, bool incremental) {
    static int env = -1;
    if (env < 0) {
        const char *v = getenv("DYG_WALK_CHUNK");
        env = v ? atoi(v) : 0;
    }
    const uint32_t want = g_tune_chunk.load() ? g_tune_chunk.load() : (uint32_t)(env > 0 ? env : 0);
    const uint64_t all = (uint64_t)n * walkers;
    uint32_t c = weighted && !incremental && all < kBigChunkWalkers ? 16u : 32u;
    if (!weighted && walkers % 64u == 0u && all >= kBigChunkWalkers * (incremental ? 1u : 2u)) c = 64u;
    if (want > 0 && want % 32 == 0 && walkers % want == 0) c = want;
    return c;
}

// The persistent grid: as many blocks as fit (or dyg_tune_set allows), but no
// more warps than there are chunks, since each idle warp costs an atomic on
// the chunk counter: a 32-edge batch has 512 chunks for 7,104 warps.
template <auto Kernel>
static uint32_t walk_blocks(uint32_t n, uint32_t walkers, uint32_t chunk) {
    static const int per_sm = [] {
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, Kernel, kWalkThreads, 0);
        return nb < 1 ? 1 : nb;
    }();
    const uint32_t t = g_tune_bpsm.load();
    const uint64_t fit = (uint64_t)((t && (int)t < per_sm) ? (int)t : per_sm) * num_sms();
    // four chunks' warps to a block of eight while SMs are idle: half-empty
    // blocks spread a small batch over more of them
    const uint64_t want = ((uint64_t)n * (walkers / chunk) + 3) / 4;
    return (uint32_t)(want < 1 ? 1 : (want < fit ? want : fit));
}

template <auto Kernel>
static void launch_walk_kernel(const WalkArgs &a, cudaStream_t st) {
    uint32_t blocks = walk_blocks<Kernel>(a.job.n_host, a.walkers, a.chunk);
    if (a.rec.heads && blocks > a.rec.threads / kWalkThreads) blocks = a.rec.threads / kWalkThreads;
    Kernel<<<blocks, kWalkThreads, 0, st>>>(a);
}

uint32_t walk_threads(uint32_t n, const dyg_walk_params &p) {
    const uint32_t c = chunk_for(n, p.walkers, p.transition == DYG_TRANSITION_WEIGHTED, false);
    return kWalkThreads * (p.transition == DYG_TRANSITION_WEIGHTED
                               ? walk_blocks<k_walk_weighted<false>>(n, p.walkers, c)
                               : walk_blocks<k_walk_uniform<false, true>>(n, p.walkers, c));
}

static void launch_walk_any(const WalkArgs &a, bool incremental, bool wtd, cudaStream_t st) {
    if (incremental) {
        if (wtd) launch_walk_kernel<k_walk_weighted<true>>(a, st);
        else launch_walk_kernel<k_walk_uniform<true, false>>(a, st);
    } else {
        if (wtd) launch_walk_kernel<k_walk_weighted<false>>(a, st);
        else if (a.rec.heads) launch_walk_kernel<k_walk_uniform<false, true>>(a, st);
        else launch_walk_kernel<k_walk_uniform<false, false>>(a, st);
    }
}

// Words the index may take: what rows filling the whole arena would need
// (fewer than 4 deg table words and 2 deg prefix words each), at most 2 GB;
// rows that do not fit stay without an index.
constexpr uint64_t kIdxWordsMax = 1ull << 29;

dyg_status index_enqueue(dyg_graph *G, uint32_t edges, const dyg_walk_params &p, bool incremental,
                         unsigned long long *halt, WalkScratch &scratch, RowIndex *out, cudaStream_t st) {
    *out = RowIndex{};
    if (p.transition != DYG_TRANSITION_WEIGHTED || !G->long_rows) return DYG_OK;
    Workspace &ws = G->ws;
    const uint32_t n = G->g.n;
    const size_t rows = ((size_t)n + 1) & ~(size_t)1;   // words before the index's, which are read in pairs
    if (!scratch.index_tried) {
        uint64_t words = 6ull * G->g.arena_cap + 2ull;
        if (words > kIdxWordsMax) words = kIdxWordsMax;
        scratch.index_tried = true;
        if (scratch_borrow(&scratch.index, sizeof(uint32_t) * (2 * rows + (size_t)words)) != cudaSuccess)
            cudaGetLastError();
    }
    // where memory is short, the walks search their long rows without an index
    if (!scratch.index.p) return DYG_OK;
    const uint64_t room = scratch.index.bytes / sizeof(uint32_t) - 2 * rows;
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    DYG_CUDA(cudaMemsetAsync(sc + S_IDX, 0, 3 * sizeof(unsigned long long), st));
    IndexArgs a{};
    a.g = G->g;
    a.rbase = ptr<uint32_t>(scratch.index);
    a.list = a.rbase + rows;
    a.words = a.list + rows;
    a.cap = (uint32_t)(room < kIdxWordsMax ? room : kIdxWordsMax);
    a.cursor = sc + S_IDX;
    a.counts = sc + S_IDXN;
    a.sums = sc + S_IDXSUM;
    a.budget = (unsigned long long)edges * p.walkers * (incremental ? kIdxInsertSlots : 1u);
    a.all = a.budget >= G->g.arena_cap;
    a.halt = halt;
    DYG_TRY(launch_phases<k_index>(2u * (uint32_t)num_sms(), st, grid_bar(G, halt), a));
    *out = RowIndex{a.rbase, a.words};
    return DYG_OK;
}

dyg_status launch_walk(dyg_graph *G, const WalkJob &job, const dyg_walk_params &p, bool incremental,
                       unsigned long long *keys, const RowIndex &ix, cudaStream_t st,
                       bool counter_zero, const PathRec *rec) {
    WalkArgs a{};
    a.g = G->g;
    a.ix = ix;
    if (rec) a.rec = *rec;
    a.job = job;
    a.walkers = p.walkers;
    a.max_steps = p.max_steps;
    a.prune = (p.flags & DYG_FLAG_EXHAUSTIVE) ? 0u : 1u;
    a.prune_every = prune_every();
    a.chunk = chunk_for(job.n_host, p.walkers, p.transition == DYG_TRANSITION_WEIGHTED, incremental);
    a.threshold = p.threshold;
    a.key = make_uint2((uint32_t)p.seed, (uint32_t)(p.seed >> 32));
    a.keys = keys;
    a.scalars = ptr<unsigned long long>(G->ws.scalars);
    if (!counter_zero) DYG_CUDA(cudaMemsetAsync(a.scalars + S_WORK, 0, sizeof(unsigned long long), st));
    ProfScope prof(incremental ? 0 : 1, st);
    launch_walk_any(a, incremental, p.transition == DYG_TRANSITION_WEIGHTED, st);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

// Same launch as launch_walk, with the kernel's counters (work chunks,
// error bits, move counts) at `scalars` instead of the handle's workspace, and
// without profiling events.
dyg_status launch_walk_scalars(const DevGraph &g, const WalkJob &job, const dyg_walk_params &p,
                               bool incremental, unsigned long long *keys,
                               unsigned long long *scalars, cudaStream_t st) {
    WalkArgs a{};
    a.g = g;
    a.job = job;
    a.walkers = p.walkers;
    a.max_steps = p.max_steps;
    a.prune = (p.flags & DYG_FLAG_EXHAUSTIVE) ? 0u : 1u;
    a.prune_every = prune_every();
    a.chunk = chunk_for(job.n_host, p.walkers, p.transition == DYG_TRANSITION_WEIGHTED, incremental);
    a.threshold = p.threshold;
    a.key = make_uint2((uint32_t)p.seed, (uint32_t)(p.seed >> 32));
    a.keys = keys;
    a.scalars = scalars;
    launch_walk_any(a, incremental, p.transition == DYG_TRANSITION_WEIGHTED, st);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

dyg_status launch_winner_paths(dyg_graph *G, const WalkJob &job, const dyg_walk_params &p,
                               const unsigned long long *keys, uint32_t n_max, uint32_t stride,
                               uint32_t *path_v, uint32_t *path_s, int32_t *path_len, const RowIndex &ix,
                               cudaStream_t st) {
    if (n_max == 0) return DYG_OK;
    const uint2 key = make_uint2((uint32_t)p.seed, (uint32_t)(p.seed >> 32));
    const int threads = 128;
    const int grid = (int)((n_max + threads - 1) / threads);
    unsigned long long *sc = ptr<unsigned long long>(G->ws.scalars);
    ProfScope prof(2, st);
    if (p.transition == DYG_TRANSITION_WEIGHTED)
        k_winner_paths_weighted<<<(unsigned)(((uint64_t)n_max * 32 + kReplayThreads - 1) / kReplayThreads),
                                  kReplayThreads, 0, st>>>(G->g, job, ix, p.max_steps, key, keys, stride,
                                                           path_v, path_s, path_len, sc);
    else
        k_winner_paths<<<grid, threads, 0, st>>>(G->g, job, p.max_steps, key, keys, stride,
                                                        path_v, path_s, path_len, sc);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

}  // namespace dyg

extern "C" {

dyg_status dyg_profile_enable(int on) {
    std::lock_guard<std::mutex> lk(dyg::g_prof_mu);
    dyg::g_prof_on = on != 0;
    return DYG_OK;
}

dyg_status dyg_profile_reset(void) {
    std::lock_guard<std::mutex> lk(dyg::g_prof_mu);
    dyg::prof_flush_locked();
    dyg::g_prof_acc = dyg_profile{};
    return DYG_OK;
}

dyg_status dyg_profile_read(dyg_profile *out) {
    if (!out) return DYG_EINVAL;
    std::lock_guard<std::mutex> lk(dyg::g_prof_mu);
    dyg::prof_flush_locked();
    *out = dyg::g_prof_acc;
    return DYG_OK;
}

}  // extern "C"

extern "C" void dyg_tune_set_prune_interval(uint32_t iterations) {
    dyg::g_tune_prune.store(iterations);
}

extern "C" void dyg_tune_set(uint32_t walk_chunk, uint32_t blocks_per_sm) {
    dyg::g_tune_chunk.store(walk_chunk);
    dyg::g_tune_bpsm.store(blocks_per_sm);
}
