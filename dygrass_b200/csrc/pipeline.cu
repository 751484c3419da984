// pipeline.cu -- the incremental and decremental update pipelines.
//
// A whole update stream is enqueued on one CUDA stream with no host
// round-trip: counts stay on the device, everything a batch does besides
// walking is one or two launches whose phases meet at grid barriers
// (gridsync.cuh, rowops.cuh), and the only host check is a single synchronize
// at the end.  A reservation that does not fit (arena or record buffers)
// halts every later kernel; the host then grows the buffer and resumes at the
// halted batch and phase, which reproduces the same results because no kernel
// changed anything after the halt.
//
// Incremental batch (one iteration of random_walk_incremental/main.cu:314-340):
//   walk H -> k_append: decode winner keys, accepted edges to H [and every
//   edge to G] in input order, reserved together.  Resumes at the batch start
//   (nothing of the batch changed).
// Decremental batch (random_walk_decremental/main.cu:413-444), phases:
//   0: k_delete: delete from G and H in input order, list the edges found in
//      both; walk G; replay winners; k_recover: path candidates in (edge,
//      step) order, then the 2-step fallback walks' candidates for the edges
//      without a path,
//   1: and their dedup (first occurrence), those in H dropped, the rest
//      appended in order (path edges, then fallback edges).
#include "dyg_internal.cuh"
#include "gridsync.cuh"
#include "rowops.cuh"

namespace dyg {

namespace {

int grid_for(uint64_t m) {
    const uint64_t b = (m + 255) / 256;
    const uint64_t cap = (uint64_t)num_sms() * 8;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

#define GSTRIDE(i, m) \
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (m); i += gridDim.x * blockDim.x)

// ------------------------------------------------------- input check

__global__ void k_validate(unsigned long long *halt, const uint32_t *src, const uint32_t *dst,
                           const float *w, uint32_t n, uint32_t nv, unsigned long long *err) {
    GSTRIDE(e, n) {
        unsigned long long bits = 0ull;
        if (src[e] >= nv || dst[e] >= nv) bits |= kErrVertex;
        if (w) {
            const float x = w[e];
            if (!(x > 0.0f) || !isfinite(x)) bits |= kErrWeight;
        }
        if (bits) {
            atomicOr(err, bits);
            atomicCAS(halt, 0ull, halt_code(0, (uint32_t)kHaltInvalid, 0));
        }
    }
}

// --------------------------------------------------------- incremental

// Incremental commit of one batch: edge e is decoded from its winner key
// (found step, conductance, accept flag; keys[e] = 0: no walker connected the
// edge); an accepted edge goes to H, u gets v, then v gets u
// (random_walk_incremental/gpu_graph.cuh:320-325), and with G every edge goes
// to G.  With `clear` the key is zeroed behind the decode, so that the next
// batch's walks need no memset.
struct IncrOp {
    static constexpr bool kList = false, kPrep = false;
    unsigned long long *keys;
    int32_t *found;
    float *cond;
    uint8_t *acc;
    uint32_t n;
    bool clear;
    __device__ uint32_t count() const { return n; }
    __device__ uint32_t take(uint32_t e) const {
        const unsigned long long k = keys[e];
        if (clear && k) keys[e] = 0ull;
        if (found) found[e] = key_found(k);
        if (cond) cond[e] = k ? __uint_as_float((uint32_t)(k >> 32)) : 0.f;
        if (acc) acc[e] = k ? 0 : 1;
        return k ? 2u : 3u;
    }
};

// ---------------------------------------------------------- decremental

// Deletion stage of a batch in one launch.
//   link    the half-edges of every deletion, endpoints ordered min -> max
//           (random_walk_decremental/gpu_graph.cuh:340-343), chained per row;
//           the rows of G and H have the same entries, so one set of chains
//           serves both
//   G, H    rows edited in list order, H's entries only where G found the
//           edge on both sides; the rows of G that are not for a lane are
//           listed first and get a phase of their own when there are any
//   list    deletion e found in G and in H goes to the walk list at its
//           position in input order: min -> max, or with file_orient in file
//           orientation; every deletion gets its status code
struct DeleteArgs {
    DevGraph G, H;
    DelList D;
    uint32_t n;
    bool file_orient;
    unsigned long long uid0;
    const unsigned long long *uids;
    uint8_t *fG, *fH;   // per half-edge: found (2-byte aligned)
    int32_t *status;
    float *cond;
    uint32_t *f_src, *f_dst, *f_idx;
    unsigned long long *f_uid;
    unsigned long long *keys, *work;   // zeroed for the walks
    uint32_t *rec_head;                // as well
    uint32_t *blk, *counts;
    unsigned long long *err;
    const unsigned long long *halt;
};

__global__ void __launch_bounds__(kOpThreads, 2) k_delete(const __grid_constant__ DeleteArgs a, GridBar bar) {
    __shared__ RowShared s;
    if (*a.halt) return;
    const uint2 rg = block_range(a.n);
    for (uint32_t e = rg.x + threadIdx.x; e < rg.y; e += blockDim.x) {
        const uint2 v = del_ends(a.D.src, a.D.dst, e);
        const bool ok = v.y < a.G.n;
        if (!ok) atomicOr(a.err, (unsigned long long)kErrVertex);
        link_entry(a.D.c, 2u * e, v.x, ok);
        link_entry(a.D.c, 2u * e + 1u, v.y, ok);
        reinterpret_cast<uint16_t *>(a.fG)[e] = 0;
        reinterpret_cast<uint16_t *>(a.fH)[e] = 0;
        a.keys[e] = 0ull;
        a.rec_head[e] = 0u;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.work = 0ull;
    if (!grid_sync(bar, [&] { *a.D.c.items = *a.D.items_h = *a.D.c.cursor = 0ull; })) return;
    const uint32_t m = 2u * a.n;
    del_list(a.G, a.H, a.D, m);
    __syncthreads();   // the marks of this block's entries are set
    del_lane_rows(a.G, a.D, m, 1u, nullptr, a.fG, false);
    if (!grid_sync(bar)) return;
    const unsigned long long items_g = __ldcg(a.D.c.items), items_h = __ldcg(a.D.items_h),
                             runs = __ldcg(a.D.c.cursor);
    if (runs >> 32) {
        fill_runs(a.D.c, m, [&](uint32_t i) { return del_row(a.D, i); });
        if (!grid_sync(bar)) return;
    }
    if (items_g) {
        del_listed_rows(a.G, a.D, a.D.c.list, items_g, m, false, nullptr, a.fG, false, s);
        if (!grid_sync(bar)) return;
    }
    del_lane_rows(a.H, a.D, m, 2u, a.fG, a.fH, true);
    del_listed_rows(a.H, a.D, a.D.list_h, items_h, m, true, a.fG, a.fH, true, s);
    if (!grid_sync(bar)) return;
    uint32_t mine = 0u;
    for (uint32_t e = rg.x + threadIdx.x; e < rg.y; e += blockDim.x) {
        const bool inG = a.fG[2 * e] && a.fG[2 * e + 1];
        const bool inH = inG && a.fH[2 * e] && a.fH[2 * e + 1];
        a.status[e] = !inG ? DYG_DEL_NOT_IN_G : (!inH ? DYG_DEL_NOT_IN_H : DYG_DEL_NO_PATH);
        a.cond[e] = 0.f;
        mine += inH ? 1u : 0u;
    }
    const uint32_t sum = block_sum(mine, s.warp);
    if (threadIdx.x == 0) a.blk[blockIdx.x] = sum;
    if (!grid_sync(bar)) return;
    uint32_t base = blocks_before(a.blk, s.warp).x;
    for (uint32_t t = rg.x; t < rg.y; t += blockDim.x) {
        const uint32_t e = t + threadIdx.x;
        // in G and H on both sides (H's flags are set only where G's are)
        const bool on = e < rg.y && a.fH[2 * e] && a.fH[2 * e + 1];
        uint32_t total;
        const uint32_t f = base + block_excl(on ? 1u : 0u, s.warp, &total);
        if (on) {
            const uint2 v = del_ends(a.D.src, a.D.dst, e);
            a.f_src[f] = a.file_orient ? a.D.src[e] : v.x;
            a.f_dst[f] = a.file_orient ? a.D.dst[e] : v.y;
            a.f_uid[f] = a.uids ? a.uids[e] : a.uid0 + e;
            a.f_idx[f] = e;
        }
        base += total;
    }
    if (blockIdx.x == gridDim.x - 1u && threadIdx.x == 0) a.counts[C_FILTERED] = base;
}

// ------------------------------------------------------------- recovery

__device__ __forceinline__ unsigned long long ekey(uint32_t x, uint32_t y) {
    const uint32_t a = min(x, y), b = max(x, y);
    return ((unsigned long long)a << 32) | b;
}
__device__ __forceinline__ uint32_t hslot(unsigned long long k, uint32_t mask) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return (uint32_t)k & mask;
}

// 2-step fallback walk j of side `side` of walk-list entry f, which found no
// path (random_walk_decremental/main.cu:243-290, with the second step reading
// the row of the vertex the walker stands on): its candidates (s0, x1) and
// (x1, x2) with their weights; x = ~0u marks none.
struct Fallback {
    uint32_t s0, x1, x2;
    float w1, w2;
};
__device__ __forceinline__ Fallback fallback_walk(const DevGraph &g, uint32_t s0,
                                                  unsigned long long uid, uint32_t walker,
                                                  uint2 key) {
    const uint4 rb = philox4x32_10(make_uint4(0u, walker, (uint32_t)uid, ctr3_of(uid, kDomainHeur)), key);
    Fallback r{s0, ~0u, ~0u, 0.f, 0.f};
    const uint2 d0 = g.desc[s0];
    if (d0.y == 0u) return r;
    const uint32_t i0 = d0.x + rb.x % d0.y;
    r.x1 = g.slots[i0].x;
    r.w1 = g.wts[i0];
    const uint2 d1 = g.desc[r.x1];
    if (d1.y != 0u) {
        uint32_t i1 = d1.x + rb.y % d1.y;
        if (g.slots[i1].x == s0) i1 = d1.x + d1.y - 1u;
        r.x2 = g.slots[i1].x;
        r.w2 = g.wts[i1];
    }
    return r;
}

// Walk results, recovery candidates and their commit in one launch.
//   results    status and conductance of each walked deletion; path lengths
//              (the winner's step count) and edges without a path summed per
//              block
//   candidates path edges of walk-list entry f at its scanned offset (one
//              thread per edge; each edge's vertices and weight from the G slots
//              the winner took, as its record or its replay has them: G is
//              unchanged since), then, after all path candidates,
//              the fallback walks of the edges without a path
//              (main.cu:400-408, 428-436); each enters the dedup table
//   keep       candidate i is kept if it is the first occurrence of its edge
//              and the edge is not in H (gpu_graph.cuh:534-538 and 599-601
//              test sparse_map the same way); H membership scans the shorter
//              of the two rows
//   emit       kept candidates to the recovered-edge records and to H
//              (x gets y, then y gets x), in candidate order
// Path recovery (gpu_graph.cuh:514-552) and the fallback edges
// (gpu_graph.cuh:577-615) in one pass keep what the two in turn keep: a
// fallback edge equal to an earlier candidate is a repeat, every other one is
// tested against H as before, and appends and records follow candidate order.
struct RecoverArgs {
    DevGraph G, H;
    AppSides A;   // H's append of the kept candidates
    WalkJob job;
    bool resume;   // the candidates are there: only their commit is missing
    unsigned long long *keys;   // winner keys of the walk list
    bool clear_keys;
    PathRec rec;                // winners' paths: records, or (rec.heads null) replayed:
    const int32_t *plen;
    const uint32_t *pv, *ps;
    uint32_t stride, hw;
    const uint32_t *f_idx;
    uint2 key;
    int32_t *status;
    float *cond;
    uint32_t *cx, *cy;
    float *cw;
    unsigned long long *tk;   // dedup table, empty (~0) between launches
    uint32_t *tv;
    uint32_t *keep;
    uint32_t *rx, *ry;
    uint8_t *rk;
    uint32_t *blk, *counts;
    unsigned long long *sc;   // G's scalars
    unsigned long long *halt;
    unsigned long long code_records, code_arena, code_paths;
};

// Mask of the dedup table for M candidates: 2M slots at least, 1,024 at least, as
// the host sizes it.  In 64 bits: 2M does not fit 32 from M = 2^31 on, and the
// doubling would not end from 2^30 + 1 on.
__host__ __device__ constexpr uint32_t dedup_mask(uint32_t M) {
    uint64_t T = 1024;
    while (T < 2ull * M) T <<= 1;
    return (uint32_t)(T - 1);
}
static_assert(dedup_mask(0) == 1023u && dedup_mask(512) == 1023u && dedup_mask(513) == 2047u, "sizes");
static_assert(dedup_mask(1u << 30) == 0x7FFFFFFFu && dedup_mask((1u << 30) + 1u) == 0xFFFFFFFFu, "sizes");

__device__ __forceinline__ void cand_put(const RecoverArgs &a, uint32_t i, uint32_t x, uint32_t y,
                                         float w, uint32_t mask, bool store) {
    if (store) {
        a.cx[i] = x;
        a.cy[i] = y;
        a.cw[i] = w;
    }
    if (x == ~0u || y == ~0u || x == y) return;
    const unsigned long long k = ekey(x, y);
    uint32_t h = hslot(k, mask);
    while (true) {
        const unsigned long long prev = atomicCAS(a.tk + h, ~0ull, k);
        if (prev == ~0ull || prev == k) {
            atomicMin(a.tv + h, i);
            return;
        }
        h = (h + 1u) & mask;
    }
}

// First occurrence of a real edge; H membership is tested unless the shorter
// row is longer than kBigRow (*big).
__device__ __forceinline__ bool cand_keep(const RecoverArgs &a, uint32_t i, uint32_t mask,
                                          RowItem *big) {
    big->cnt = 0u;
    const uint32_t x = a.cx[i], y = a.cy[i];
    if (x == ~0u || y == ~0u || x == y) return false;
    const unsigned long long k = ekey(x, y);
    uint32_t h = hslot(k, mask);
    while (a.tk[h] != k) h = (h + 1u) & mask;
    if (a.tv[h] != i) return false;
    const uint2 dx = a.H.desc[x], dy = a.H.desc[y];
    const bool xs = dx.y <= dy.y;
    const uint2 d = xs ? dx : dy;
    const uint32_t other = xs ? y : x;
    if (d.y > kBigRow) {
        *big = RowItem{other, 1u, 0u, d.x, d.y, i};
        return true;
    }
    // eight columns loaded before they are compared
    for (uint32_t j0 = 0; j0 < d.y; j0 += 8u) {
        uint32_t cv[8];
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u) cv[u] = j0 + u < d.y ? a.H.slots[d.x + j0 + u].x : ~0u;
        bool hit = false;
#pragma unroll
        for (uint32_t u = 0; u < 8u; ++u) hit |= cv[u] == other;
        if (hit) return false;
    }
    return true;
}

__global__ void __launch_bounds__(kOpThreads, 2) k_recover(const __grid_constant__ RecoverArgs a,
                                                           GridBar bar) {
    __shared__ RowShared s;
    __shared__ uint32_t s_off[kOpThreads], s_rec[kOpThreads], s_none[kOpThreads];
    if (*a.halt) return;
    uint32_t n_path, M;
    uint32_t mask;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.sc[S_WORK] = 0ull;   // the next walk's chunk counter
    if (!a.resume) {
        const uint32_t F = job_count(a.job);
        const uint2 rg = block_range(F);
        uint32_t len = 0u, none = 0u;
        for (uint32_t f = rg.x + threadIdx.x; f < rg.y; f += blockDim.x) {
            const uint32_t e = a.f_idx[f];
            const unsigned long long k = a.keys[f];
            const int32_t L = a.rec.heads ? key_found(k) : a.plen[f];
            a.status[e] = L > 0 ? L : DYG_DEL_NO_PATH;
            a.cond[e] = k ? __uint_as_float((uint32_t)(k >> 32)) : 0.f;
            if (L > 0) len += (uint32_t)L;
            else ++none;
        }
        len = block_sum(len, s.warp);
        none = block_sum(none, s.warp);
        if (threadIdx.x == 0) {
            a.blk[blockIdx.x] = len;
            a.blk[kOpBlocksMax + blockIdx.x] = none;
        }
        // path records that did not fit halt the batch before anything else of
        // it changes; its walks are repeated with room for them
        if (!grid_sync(bar, [&] {
                if (!a.rec.heads) return;
                const unsigned long long used = __ldcg(a.rec.cursor);
                *a.rec.cursor = 0ull;
                if (used > a.rec.cap) {
                    a.sc[S_RECNEED] = used;
                    *a.halt = a.code_paths;
                }
            }))
            return;
        if (*(volatile unsigned long long *)a.halt == a.code_paths) {
            for (uint32_t f = rg.x + threadIdx.x; f < rg.y; f += blockDim.x) {
                a.rec.heads[f] = 0u;
                if (a.clear_keys) a.keys[f] = 0ull;
            }
            return;
        }
        const uint2 pl = blocks_before(a.blk, s.warp);
        const uint2 pn = blocks_before(a.blk + kOpBlocksMax, s.warp);
        n_path = pl.y;
        M = n_path + pn.y * 4u * a.hw;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.counts[C_CANDS] = n_path;
            a.counts[C_CANDS_ALL] = M;
        }
        mask = dedup_mask(M);
        uint32_t at = pl.x, nth = pn.x;
        for (uint32_t t = rg.x; t < rg.y; t += blockDim.x) {
            // one thread per walked deletion finds its winner's path and where
            // its candidates go ...
            const uint32_t q = threadIdx.x, f = t + q;
            uint32_t l = 0u, z = 0u;
            if (f < rg.y) {
                const unsigned long long key = a.keys[f];
                const int32_t L = a.rec.heads ? key_found(key) : a.plen[f];
                l = L > 0 ? (uint32_t)L : 0u;
                z = l ? 0u : 1u;
                if (a.rec.heads) {
                    uint32_t r = a.rec.heads[f];
                    a.rec.heads[f] = 0u;
                    if (l)
                        while (a.rec.words[r] != (uint32_t)key || a.rec.words[r + 1u] != (uint32_t)(key >> 32))
                            r = a.rec.words[r - 1u];
                    s_rec[q] = r + 2u;
                }
                if (a.clear_keys) a.keys[f] = 0ull;
            }
            uint32_t tl, tz;
            const uint32_t ol = block_excl(l, s.warp, &tl), oz = block_excl(z, s.warp, &tz);
            s_off[q] = ol;
            if (z) s_none[oz] = q;
            __syncthreads();
            // ... and one per candidate writes it
            for (uint32_t c = threadIdx.x; c < tl; c += blockDim.x) {
                uint32_t lo = 0u, hi = blockDim.x;   // the last path that starts at or before c
                while (hi - lo > 1u) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (s_off[mid] <= c) lo = mid;
                    else hi = mid;
                }
                const uint32_t fq = t + lo, j = c - s_off[lo];
                if (a.rec.heads) {
                    const uint32_t *sl = a.rec.words + s_rec[lo];
                    const uint32_t slot = sl[j];
                    const uint32_t x = j ? a.G.slots[sl[j - 1u]].x : a.job.src[fq];
                    cand_put(a, at + c, x, a.G.slots[slot].x, a.G.wts[slot], mask, true);
                } else {
                    const uint32_t *v = a.pv + (size_t)fq * a.stride, *sl = a.ps + (size_t)fq * a.stride;
                    cand_put(a, at + c, v[j], v[j + 1], a.G.wts[sl[j + 1]], mask, true);
                }
            }
            const uint32_t per = 2u * a.hw;   // fallback walks of an edge without a path
            for (uint32_t c = threadIdx.x; c < tz * per; c += blockDim.x) {
                const uint32_t k = c / per, j = c - k * per, fq = t + s_none[k];
                const uint32_t base = n_path + ((nth + k) * per + j) * 2u;
                const Fallback r = fallback_walk(a.G, j < a.hw ? a.job.src[fq] : a.job.dst[fq], a.job.uid[fq],
                                                 j, a.key);
                cand_put(a, base, r.x1 == ~0u ? ~0u : r.s0, r.x1, r.w1, mask, true);
                cand_put(a, base + 1u, r.x2 == ~0u ? ~0u : r.x1, r.x2, r.w2, mask, true);
            }
            at += tl;
            nth += tz;
            __syncthreads();   // the tile's shared arrays are written again by the next
        }
    } else {
        n_path = a.counts[C_CANDS];
        M = a.counts[C_CANDS_ALL];
        mask = dedup_mask(M);
        GSTRIDE(i, M) cand_put(a, i, a.cx[i], a.cy[i], 0.f, mask, false);
    }
    if (!grid_sync(bar)) return;
    const uint2 rg = block_range(M);
    uint32_t kept = 0u;
    for (uint32_t t = rg.x; t < rg.y; t += blockDim.x) {
        if (threadIdx.x == 0) s.nbig = 0u;
        __syncthreads();
        const uint32_t i = t + threadIdx.x;
        bool kp = false;
        if (i < rg.y) {
            RowItem b;
            kp = cand_keep(a, i, mask, &b);
            if (b.cnt) s.item[atomicAdd(&s.nbig, 1u)] = b;
            a.keep[i] = kp ? 1u : 0u;
        }
        __syncthreads();
        const uint32_t nbig = s.nbig;
        for (uint32_t q = 0; q < nbig; ++q) {   // both rows are hub rows
            const RowItem b = s.item[q];
            if (block_find(a.H.slots, b.old_off, b.deg, b.x, &s.best) != ~0u && i == b.off) {
                a.keep[i] = 0u;
                kp = false;
            }
        }
        kept += kp ? 1u : 0u;
        __syncthreads();
    }
    kept = block_sum(kept, s.warp);
    if (threadIdx.x == 0) {
        a.blk[blockIdx.x] = kept;
        if (kept) atomicAdd(a.sc + S_KEPT, (unsigned long long)kept);
    }
    // the kept edges must fit the record buffers, or the batch halts here and
    // is resumed with larger ones
    if (!grid_sync(bar, [&] {
            const unsigned long long k = __ldcg(a.sc + S_KEPT);
            a.sc[S_KEPT] = 0ull;
            *a.A.s[0].c.items = *a.A.s[0].c.cursor = 0ull;
            if (a.sc[S_RECCNT] + k > a.sc[S_RECCAP]) *a.halt = a.code_records;
        }))
        return;
    for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= mask; i += gridDim.x * blockDim.x) {
        a.tk[i] = ~0ull;   // the table as it was found
        a.tv[i] = ~0u;
    }
    if (*(volatile unsigned long long *)a.halt == a.code_records) return;
    const uint2 pk = blocks_before(a.blk, s.warp);
    const unsigned long long rec0 = a.sc[S_RECCNT];
    uint32_t base = pk.x;
    for (uint32_t t = rg.x; t < rg.y; t += blockDim.x) {
        const uint32_t i = t + threadIdx.x;
        const uint32_t kp = i < rg.y ? a.keep[i] : 0u;
        uint32_t total;
        const uint32_t q = base + block_excl(kp, s.warp, &total);
        base += total;
        if (i < rg.y) {
            const uint32_t x = a.cx[i], y = a.cy[i];
            link_entry(a.A.s[0].c, 2u * i, x, kp && x < a.H.n);
            link_entry(a.A.s[0].c, 2u * i + 1u, y, kp && y < a.H.n);
            if (kp) {
                a.rx[rec0 + q] = x;
                a.ry[rec0 + q] = y;
                a.rk[rec0 + q] = i < n_path ? DYG_REC_PATH : DYG_REC_FALLBACK;
            }
        }
    }
    if (!grid_sync(bar)) return;
    app_commit(a.A, 2u * M, bar, a.halt, a.code_arena, s, [&] { a.sc[S_RECCNT] = rec0 + pk.y; });
}

}  // namespace

dyg_status validate_enqueue(unsigned long long *halt, unsigned long long *err,
                            const uint32_t *src, const uint32_t *dst, const float *w, uint32_t n,
                            uint32_t nv, cudaStream_t st) {
    if (n == 0) return DYG_OK;
    k_validate<<<grid_for(n), 256, 0, st>>>(halt, src, dst, w, n, nv, err);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

// A call whose device-resident inputs failed k_validate: clear the halt and
// the error bits, and report which check failed.  Nothing was changed.
dyg_status rejected_inputs(dyg_graph *D, cudaStream_t st) {
    const unsigned long long err = D->ws.host_scalars[S_ERR];
    DYG_CUDA(cudaMemsetAsync(ptr<unsigned long long>(D->ws.scalars) + S_ERR, 0,
                             sizeof(unsigned long long), st));
    DYG_CUDA(cudaMemsetAsync(ptr<unsigned long long>(D->ws.scalars) + S_HALT, 0,
                             sizeof(unsigned long long), st));
    DYG_CUDA(cudaStreamSynchronize(st));
    D->ws.host_scalars[S_ERR] = 0ull;
    D->ws.host_scalars[S_HALT] = 0ull;
    if (err & kErrVertex)
        set_error("a batch endpoint is not a vertex of the graph (the call changed nothing)");
    else
        set_error("a batch weight is not finite and > 0 (the call changed nothing)");
    return DYG_EINVAL;
}

dyg_status grow_keep(Buf &b, size_t bytes, size_t used, cudaStream_t st) {
    if (b.bytes >= bytes) return DYG_OK;
    Buf nb;
    DYG_TRY(ensure(nb, bytes));
    if (used && b.p) {
        DYG_CUDA(cudaMemcpyAsync(nb.p, b.p, used, cudaMemcpyDeviceToDevice, st));
        DYG_CUDA(cudaStreamSynchronize(st));
    }
    if (b.p) {
        if (!used) DYG_CUDA(cudaStreamSynchronize(st));
        dev_free(b.p);
    }
    b = nb;
    return DYG_OK;
}

// ------------------------------------------------------------ batches

// Commit half of an incremental batch from its winner keys (keys[e] = 0: no
// walker connected edge e): accepted edges to H [and every edge to G],
// reserved together.
dyg_status incr_commit_enqueue(dyg_graph *H, dyg_graph *G, const uint32_t *src,
                               const uint32_t *dst, const float *w, uint32_t n,
                               unsigned long long *keys, bool clear_keys,
                               unsigned long long *halt, uint32_t batch, int32_t *found,
                               float *cond, uint8_t *acc, cudaStream_t st) {
    const EdgeList E{src, dst, w};
    return append_enqueue(IncrOp{keys, found, cond, acc, n, clear_keys}, n, H, E, G, E,
                          ptr<unsigned long long>(H->ws.scalars) + S_WORK, halt,
                          halt_code(batch, (uint32_t)kHaltArena, 0), st);
}

// Incremental batch `batch` (edges src/dst/w[0, n), update ids uid0 + e).
// Outputs go to found/cond/acc (device, may be null).  walk_ready: the commit
// of the batch before left the keys and the walk's chunk counter zero.
static dyg_status incr_enqueue(dyg_graph *H, dyg_graph *G, const uint32_t *src, const uint32_t *dst,
                               const float *w, uint32_t n, uint64_t uid0,
                               const unsigned long long *uids, const dyg_walk_params &p,
                               unsigned long long *halt, uint32_t batch, int32_t *found, float *cond,
                               uint8_t *acc, cudaStream_t st, bool walk_ready, WalkScratch &scratch) {
    unsigned long long *keys = ptr<unsigned long long>(H->ws.keys);
    if (!walk_ready) DYG_CUDA(cudaMemsetAsync(keys, 0, sizeof(unsigned long long) * n, st));
    WalkJob job{halt, src, dst, w, uids, (unsigned long long)uid0, nullptr, n, kDomainIncr, 0u};
    RowIndex ix{};
    DYG_TRY(index_enqueue(H, n, p, true, halt, scratch, &ix, st));
    DYG_TRY(launch_walk(H, job, p, true, keys, ix, st, walk_ready));
    return incr_commit_enqueue(H, G, src, dst, w, n, keys, true, halt, batch, found, cond, acc, st);
}

dyg_status decr_delete_ensure(dyg_graph *G, dyg_graph *H, uint32_t n, cudaStream_t st) {
    Workspace &ws = G->ws;
    const uint64_t m = 2ull * n;
    DYG_TRY(rowops_ensure(G, m, st));
    DYG_TRY(rowops_ensure(H, m, st));
    DYG_TRY(ensure(ws.found, (size_t)m * 2));
    DYG_TRY(ensure(ws.keys, sizeof(unsigned long long) * n));
    DYG_TRY(ensure(ws.f_src, sizeof(uint32_t) * n));
    DYG_TRY(ensure(ws.f_dst, sizeof(uint32_t) * n));
    DYG_TRY(ensure(ws.f_idx, sizeof(uint32_t) * n));
    DYG_TRY(ensure(ws.f_uid, sizeof(unsigned long long) * n));
    return ensure(ws.rec_head, sizeof(uint32_t) * n);
}

// Deletion stage of a decremental batch: delete every edge from G (swap with
// the row's last slot, in input order), erase the ones also in H, and list
// the edges found in both (gpu_graph.cuh:338-458), each walked min -> max
// (random_walk_decremental/gpu_graph.cuh:342) or, with file_orient, src -> dst
// (dynamic_update/gpu_graph.cuh:874-875).  status/cond (device, length n) get
// the per-deletion codes.
dyg_status decr_delete_enqueue(dyg_graph *G, dyg_graph *H, const uint32_t *src,
                               const uint32_t *dst, uint32_t n, uint64_t uid0,
                               const unsigned long long *uids, bool file_orient,
                               unsigned long long *halt, int32_t *status, float *cond,
                               cudaStream_t st) {
    Workspace &ws = G->ws;
    const uint64_t m = 2ull * n;
    DYG_TRY(decr_delete_ensure(G, H, n, st));
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    DeleteArgs a{};
    a.G = G->g;
    a.H = H->g;
    a.D = DelList{append_side(G, src, dst, nullptr).c, src, dst, ptr<uint32_t>(H->ws.rowlist), ptr<unsigned long long>(H->ws.scalars) + S_ITEMS};
    a.n = n;
    a.file_orient = file_orient;
    a.uid0 = uid0;
    a.uids = uids;
    a.fG = ptr<uint8_t>(ws.found);
    a.fH = a.fG + m;
    a.status = status;
    a.cond = cond;
    a.f_src = ptr<uint32_t>(ws.f_src);
    a.f_dst = ptr<uint32_t>(ws.f_dst);
    a.f_idx = ptr<uint32_t>(ws.f_idx);
    a.f_uid = ptr<unsigned long long>(ws.f_uid);
    a.keys = ptr<unsigned long long>(ws.keys);
    a.work = sc + S_WORK;
    a.rec_head = ptr<uint32_t>(ws.rec_head);
    a.blk = ptr<uint32_t>(ws.blk);
    a.counts = ptr<uint32_t>(ws.counts);
    a.err = sc + S_ERR;
    a.halt = halt;
    return launch_phases<k_delete>(op_blocks(m, G->long_rows || H->long_rows), st, grid_bar(G, halt), a);
}

void WalkScratch::open_paths(dyg_graph *G, uint32_t n, const dyg_walk_params &p) {
    if (p.max_steps > kPathSteps || n == 0) return;
    if (p.transition == DYG_TRANSITION_UNIFORM && (uint64_t)n * p.walkers > kPathWalkers) return;
    Workspace &ws = G->ws;
    const uint32_t threads = walk_threads(n, p);
    const size_t hist_bytes = sizeof(uint32_t) * (size_t)threads * ((p.max_steps + 3u) & ~3u);
    // some paths of a few moves per edge to begin with
    const uint64_t want = (uint64_t)n * ws.rec_each + 4096u;
    edges = n;
    if (scratch_borrow(&hist, hist_bytes) != cudaSuccess ||
        scratch_borrow(&words, sizeof(uint32_t) * want) != cudaSuccess) {
        cudaGetLastError();
        scratch_return(&hist);   // nothing has used it
        return;
    }
    const uint64_t room = words.bytes / sizeof(uint32_t);
    rec.heads = ptr<uint32_t>(ws.rec_head);
    rec.words = ptr<uint32_t>(words);
    rec.cap = (uint32_t)(room > 0xFFFFFF00u ? 0xFFFFFF00u : room);
    rec.cursor = ptr<unsigned long long>(ws.scalars) + S_RECW;
    rec.hist = ptr<uint32_t>(hist);
    rec.threads = threads;
}

void WalkScratch::grow_paths(dyg_graph *G) {
    const unsigned long long need = G->ws.host_scalars[S_RECNEED] + G->ws.host_scalars[S_RECNEED] / 4;
    scratch_return(&words);   // the stream was waited for
    if (need > 0xFFFFFF00ull || scratch_borrow(&words, sizeof(uint32_t) * need) != cudaSuccess) {
        cudaGetLastError();
        rec = PathRec{};   // replay the winners instead
        return;
    }
    // the next call begins with as much, within reason: its edges may be others
    const unsigned long long each = need / edges + 1u;
    if (each > G->ws.rec_each) G->ws.rec_each = each < kPathSteps ? (uint32_t)each : kPathSteps;
    rec.words = ptr<uint32_t>(words);
    rec.cap = (uint32_t)need;
}

bool WalkScratch::release() {
    if (!hist.p && !words.p && !index.p) return false;
    cudaStreamSynchronize(st);
    for (Buf *b : {&hist, &words, &index}) scratch_return(b);
    rec = PathRec{};
    return true;
}

static uint32_t path_stride(const dyg_walk_params &p) { return p.max_steps > 2 ? p.max_steps : 2; }

dyg_status decr_walk_ensure(dyg_graph *G, dyg_graph *H, uint32_t n, const dyg_walk_params &p, cudaStream_t st) {
    Workspace &ws = G->ws;
    DYG_TRY(ensure(ws.keys, sizeof(unsigned long long) * n));
    // path candidates at [0, C_CANDS), then the fallback candidates
    const size_t n_path = (size_t)n * (path_stride(p) - 1u), n_fb = (size_t)n * 4u * p.heuristic_walkers,
                 M = n_path + n_fb;
    DYG_TRY(ensure(ws.cand_x, sizeof(uint32_t) * M));
    DYG_TRY(ensure(ws.cand_y, sizeof(uint32_t) * M));
    DYG_TRY(ensure(ws.cand_w, sizeof(float) * M));
    DYG_TRY(ensure(ws.keep, sizeof(uint32_t) * M));
    uint64_t T = 1024;
    while (T < 2ull * M) T <<= 1;
    if (ws.htab_k.bytes < sizeof(unsigned long long) * T || ws.htab_v.bytes < sizeof(uint32_t) * T) {
        // empty when allocated, and left empty by every recovery
        DYG_TRY(ensure(ws.htab_k, sizeof(unsigned long long) * T));
        DYG_TRY(ensure(ws.htab_v, sizeof(uint32_t) * T));
        DYG_CUDA(cudaMemsetAsync(ws.htab_k.p, 0xFF, ws.htab_k.bytes, st));
        DYG_CUDA(cudaMemsetAsync(ws.htab_v.p, 0xFF, ws.htab_v.bytes, st));
    }
    DYG_TRY(rowops_ensure(G, 1, st));
    return rowops_ensure(H, 2ull * M, st);
}

// Walk-and-recover stage over walk-list entries [f0, f0 + nf) (nf a host
// bound; F_dev, if given, is the device count of the whole list), from phase
// `phase0` (0 = walks, 1 = recovery, 2 = walks repeated with more room for
// their paths: the deletions are done).
dyg_status decr_walk_enqueue(dyg_graph *G, dyg_graph *H, uint32_t f0, uint32_t nf,
                             const uint32_t *F_dev, const dyg_walk_params &p,
                             unsigned long long *halt, uint32_t batch, uint32_t phase0,
                             int32_t *status, float *cond, cudaStream_t st, bool walk_ready,
                             WalkScratch &scratch, const unsigned long long *keys_given) {
    if (nf == 0) return DYG_OK;
    Workspace &ws = G->ws;
    const uint32_t n = nf;
    const uint32_t stride = path_stride(p);
    const uint32_t hwk = p.heuristic_walkers;
    DYG_TRY(decr_walk_ensure(G, H, n, p, st));
    const bool replay = keys_given || !scratch.rec.heads;
    if (replay) {
        DYG_TRY(ensure(ws.path_v, sizeof(uint32_t) * (size_t)n * stride));
        DYG_TRY(ensure(ws.path_s, sizeof(uint32_t) * (size_t)n * stride));
        DYG_TRY(ensure(ws.path_len, sizeof(int32_t) * n));
    }
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    WalkJob job{halt, ptr<uint32_t>(ws.f_src) + f0, ptr<uint32_t>(ws.f_dst) + f0, nullptr,
                ptr<unsigned long long>(ws.f_uid) + f0, 0ull, F_dev, n, kDomainDecr, f0};
    unsigned long long *own = ptr<unsigned long long>(ws.keys);
    RecoverArgs a{};
    a.G = G->g;
    a.H = H->g;
    a.A.s[0] = append_side(H, ptr<uint32_t>(ws.cand_x), ptr<uint32_t>(ws.cand_y), ptr<float>(ws.cand_w));
    a.A.n = 1;
    a.job = job;
    a.resume = phase0 == 1;
    a.keys = keys_given ? const_cast<unsigned long long *>(keys_given) : own;
    a.clear_keys = !keys_given;
    if (!replay) a.rec = scratch.rec;
    a.plen = ptr<int32_t>(ws.path_len);
    a.pv = ptr<uint32_t>(ws.path_v);
    a.ps = ptr<uint32_t>(ws.path_s);
    a.stride = stride;
    a.hw = hwk;
    a.f_idx = ptr<uint32_t>(ws.f_idx) + f0;
    a.key = make_uint2((uint32_t)p.seed, (uint32_t)(p.seed >> 32));
    a.status = status;
    a.cond = cond;
    a.cx = ptr<uint32_t>(ws.cand_x);
    a.cy = ptr<uint32_t>(ws.cand_y);
    a.cw = ptr<float>(ws.cand_w);
    a.tk = ptr<unsigned long long>(ws.htab_k);
    a.tv = ptr<uint32_t>(ws.htab_v);
    a.keep = ptr<uint32_t>(ws.keep);
    a.rx = ptr<uint32_t>(ws.rx2);
    a.ry = ptr<uint32_t>(ws.ry2);
    a.rk = ptr<uint8_t>(ws.rk2);
    a.blk = ptr<uint32_t>(ws.blk);
    a.counts = ptr<uint32_t>(ws.counts);
    a.sc = sc;
    a.halt = halt;
    a.code_records = halt_code(batch, (uint32_t)kHaltRecords, 1);
    a.code_arena = halt_code(batch, (uint32_t)kHaltArena, 1);
    a.code_paths = halt_code(batch, (uint32_t)kHaltPaths, 2);
    if (phase0 != 1) {
        // walks on the updated G (main.cu:392, 420)
        RowIndex ix{};   // of the walks, and of the replays of their winners
        DYG_TRY(index_enqueue(G, n, p, false, halt, scratch, &ix, st));
        if (!keys_given) {
            if (!walk_ready) DYG_CUDA(cudaMemsetAsync(own, 0, sizeof(unsigned long long) * n, st));
            DYG_TRY(launch_walk(G, job, p, false, own, ix, st, walk_ready, replay ? nullptr : &scratch.rec));
        }
        if (replay)
            DYG_TRY(launch_winner_paths(G, job, p, a.keys, n, stride, ptr<uint32_t>(ws.path_v),
                                    ptr<uint32_t>(ws.path_s), ptr<int32_t>(ws.path_len), ix, st));
    }
    // blocks for what a batch usually brings: a few candidates per deletion
    return launch_phases<k_recover>(op_blocks(4ull * n, H->long_rows), st, grid_bar(G, halt), a);
}

// Decremental batch `batch` of the standalone updater: deletion stage, then
// walks over the batch's whole walk list.
static dyg_status decr_enqueue(dyg_graph *G, dyg_graph *H, const uint32_t *src, const uint32_t *dst,
                               uint32_t n, uint64_t uid0, const unsigned long long *uids,
                               const dyg_walk_params &p, WalkScratch &scratch,
                               unsigned long long *halt, uint32_t batch, uint32_t phase0,
                               int32_t *status, float *cond, cudaStream_t st) {
    if (phase0 == 0)
        DYG_TRY(decr_delete_enqueue(G, H, src, dst, n, uid0, uids, false, halt, status, cond, st));
    return decr_walk_enqueue(G, H, 0, n, ptr<uint32_t>(G->ws.counts) + C_FILTERED, p, halt, batch,
                             phase0, status, cond, st, true, scratch);
}

// --------------------------------------------------------- stream drivers

namespace {

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

}  // namespace

dyg_status incremental_run(dyg_graph *H, dyg_graph *G, const uint32_t *src, const uint32_t *dst,
                           const float *w, uint32_t n, uint32_t B, uint64_t uid_base,
                           const unsigned long long *uids, const dyg_walk_params &p, int32_t *found, float *cond, uint8_t *acc,
                           cudaStream_t st, bool check_inputs,
                           const std::function<void()> *during,
                           const std::function<dyg_status()> *fetch) {
    unsigned long long *sc = ptr<unsigned long long>(H->ws.scalars);
    unsigned long long *halt = sc + S_HALT;
    DYG_TRY(check_usable(H, G));
    DYG_TRY(clear_halt(H, st));
    if (check_inputs) DYG_TRY(validate_enqueue(halt, sc + S_ERR, src, dst, w, n, H->g.n, st));
    // no batch is larger than the first, so the keys it clears are clear for
    // the later ones
    const uint32_t b_max = B < n ? B : n;
    DYG_TRY(ensure(H->ws.keys, sizeof(unsigned long long) * b_max));
    DYG_TRY(rowops_ensure(H, 2ull * b_max, st));
    if (G) DYG_TRY(rowops_ensure(G, 2ull * b_max, st));
    WalkScratch scratch(st);
    uint32_t b_start = 0;
    for (int round = 0; round < 64; ++round) {
        for (uint32_t b = b_start; (uint64_t)b * B < n; ++b) {
            const uint32_t b0 = b * B, nb = (n - b0 < B) ? n - b0 : B;
            DYG_TRY(incr_enqueue(H, G, src + b0, dst + b0, w + b0, nb, uid_base + b0,
                                 uids ? uids + b0 : nullptr, p, halt, b,
                                 found ? found + b0 : nullptr, cond ? cond + b0 : nullptr,
                                 acc ? acc + b0 : nullptr, st, b > b_start, scratch));
        }
        if (during && round == 0) (*during)();
        if (fetch) DYG_TRY((*fetch)());
        DYG_TRY(read_scalars2(H, G, st));
        const unsigned long long h = H->ws.host_scalars[S_HALT];
        if (!h) return DYG_OK;
        const HaltInfo hi = decode_halt(h);
        if (hi.kind == kHaltInvalid) return rejected_inputs(H, st);
        for (dyg_graph *X : {H, G})
            if (X) DYG_TRY(scratch.with_room([&] { return grow_arena(X, X->g.arena_cap * 2, st); }));
        DYG_TRY(clear_halt(H, st));
        b_start = hi.batch;   // nothing of the halted batch changed: redo it whole
    }
    set_error("incremental stream: too many arena regrowths");
    return DYG_ENOMEM;
}

dyg_status decremental_run(dyg_graph *G, dyg_graph *H, const uint32_t *src, const uint32_t *dst,
                           uint32_t n, uint32_t B, uint64_t uid_base,
                           const unsigned long long *uids, const dyg_walk_params &p,
                           int32_t *status, float *cond, uint64_t *n_rec, cudaStream_t st,
                           bool check_inputs, const std::function<void()> *during,
                           const std::function<dyg_status()> *fetch) {
    Workspace &ws = G->ws;
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    unsigned long long *halt = sc + S_HALT;
    DYG_TRY(check_usable(G, H));
    // record buffers: start at 4 per deletion, grown on demand (halt + resume)
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
    if (check_inputs) DYG_TRY(validate_enqueue(halt, sc + S_ERR, src, dst, nullptr, n, G->g.n, st));
    const uint32_t b_max = B < n ? B : n;
    DYG_TRY(decr_delete_ensure(G, H, b_max, st));
    DYG_TRY(decr_walk_ensure(G, H, b_max, p, st));
    WalkScratch scratch(st);
    scratch.open_paths(G, b_max, p);
    uint32_t b_start = 0, ph_start = 0;
    for (int round = 0; round < 64; ++round) {
        for (uint32_t b = b_start; (uint64_t)b * B < n; ++b) {
            const uint32_t b0 = b * B, nb = (n - b0 < B) ? n - b0 : B;
            DYG_TRY(decr_enqueue(G, H, src + b0, dst + b0, nb, uid_base + b0,
                                 uids ? uids + b0 : nullptr, p, scratch, halt, b,
                                 b == b_start ? ph_start : 0, status + b0, cond + b0, st));
        }
        if (during && round == 0) (*during)();
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
        b_start = hi.batch;
        ph_start = hi.phase;   // deletions and walks of this batch are done: resume there
    }
    set_error("decremental stream: too many buffer regrowths");
    return DYG_ENOMEM;
}

}  // namespace dyg
