// dyg_internal.cuh -- device data layout, Philox stream and shared helpers of
// the B200 dyGRASS update path.
//
// HBM layout of one graph (a dynamic CSR with per-row slack):
//   desc[v]   uint2 {offset, degree}: one 8-byte load gives a walker both the
//             row start and its live length.
//   cap[v]    u32 row capacity (slots reserved at `offset`), touched only by
//             commits and compaction, never by walkers.
//   slots[i]  uint2 {column, bits of 1/weight}: the neighbour id and the
//             resistance a walker adds arrive in one 8-byte load (the
//             reference stores them degree floats apart through a pointer
//             table, gpu_graph.cuh:205-235).  1/w is the correctly rounded
//             float reciprocal, so R += 1/w is bit-identical to dividing on
//             every move.
//   wts[i]    f32 weight of slot i (same offsets as slots); read by exports,
//             recovered edges and the weight-proportional mode, never by the
//             uniform walk.
//   top       arena bump pointer; rows that outgrow their capacity move to
//             [top, top + new_cap) and leave a hole reclaimed by compaction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <string>
#include <vector>

#include "../../include/dyg.h"

namespace dyg {

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr uint32_t kDomainIncr = 0u;   // incremental walks
constexpr uint32_t kDomainDecr = 1u;   // decremental walks
constexpr uint32_t kDomainHeur = 2u;   // 2-step fallback walks

// Device error bits (sticky per workspace until read).
constexpr uint32_t kErrVertex = 1u;    // vertex id >= n in a batch
constexpr uint32_t kErrPath = 2u;      // winner re-walk disagreed with its key
constexpr uint32_t kErrArena = 4u;     // arena overflow in a commit
constexpr uint32_t kErrWeight = 8u;    // weight not finite and > 0 in a batch
constexpr uint32_t kErrScan = 16u;     // a scan tile gave up waiting for its predecessor
constexpr uint32_t kErrBarrier = 32u;  // a block gave up waiting at a grid barrier

struct DevGraph {
    uint2 *desc;
    uint32_t *cap;
    uint2 *slots;
    float *wts;
    unsigned long long *top;   // device scalar
    uint64_t arena_cap;        // slots
    uint32_t n;
};

// ------------------------------------------------------------------ Philox
// Philox4x32-10 (Salmon et al., SC'11).  Counter = {draw block, walker,
// update id low, update id high | domain << 24}, key = seed.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

__device__ __forceinline__ uint32_t pick4(uint4 v, uint32_t i) {
    return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

__host__ __device__ __forceinline__ uint32_t ctr3_of(uint64_t uid, uint32_t domain) {
    return ((uint32_t)(uid >> 32) & 0x00FFFFFFu) | (domain << 24);
}

// Winner key: max conductance 1/R, then lowest walker id; the low bits carry
// the winner's step count.  0 means no walker reached the target.
__device__ __forceinline__ unsigned long long pack_key(float cond, uint32_t walker,
                                                       uint32_t found) {
    return ((unsigned long long)__float_as_uint(cond) << 32) |
           ((unsigned long long)(1023u - walker) << 22) |
           (unsigned long long)(found & 0x3FFFFFu);
}
__host__ __device__ __forceinline__ uint32_t key_walker(unsigned long long k) {
    return 1023u - (uint32_t)((k >> 22) & 0x3FFu);
}
__host__ __device__ __forceinline__ int32_t key_found(unsigned long long k) {
    return k ? (int32_t)(k & 0x3FFFFFu) : -1;
}

// Fixed-point weight of the weight-proportional mode (exact w * 2^32,
// truncated) so that prefix sums are associative and match the host: the
// 24-bit significand m shifted by the exponent.  w = m * 2^(ex - 150), so
// w * 2^32 = (m * 2^40) >> (158 - ex); m * 2^40 has an empty low word.
// Weights are not negative; from 2^32 on (infinity included) the value is all
// ones, and below 2^-32 (0 included) the shift leaves nothing.
__device__ __forceinline__ unsigned long long wq(float w) {
    const uint32_t b = __float_as_uint(w), ex = b >> 23;
    const unsigned long long top = (unsigned long long)((b << 8) | 0x80000000u) << 32;
    unsigned long long q;
    asm("shr.u64 %0, %1, %2;" : "=l"(q) : "l"(top), "r"(158u - ex));   // shifts of 64 and more give 0
    return ex >= 159u ? 0xFFFFFFFFFFFFFFFFull : q;
}
__device__ __forceinline__ unsigned long long mul_hi32(uint32_t r, unsigned long long total) {
    // floor(r * total / 2^32) for a 96-bit product
    const unsigned long long lo = (unsigned long long)r * (total & 0xFFFFFFFFull);
    const unsigned long long hi = (unsigned long long)r * (total >> 32);
    return hi + (lo >> 32);
}

// ------------------------------------------------------------- long rows
// Rows longer than kBigRow are scanned and moved by a whole block instead of
// one thread, lane group or warp: on power-law graphs a hub row holds tens of
// thousands of slots, and a serial scan of it would bound the whole launch.
// kBigThreads: threads of the stream files' search blocks.
constexpr uint32_t kBigRow = 256;
constexpr uint32_t kBigThreads = 256;

// First j < deg with slots[off + j].x == y, or ~0u.  Every thread of the block
// calls it; s_best is one shared word.  Tiles of kFindUnroll * blockDim.x
// slots whose loads are all issued before any compare, so a hub row costs a
// few dependent round trips instead of one per 4 * blockDim.x slots, and a
// match ends the scan at the end of its tile.
constexpr uint32_t kFindUnroll = 16;
__device__ __forceinline__ uint32_t block_find(const uint2 *slots, uint32_t off, uint32_t deg,
                                               uint32_t y, uint32_t *s_best) {
    const uint32_t *cols = reinterpret_cast<const uint32_t *>(slots + off);
    for (uint32_t base = 0; base < deg; base += kFindUnroll * blockDim.x) {
        if (threadIdx.x == 0) *s_best = ~0u;
        __syncthreads();
        uint32_t v[kFindUnroll];
#pragma unroll
        for (uint32_t u = 0; u < kFindUnroll; ++u) {
            const uint32_t j = base + u * blockDim.x + threadIdx.x;
            v[u] = j < deg ? cols[2u * j] : ~0u;   // vertex ids are never ~0u
        }
#pragma unroll
        for (uint32_t u = 0; u < kFindUnroll; ++u)
            if (v[u] == y) {   // this thread's first match is its smallest j
                atomicMin(s_best, base + u * blockDim.x + threadIdx.x);
                break;
            }
        __syncthreads();
        const uint32_t b = *s_best;
        __syncthreads();   // every thread has read it before the next reset
        if (b != ~0u) return b;
    }
    return ~0u;
}

// ------------------------------------------------------------- workspace
// Lookup index of a graph's long rows for the weight-proportional walks (k_index,
// walk.cu), rebuilt for every launch: rbase[v] is the word offset of row v's
// region in `words`, 0 for a row without one.  A region is a hash table of
// 2^k >= 2 deg words (position + 1 of a column, 0 empty) and the row's deg
// inclusive prefix sums of wq (two words each).
struct RowIndex {
    const uint32_t *rbase;   // null: no row has an index
    const uint32_t *words;
};

struct Buf {
    void *p = nullptr;
    size_t bytes = 0;
};

// Paths of decremental walkers, kept while they walk.  Every thread of the
// walk keeps the slots its walker took in `hist` (move j of thread t at word
// j * threads + t, or four moves to a uint4 there); a walker that improves its
// edge's best copies its path to `words` as a record {previous record of the
// edge + 1, key (two words), slots...} and puts it on the edge's list.  The
// winner's record is the one with the winner's key.
struct PathRec {
    uint32_t *heads;              // per walk-list entry: last record + 1 (0: none); null: not kept
    uint32_t *words;
    uint32_t cap;                 // words
    unsigned long long *cursor;   // words asked for (S_RECW)
    uint32_t *hist;
    uint32_t threads;             // most threads a walk may have
};

// Device scratch owned by a graph handle, grown on demand.
struct Workspace {
    Buf keys;                                 // u64 per edge
    Buf flags, pos;                           // u32 per edge / per vertex (compaction)
    Buf f_src, f_dst, f_idx;                  // walk list (filtered deletions / new insertions)
    Buf f_uid;                                // u64 per walk-list entry
    Buf f_w;                                  // f32 per walk-list entry (insertions)
    Buf found;                                // u8 per half-edge
    Buf path_v, path_s;                       // replayed winner paths: vertices, taken slots
    Buf path_len;                             // i32 per filtered edge
    Buf rec_head;                             // path records of the walks: last of each edge
    uint32_t rec_each = 48;                   // words to begin with for each edge: as a call came to need
    Buf cand_x, cand_y, cand_w;               // recovery candidates
    Buf keep;                                 // u32 per candidate
    Buf htab_k, htab_v;                       // dedup hash table
    Buf scan_status;                          // u64 per tile of the single-pass scan
    unsigned long long scan_tickets = 0;      // tile tickets handed out so far (S_SCAN)
    uint32_t scan_epoch = 0;                  // tags this workspace's scan statuses per call
    Buf s_src, s_dst, s_w, s_o1, s_o2, s_o3;  // whole-stream staging
    Buf rx2, ry2;                             // recovered edges of a whole stream
    Buf rk2;
    Buf nxt, runs;                            // row operations: per-entry chain link / ordered entries
    Buf rowcnt, rowhead;                      // row operations: per-row entries / last entry + 1
    Buf rowlist;                              // row operations: rows for warps and blocks
    Buf blk;                                  // row operations: per-block words
    Buf st_key, st_cnt;                       // stream file: table of (min, max) keys; counts, heads
    Buf st_val;                               // stream file: chain links and table slots of the edges
    Buf st_pos;                               // stream file: uint4 slot positions in G and H
    Buf st_wapp;                              // stream file: G weight of each new edge
    Buf big;                                  // stream file: uint4 per long-row search
    Buf s_uid;                                // staged per-edge update ids
    Buf scalars;                              // u64 scalars (see Scalar)
    Buf counts;                               // u32 counts (see Count), behind the scalars
    unsigned long long *host_scalars = nullptr;   // pinned mirror of scalars and counts
    uint32_t *host_counts = nullptr;
    Buf io_in, io_out;                        // a call's host arrays, packed
    Buf pin_in, pin_out;                      // pinned host memory beside them
};

// Indices into Workspace::scalars (u64, device) and Workspace::counts (u32).
enum Scalar : int {
    S_NEED = 0,       // arena slots a pending append needs (zero between appends)
    S_CURSOR = 1,     // arena cursor of the moves of that append
    S_KEPT = 2,       // recovery candidates kept so far (zero between recoveries)
    S_NBIG = 3,       // stream file: entries on the long-row list
    S_RUNS = 4,       // row operations: next free word of the runs (low word), runs to fill (high word)
    S_ERR = 5,        // device error bits (kErr*)
    S_MOVES = 6,      // walker moves (accumulating)
    S_WALKS = 7,      // walks finished (accumulating)
    S_TOP = 8,        // arena bump pointer of the owning graph
    S_WORK = 9,       // work-chunk counter of the persistent walk kernel
    S_HALT = 10,      // halt code of a stream this handle drives (0 = running)
    S_RECCNT = 11,    // recovered edges recorded so far in a decremental stream
    S_RECCAP = 12,    // capacity of the record buffers (follows S_RECCNT)
    S_LONG = 13,      // set by an append that made a row longer than kBigRow
    S_SCAN = 14,      // tile tickets of the single-pass scan (accumulating)
    S_BAR = 15,       // grid barrier: arrivals (low word), generation (high word)
    S_IDX = 16,       // row index: next free word
    S_IDXN = 17,      // row index: rows for a warp (low word), for a block (high word)
    S_IDXSUM = 18,    // row index: slots of rows a lane can search (low word), of longer ones (high word)
    S_SLOTS = 19,     // live slots, summed for dyg_graph_info
    S_RECW = 20,      // path records: words asked for (zero between walks)
    S_RECNEED = 21,   // path records: words a halted walk asked for
    S_ITEMS = 22,     // row operations: rows for a block (low word), for a warp (high word)
    S_FOLD = 23,      // stream file: words of the often repeated edges' runs (low word), such edges (high word)
    S_NSCALARS = 24
};
enum Count : int {
    C_FILTERED = 0,   // decremental: edges to walk
    C_CANDS = 1,      // path candidates of a recovery (fallback candidates follow)
    C_CANDS_ALL = 2,  // all candidates of a recovery
    C_WALKLIST = 3,   // stream file: new insertions to walk
    C_NCOUNTS = 4
};

constexpr size_t kScalarBytes = sizeof(unsigned long long) * S_NSCALARS + sizeof(uint32_t) * C_NCOUNTS;

// Halt codes: (batch + 1) << 8 | kind << 4 | phase.
constexpr unsigned long long kHaltArena = 1;    // an arena reservation did not fit
constexpr unsigned long long kHaltRecords = 2;  // the recovered-edge buffers are full
constexpr unsigned long long kHaltInvalid = 3;  // a device-resident batch failed its input check
constexpr unsigned long long kHaltPaths = 4;    // the path records did not fit (the walks are repeated)
constexpr unsigned long long kHaltBroken = 5;   // a block gave up at a grid barrier (nothing resumes)
__host__ __device__ __forceinline__ unsigned long long halt_code(uint32_t batch, uint32_t kind,
                                                                 uint32_t phase) {
    return ((unsigned long long)(batch + 1) << 8) | (kind << 4) | phase;
}

// Reads of a grid barrier's word before a block gives up: a phase may rightly
// last a while (a block rewriting hub rows), so about a minute.
constexpr uint32_t kBarSpinLimit = 1u << 26;

}  // namespace dyg

struct dyg_graph {
    int device = 0;
    dyg::DevGraph g{};
    uint32_t slack = 2;
    double headroom = 0.5;
    dyg::Workspace ws;
    uint64_t moves_total = 0, walks_total = 0;
    // Recovered edges recorded by the last decremental call on this handle
    // (as G); they stay in ws.rx2 / ry2 / rk2 until the next such call.
    uint64_t last_rec = 0;
    // The graph has (or may have) a row longer than kBigRow: row operations
    // then spread their entries over every SM, and stream files search such
    // rows with whole blocks (the results do not depend on it).
    bool long_rows = false;
    // A launch that updated the graph was cut short (kErrBarrier): its rows may
    // hold part of a batch.  Updates are refused until a whole graph is copied
    // over it.
    bool broken = false;
    bool counted = false;   // among its device's handles
    uint32_t bar_limit = dyg::kBarSpinLimit;   // GridBar::limit
};

namespace dyg {

void set_error(const std::string &msg);
dyg_status cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define DYG_CUDA(call)                                                          \
    do {                                                                        \
        cudaError_t _e = (call);                                                \
        if (_e != cudaSuccess) return ::dyg::cuda_fail(_e, #call, __FILE__, __LINE__); \
    } while (0)

#define DYG_TRY(call)                      \
    do {                                   \
        dyg_status _s = (call);            \
        if (_s != DYG_OK) return _s;       \
    } while (0)

// --- memory.cu
// Device memory from the current device's pool.  dev_free: the device has
// finished with the block (or the caller has synchronized it).
cudaError_t dev_alloc(void **out, size_t bytes);
void dev_free(void *p);
// Scratch that a call can do without: a kept block of the device if one is free
// and large enough, else a new one; returned once the device has finished with
// it.  A device keeps at most 3 GB of it, 256 MB once it has no handles
// (scratch_handles counts them; the device is current).  scratch_drop frees
// what is kept; an allocation that does not fit otherwise does so first.
struct Buf;
cudaError_t scratch_borrow(Buf *b, size_t bytes);
void scratch_return(Buf *b);
void scratch_drop();
void scratch_handles(int dev, int change);
// For tests: this thread's next `pass` allocations go through, the `fail` after
// them do not.
void fail_allocations(uint32_t pass, uint32_t fail);
// Pinned host memory; host_free takes the size given to host_alloc, once the
// device has finished with the block.
cudaError_t host_alloc(void **out, size_t bytes);
void host_free(void *p, size_t bytes);
template <typename T>
inline cudaError_t dev_alloc(T **out, size_t bytes) { return dev_alloc(reinterpret_cast<void **>(out), bytes); }
// Unique id of the context current on this thread (cuCtxGetId, reached through
// the runtime's driver entry points, so no libcuda link is needed); 0 when the
// driver does not provide it.
unsigned long long current_context_id();

dyg_status ensure(Buf &b, size_t bytes);
// Where a caller's pointer lives as seen from `device`: host memory (pageable
// or pinned), device memory this device's kernels may read (its own, or
// managed), or device memory of another GPU, which a kernel on `device`
// must not be given.
enum PtrPlace : int { kOnHost = 0, kOnDevice = 1, kOnOtherDevice = 2 };
PtrPlace ptr_place(const void *p, int device);
// DYG_EINVAL (with the argument's name in the message) if any non-null
// pointer of `ptrs` is device memory of another GPU than `device`.
dyg_status check_same_device(int device, const void *const *ptrs, const char *const *names,
                             int count);
template <typename T>
inline T *ptr(const Buf &b) { return static_cast<T *>(b.p); }

int num_sms();
// Counts launches of this library's kernels.
void count_launch();

// --- walk.cu
struct WalkJob {
    const unsigned long long *halt;  // kernels return at once when *halt != 0 (may be null)
    const uint32_t *src, *dst;
    const float *w;              // incremental: per-edge weight; else null
    const unsigned long long *uid;   // per-edge update id, or null -> uid0 + e
    unsigned long long uid0;
    const uint32_t *n_dev;       // device count of the whole list, or null -> n_host edges
    uint32_t n_host;             // edges of this range at most
    uint32_t domain;
    uint32_t f0;                 // this range's first entry in the list n_dev counts
};
// Edges of a job: those of [f0, f0 + n_host) the list has.
__device__ __forceinline__ uint32_t job_count(const WalkJob &j) {
    if (!j.n_dev) return j.n_host;
    const uint32_t n = *j.n_dev;
    return n > j.f0 ? min(n - j.f0, j.n_host) : 0u;
}
// counter_zero: the kernel's chunk counter is known to be zero (the commit
// of the batch before reset it), so no memset precedes the launch.
dyg_status launch_walk(dyg_graph *G, const WalkJob &job, const dyg_walk_params &p, bool incremental,
                       unsigned long long *keys, const RowIndex &ix, cudaStream_t st,
                       bool counter_zero = false, const PathRec *rec = nullptr);
// Threads of a walk over up to n edges (the most a later launch takes unless
// the tuning changes; a launch given fewer takes fewer).
uint32_t walk_threads(uint32_t n, const dyg_walk_params &p);
dyg_status launch_walk_scalars(const DevGraph &g, const WalkJob &job, const dyg_walk_params &p,
                               bool incremental, unsigned long long *keys,
                               unsigned long long *scalars, cudaStream_t st);
// The row index for weighted walks from up to n edges on G as it is now; empty
// for a uniform transition or a graph without hub rows.  The walks that use it
// test the same halt word: an index whose launch was cut short must not be read.
struct WalkScratch;
dyg_status index_enqueue(dyg_graph *G, uint32_t n, const dyg_walk_params &p, bool incremental,
                         unsigned long long *halt, WalkScratch &scratch, RowIndex *out, cudaStream_t st);
dyg_status launch_winner_paths(dyg_graph *G, const WalkJob &job, const dyg_walk_params &p,
                               const unsigned long long *keys, uint32_t n_max, uint32_t path_stride,
                               uint32_t *path_v, uint32_t *path_s, int32_t *path_len, const RowIndex &ix,
                               cudaStream_t st);
// --- capi.cu
// After a run: DYG_OK, or the error the kernels flagged in G's scalars (last
// read by the run), which are cleared.
dyg_status device_errors(dyg_graph *G, cudaStream_t st);
// DYG_OK, or DYG_EINVAL with the message set, for walk parameters.
dyg_status check_walk_params(const dyg_walk_params *p);

// --- pipeline.cu
// Checks a device-resident batch before anything else of the call runs: an
// endpoint >= nv (kErrVertex) or a weight that is not finite and > 0
// (kErrWeight, when w is given) sets the error bits and the halt code
// kHaltInvalid, so every later kernel of the call returns at once and the
// graphs stay exactly as they were.
dyg_status validate_enqueue(unsigned long long *halt, unsigned long long *err,
                            const uint32_t *src, const uint32_t *dst, const float *w, uint32_t n,
                            uint32_t nv, cudaStream_t st);
// After a run halted with kHaltInvalid: clears the halt and the error bits of
// D (the handle whose scalars held them) and returns DYG_EINVAL with the
// failed check as the message.
dyg_status rejected_inputs(dyg_graph *D, cudaStream_t st);
// uids (device, may be null): per-edge update ids instead of uid_base + e.
// `during`, if given, runs on the host once the first pass of batches is
// enqueued and before the call waits for them: host work that overlaps the
// device work.  `fetch`, if given, runs before every wait and enqueues copies
// of the results, so that the last wait covers them.
dyg_status incremental_run(dyg_graph *H, dyg_graph *G, const uint32_t *src, const uint32_t *dst,
                           const float *w, uint32_t n, uint32_t B, uint64_t uid_base,
                           const unsigned long long *uids, const dyg_walk_params &p, int32_t *found, float *cond, uint8_t *acc,
                           cudaStream_t st, bool check_inputs = false,
                           const std::function<void()> *during = nullptr,
                           const std::function<dyg_status()> *fetch = nullptr);
dyg_status decremental_run(dyg_graph *G, dyg_graph *H, const uint32_t *src, const uint32_t *dst,
                           uint32_t n, uint32_t B, uint64_t uid_base,
                           const unsigned long long *uids, const dyg_walk_params &p,
                           int32_t *status, float *cond, uint64_t *n_rec, cudaStream_t st,
                           bool check_inputs = false,
                           const std::function<void()> *during = nullptr,
                           const std::function<dyg_status()> *fetch = nullptr);

struct WalkScratch;
// The buffers that the deletion stage of n edges and the walks and recoveries
// of n walked ones cannot do without.
dyg_status decr_delete_ensure(dyg_graph *G, dyg_graph *H, uint32_t n, cudaStream_t st);
dyg_status decr_walk_ensure(dyg_graph *G, dyg_graph *H, uint32_t n, const dyg_walk_params &p, cudaStream_t st);
dyg_status decr_delete_enqueue(dyg_graph *G, dyg_graph *H, const uint32_t *src,
                               const uint32_t *dst, uint32_t n, uint64_t uid0,
                               const unsigned long long *uids, bool file_orient,
                               unsigned long long *halt, int32_t *status, float *cond,
                               cudaStream_t st);
// keys_given (device, may be null): the walk list's winner keys, computed
// elsewhere (a sharded batch); the walks are then skipped.  walk_ready: the
// handle's own keys and chunk counter are zero (the launch before left them so).
dyg_status decr_walk_enqueue(dyg_graph *G, dyg_graph *H, uint32_t f0, uint32_t nf,
                             const uint32_t *F_dev, const dyg_walk_params &p,
                             unsigned long long *halt, uint32_t batch, uint32_t phase0,
                             int32_t *status, float *cond, cudaStream_t st, bool walk_ready,
                             WalkScratch &scratch, const unsigned long long *keys_given = nullptr);
// Path records are kept for walks of up to kPathSteps steps and for up to
// kPathWalkers uniform ones.  Replays last as long as one longest path whatever the
// batch; keeping paths costs the uniform walk nothing while it is bound by the
// latency of its longest walks, and a sixth of its time once it is bound by
// throughput: 1,013 deletions of a 37 x 41 x 29 mesh (160 walkers) take 57 us
// of walks and 41 of replays against 55 and 0, 29,700 deletions of a 100^3
// mesh (512 walkers) 230 and 22 against 267 and 0.  A weighted move costs so
// much that keeping its slot is nothing.
constexpr uint32_t kPathSteps = 256;
constexpr uint64_t kPathWalkers = 2u << 20;
// What the walks of one call borrow and can do without: path records (else
// winners are replayed) and the row index (else the warp searches the rows).
// Asked for after what the call needs; given back when the call ends, or
// earlier if something that it needs does not fit otherwise.
struct WalkScratch {
    cudaStream_t st;
    PathRec rec{};      // heads null: replay
    Buf hist, words;
    uint32_t edges = 0;   // that records were opened for
    Buf index;
    bool index_tried = false;
    explicit WalkScratch(cudaStream_t stream) : st(stream) {}
    WalkScratch(const WalkScratch &) = delete;
    WalkScratch &operator=(const WalkScratch &) = delete;
    ~WalkScratch() { release(); }
    // Records for calls of up to n walked deletions.
    void open_paths(dyg_graph *G, uint32_t n, const dyg_walk_params &p);
    // After a kHaltPaths halt (scalars just read): room for what was asked for.
    void grow_paths(dyg_graph *G);
    // Waits for the stream and gives everything back; false: there was nothing.
    bool release();
    // Runs f, and once more without the scratch if memory was short.
    template <class F>
    dyg_status with_room(F f) {
        dyg_status rc = f();
        if (rc != DYG_ENOMEM || !release()) return rc;
        scratch_drop();
        set_error("");
        return f();
    }
};
// The commit reads keys; clear_keys zeroes them behind it for the next walk.
dyg_status incr_commit_enqueue(dyg_graph *H, dyg_graph *G, const uint32_t *src,
                               const uint32_t *dst, const float *w, uint32_t n,
                               unsigned long long *keys, bool clear_keys,
                               unsigned long long *halt, uint32_t batch, int32_t *found,
                               float *cond, uint8_t *acc, cudaStream_t st);
// Grows b to `bytes`, keeping its first `used` bytes.
dyg_status grow_keep(Buf &b, size_t bytes, size_t used, cudaStream_t st);

// --- stream.cu
uint32_t stream_default_chunk(uint32_t n_vertices);
dyg_status stream_file_run(dyg_graph *G, dyg_graph *H, uint32_t op, const uint32_t *src,
                           const uint32_t *dst, const float *w, uint32_t n, uint64_t uid0,
                           uint32_t chunk, const dyg_walk_params &p, int32_t *status, float *cond,
                           uint64_t *n_rec, cudaStream_t st, bool check_inputs = false,
                           const std::function<dyg_status()> *fetch = nullptr);

// --- graph.cu
dyg_status upload_graph(dyg_graph *G, uint32_t n, const uint64_t *row_ptr, const uint32_t *col,
                        const float *w);
// The graph of an edge list (host arrays) with rows in list order, built on
// the device; *bad is set, and nothing else happens, if an id or a weight is
// not valid.
dyg_status build_graph(dyg_graph *G, uint32_t n, uint64_t m, const uint32_t *src, const uint32_t *dst,
                       const float *w, bool *bad);
// Rows as a CSR into host arrays (col, w may be null); at most slot_cap slots
// are copied.
dyg_status export_graph(dyg_graph *G, uint64_t *row_ptr, uint32_t *col, float *w, uint64_t slot_cap);
// Sums the degrees into S_SLOTS.
dyg_status count_slots_enqueue(dyg_graph *G, cudaStream_t st);
// Copies both graphs' scalars and counts to the host with one synchronize.
// DYG_ESTATE if a launch on either was cut short at a grid barrier: both are
// then marked broken, their workspaces as new.
dyg_status read_scalars2(dyg_graph *A, dyg_graph *B, cudaStream_t st);
// DYG_ESTATE for a broken graph (B may be null).
dyg_status check_usable(const dyg_graph *A, const dyg_graph *B);
// Exclusive scan of in[0, m) into out.
dyg_status exclusive_scan_u32(Workspace &ws, const uint32_t *in, uint32_t *out, uint32_t m,
                              cudaStream_t st);
dyg_status compact_graph(dyg_graph *G, cudaStream_t st);
// src's rows, capacities and arena top into dst, whose arena holds them.
dyg_status copy_graph_enqueue(dyg_graph *dst, const dyg_graph *src, cudaStream_t st);
dyg_status grow_arena(dyg_graph *G, uint64_t min_cap, cudaStream_t st);
dyg_status read_scalars(dyg_graph *G, cudaStream_t st);
// Rows of local graph [v0, v0 + n) of a pool graph: load places them at the
// arena top (compacting, then growing, when they do not fit) with columns
// shifted by v0 and sets the range's descriptors; save copies them back
// (columns local again, row order kept); clear empties the range (its old
// slots become a hole that compaction reclaims).  load and save synchronize.
dyg_status load_range(dyg_graph *G, uint32_t v0, uint32_t n, const uint64_t *row_ptr,
                      const uint32_t *col, const float *w, cudaStream_t st);
dyg_status save_range(dyg_graph *G, uint32_t v0, uint32_t n, std::vector<uint64_t> &row_ptr,
                      std::vector<uint32_t> &col, std::vector<float> &w, cudaStream_t st);
dyg_status clear_range(dyg_graph *G, uint32_t v0, uint32_t n, cudaStream_t st);
// A graph of n vertices with no slots and an arena of arena_slots (a pool).
dyg_status create_empty_graph(uint32_t n, uint64_t arena_slots, int device, uint32_t slack,
                              double headroom, dyg_graph **out);
void destroy_graph(dyg_graph *G);

}  // namespace dyg
