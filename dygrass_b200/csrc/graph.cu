// graph.cu -- device-resident dynamic CSR: upload, arena growth, compaction
// and the small shared helpers (allocation, scans, scalar read-back).  Row
// updates live in rowops.cuh.  Row moves (capacity exceeded) take space from a
// bump arena: offsets differ from run to run but contents never do.

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "dyg_internal.cuh"
#include "scan.cuh"

namespace dyg {

static std::atomic<unsigned long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int num_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms < 1) sms = 1;
    }
    return sms;
}

dyg_status ensure(Buf &b, size_t bytes) {
    if (bytes == 0) bytes = 16;
    if (b.bytes >= bytes) return DYG_OK;
    if (b.p) {
        DYG_CUDA(cudaDeviceSynchronize());   // launches before may still use it
        dev_free(b.p);
        b.p = nullptr;
        b.bytes = 0;
    }
    size_t want = bytes + bytes / 4;
    want = (want + 255) & ~(size_t)255;
    cudaError_t e = dev_alloc(&b.p, want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
        set_error(std::string("allocation of ") + std::to_string(want) + " bytes failed: " +
                  cudaGetErrorString(e));
        return DYG_ENOMEM;
    }
    b.bytes = want;
    return DYG_OK;
}

// The workspace of a graph whose update was cut short: what the operations
// expect to find as the one before left it (chains, hash tables, counters) is
// made as new.
static dyg_status recover_workspace(dyg_graph *G) {
    Workspace &ws = G->ws;
    DYG_CUDA(cudaDeviceSynchronize());
    for (Buf *b : {&ws.rowcnt, &ws.rowhead, &ws.htab_k, &ws.htab_v, &ws.st_key, &ws.st_cnt}) {
        dev_free(b->p);
        *b = Buf{};
    }
    for (int s : {S_NEED, S_CURSOR, S_KEPT, S_NBIG, S_RUNS, S_ERR, S_WORK, S_HALT, S_BAR, S_RECW, S_ITEMS, S_FOLD}) {
        DYG_CUDA(cudaMemset(ptr<unsigned long long>(ws.scalars) + s, 0, sizeof(unsigned long long)));
        ws.host_scalars[s] = 0ull;
    }
    DYG_CUDA(cudaDeviceSynchronize());
    G->bar_limit = kBarSpinLimit;
    return DYG_OK;
}

dyg_status read_scalars(dyg_graph *G, cudaStream_t st) { return read_scalars2(G, nullptr, st); }

dyg_status read_scalars2(dyg_graph *A, dyg_graph *B, cudaStream_t st) {
    if (B == A) B = nullptr;
    for (dyg_graph *G : {A, B})
        if (G)
            DYG_CUDA(cudaMemcpyAsync(G->ws.host_scalars, G->ws.scalars.p, kScalarBytes,
                                     cudaMemcpyDeviceToHost, st));
    DYG_CUDA(cudaStreamSynchronize(st));
    unsigned long long err = 0ull;
    for (dyg_graph *G : {A, B})
        if (G) {
            if (G->ws.host_scalars[S_LONG]) G->long_rows = true;
            err |= G->ws.host_scalars[S_ERR];
        }
    if (!(err & kErrBarrier)) return DYG_OK;
    for (dyg_graph *G : {A, B})
        if (G) {
            G->broken = true;
            DYG_TRY(recover_workspace(G));
        }
    set_error("a block timed out waiting at a grid barrier: the graphs hold part of an update");
    return DYG_ESTATE;
}

// After a scan on G and read_scalars: DYG_ESTATE if a tile of it gave up, so
// that nothing is placed or copied by its results.
static dyg_status check_scan(dyg_graph *G) {
    Workspace &ws = G->ws;
    if (!(ws.host_scalars[S_ERR] & kErrScan)) return DYG_OK;
    ws.host_scalars[S_ERR] &= ~(unsigned long long)kErrScan;
    DYG_CUDA(cudaMemcpy(ptr<unsigned long long>(ws.scalars) + S_ERR, ws.host_scalars + S_ERR,
                        sizeof(unsigned long long), cudaMemcpyHostToDevice));
    ws.scan_tickets = ws.host_scalars[S_SCAN];   // in step again
    set_error("a prefix scan tile timed out waiting for its predecessor");
    return DYG_ESTATE;
}

dyg_status check_usable(const dyg_graph *A, const dyg_graph *B) {
    if (!A->broken && (!B || !B->broken)) return DYG_OK;
    set_error("an earlier call was cut short and the graph holds part of its update; copy a whole graph over it");
    return DYG_ESTATE;
}

// ------------------------------------------------------------------ upload

dyg_status upload_graph(dyg_graph *G, uint32_t n, const uint64_t *row_ptr, const uint32_t *col,
                        const float *w) {
    const uint64_t slots = row_ptr[n];
    std::string msg;
    uint2 *h_desc = (uint2 *)malloc(sizeof(uint2) * (size_t)(n ? n : 1));
    uint32_t *h_cap = (uint32_t *)malloc(sizeof(uint32_t) * (size_t)(n ? n : 1));
    if (!h_desc || !h_cap) {
        free(h_desc);
        free(h_cap);
        set_error("host allocation failed");
        return DYG_ENOMEM;
    }
    uint64_t off = 0;
    for (uint32_t v = 0; v < n; ++v) {
        const uint64_t deg = row_ptr[v + 1] - row_ptr[v];
        const uint64_t cap = deg + G->slack;
        if (deg > kBigRow) G->long_rows = true;
        h_desc[v] = make_uint2((uint32_t)off, (uint32_t)deg);
        h_cap[v] = (uint32_t)cap;
        off += cap;
    }
    const uint64_t used = off;
    uint64_t arena = used + (uint64_t)((double)slots * G->headroom) + 1024;
    if (arena >= 0xFFFFFFFFull) {
        free(h_desc);
        free(h_cap);
        set_error("graph too large for 32-bit slot offsets");
        return DYG_EINVAL;
    }
    uint2 *h_slots = (uint2 *)calloc((size_t)(used ? used : 1), sizeof(uint2));
    float *h_w = (float *)calloc((size_t)(used ? used : 1), sizeof(float));
    if (!h_slots || !h_w) {
        free(h_desc);
        free(h_cap);
        free(h_slots);
        free(h_w);
        set_error("host allocation failed");
        return DYG_ENOMEM;
    }
    for (uint32_t v = 0; v < n; ++v) {
        const uint64_t o = h_desc[v].x;
        for (uint64_t j = row_ptr[v]; j < row_ptr[v + 1]; ++j) {
            const float rw = 1.0f / w[j];   // IEEE division: equals __frcp_rn(w)
            uint32_t rb;
            memcpy(&rb, &rw, 4);
            h_slots[o + (j - row_ptr[v])] = make_uint2(col[j], rb);
            h_w[o + (j - row_ptr[v])] = w[j];
        }
    }
    dyg_status rc = DYG_OK;
    G->g.n = n;
    G->g.arena_cap = arena;
    if (dev_alloc(&G->g.desc, sizeof(uint2) * (size_t)(n ? n : 1)) != cudaSuccess ||
        dev_alloc(&G->g.cap, sizeof(uint32_t) * (size_t)(n ? n : 1)) != cudaSuccess ||
        dev_alloc(&G->g.slots, sizeof(uint2) * (size_t)arena) != cudaSuccess ||
        dev_alloc(&G->g.wts, sizeof(float) * (size_t)arena) != cudaSuccess) {
        cudaGetLastError();
        set_error("cudaMalloc of the graph arena failed");
        rc = DYG_ENOMEM;
    }
    if (rc == DYG_OK) {
        cudaError_t e = cudaMemcpy(G->g.desc, h_desc, sizeof(uint2) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(G->g.cap, h_cap, sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(G->g.slots, h_slots, sizeof(uint2) * used, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemcpy(G->g.wts, h_w, sizeof(float) * used, cudaMemcpyHostToDevice);
        unsigned long long top = used;
        if (e == cudaSuccess) e = cudaMemcpy(G->g.top, &top, sizeof(top), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) rc = cuda_fail(e, "graph upload", __FILE__, __LINE__);
    }
    free(h_desc);
    free(h_cap);
    free(h_slots);
    free(h_w);
    return rc;
}

// ------------------------------------------------------------------ build
// Rows of an edge list in list order (functions.cpp:130-232): half-edge
// i = 2e enters row src[e] with column dst[e], i = 2e + 1 the other way.
//   count   degrees, by one atomic per half-edge, with the input checks
//   place   capacities scanned to row offsets; half-edge indices put into
//           their rows in any order (again one atomic each)
//   rows    each row's indices sorted, and its slots written from them
// The host built the rows with two passes of dependent loads over the edges
// and uploaded them with their padding; with the allocations 5 to 8 ms for the
// 116,000 and the 324,000 edges of a 48^3 mesh's two graphs, now 0.24 and
// 0.40.  Bound by the host's copy of the edges.

namespace {

__global__ void k_build_count(const uint32_t *src, const uint32_t *dst, const float *w, uint32_t m,
                              uint32_t n, uint32_t *cnt, unsigned long long *err) {
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
        const uint32_t u = src[e], v = dst[e];
        const float x = w[e];
        if (u >= n || v >= n || !(x > 0.0f) || !isfinite(x)) {
            atomicOr(err, (unsigned long long)kErrVertex);
            continue;
        }
        atomicAdd(cnt + u, 1u);
        atomicAdd(cnt + v, 1u);
    }
}

// Row offsets; the counters start over for the placement.
struct BuildScan {
    uint32_t *cnt;
    uint2 *desc;
    uint32_t *cap;
    uint32_t slack;
    unsigned long long *long_flag, *top;
    __device__ uint32_t load(uint32_t v) const { return cnt[v] + slack; }
    __device__ void store(uint32_t v, uint32_t off, uint32_t c) const {
        const uint32_t deg = c - slack;
        desc[v] = make_uint2(off, deg);
        cap[v] = c;
        cnt[v] = 0u;
        if (deg > kBigRow) *long_flag = 1ull;
    }
    __device__ void last(uint32_t total) const { *top = total; }
};

// With an error of the scan before it, the offsets are not to be used: the
// rows are left alone, and the call fails.
__global__ void k_build_place(const uint32_t *src, const uint32_t *dst, uint32_t m, const uint2 *desc,
                              uint32_t *cnt, uint32_t *idx, const unsigned long long *err) {
    if (*err) return;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < m; e += gridDim.x * blockDim.x) {
        const uint32_t u = src[e], v = dst[e];
        idx[desc[u].x + atomicAdd(cnt + u, 1u)] = 2u * e;
        idx[desc[v].x + atomicAdd(cnt + v, 1u)] = 2u * e + 1u;
    }
}

struct BuildList {
    const uint32_t *src, *dst;
    const float *w;
};
__device__ __forceinline__ void build_slot(const DevGraph &g, const BuildList &L, uint32_t at, uint32_t i) {
    const float x = L.w[i >> 1];
    g.slots[at] = make_uint2((i & 1u) ? L.src[i >> 1] : L.dst[i >> 1], __float_as_uint(__frcp_rn(x)));
    g.wts[at] = x;
}

constexpr uint32_t kBuildLane = 8;       // rows up to this length are sorted by one lane
constexpr uint32_t kBuildTile = 4096;    // indices a block sorts in shared memory at a time
constexpr uint32_t kBuildThreads = 256;

// Rows of up to kBigRow slots: by a lane, or by the warp 32 indices at a
// time, each index's rank counted against the row's others.  Longer rows go
// to `big` (n words) for k_build_big.
__global__ void __launch_bounds__(kBuildThreads)
k_build_rows(DevGraph g, BuildList L, const uint32_t *idx, uint32_t *big, unsigned long long *nbig,
             const unsigned long long *err) {
    if (*err) return;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t vb = first - lane; vb < g.n; vb += gridDim.x * blockDim.x) {
        const uint32_t v = vb + lane;
        const uint2 d = v < g.n ? g.desc[v] : make_uint2(0u, 0u);
        if (d.y <= kBuildLane) {
            uint32_t i[kBuildLane];
#pragma unroll
            for (uint32_t u = 0; u < kBuildLane; ++u) i[u] = u < d.y ? idx[d.x + u] : ~0u;
#pragma unroll
            for (uint32_t u = 0; u < kBuildLane; ++u)
                if (u < d.y) {
                    uint32_t r = 0;
#pragma unroll
                    for (uint32_t q = 0; q < kBuildLane; ++q) r += i[q] < i[u] ? 1u : 0u;
                    build_slot(g, L, d.x + r, i[u]);
                }
        } else if (d.y > kBigRow) {
            big[atomicAdd(nbig, 1ull)] = v;
        }
        unsigned todo = __ballot_sync(kFull, d.y > kBuildLane && d.y <= kBigRow);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1u;
            const uint32_t off = __shfl_sync(kFull, d.x, src), deg = __shfl_sync(kFull, d.y, src);
            for (uint32_t j0 = 0; j0 < deg; j0 += 32u) {
                const uint32_t mine = j0 + lane < deg ? idx[off + j0 + lane] : ~0u;
                uint32_t r = 0;
                for (uint32_t t0 = 0; t0 < deg; t0 += 32u) {
                    const uint32_t other = t0 + lane < deg ? idx[off + t0 + lane] : ~0u;
#pragma unroll
                    for (uint32_t q = 0; q < 32u; ++q)
                        r += __shfl_sync(kFull, other, q) < mine ? 1u : 0u;
                }
                if (mine != ~0u) build_slot(g, L, off + r, mine);
            }
        }
    }
}

// Rows longer than kBigRow, one block each: sorted in shared memory a tile at
// a time; an index of a row of several tiles then takes the place given by
// its rank in every tile (binary searches: the indices are distinct).
__global__ void __launch_bounds__(kBuildThreads)
k_build_big(DevGraph g, BuildList L, uint32_t *idx, const uint32_t *big, const unsigned long long *nbig) {
    __shared__ uint32_t s[kBuildTile];
    const uint32_t nb = (uint32_t)*nbig;
    for (uint32_t q = blockIdx.x; q < nb; q += gridDim.x) {
        const uint2 d = g.desc[big[q]];
        for (uint32_t t0 = 0; t0 < d.y; t0 += kBuildTile) {
            const uint32_t c = min(kBuildTile, d.y - t0);
            uint32_t N = 512u;
            while (N < c) N <<= 1;
            for (uint32_t j = threadIdx.x; j < N; j += blockDim.x) s[j] = j < c ? idx[d.x + t0 + j] : ~0u;
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
            if (d.y <= kBuildTile)
                for (uint32_t j = threadIdx.x; j < c; j += blockDim.x) build_slot(g, L, d.x + j, s[j]);
            else
                for (uint32_t j = threadIdx.x; j < c; j += blockDim.x) idx[d.x + t0 + j] = s[j];
            __syncthreads();
        }
        if (d.y <= kBuildTile) continue;
        for (uint32_t j = threadIdx.x; j < d.y; j += blockDim.x) {
            const uint32_t i = idx[d.x + j], own = j / kBuildTile;
            uint32_t r = j - own * kBuildTile;
            for (uint32_t t = 0; t * kBuildTile < d.y; ++t) {
                if (t == own) continue;
                uint32_t lo = 0, hi = min(kBuildTile, d.y - t * kBuildTile);
                while (lo < hi) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (idx[d.x + t * kBuildTile + mid] < i) lo = mid + 1u;
                    else hi = mid;
                }
                r += lo;
            }
            build_slot(g, L, d.x + r, i);
        }
        __syncthreads();
    }
}

// Device blocks of one call, freed when it leaves (after its work is done).
struct Temps {
    void *p[8];
    int k = 0;
    cudaError_t get(void **out, size_t bytes) {
        const cudaError_t e = dev_alloc(out, bytes ? bytes : 16);
        if (e == cudaSuccess) p[k++] = *out;
        return e;
    }
    void release() {
        if (k) cudaStreamSynchronize(nullptr);
        while (k) dev_free(p[--k]);
    }
    ~Temps() { release(); }
};

int grid_of(uint64_t items, uint32_t threads) {
    const uint64_t b = (items + threads - 1) / threads, cap = (uint64_t)num_sms() * 16;
    return (int)(b < 1 ? 1 : (b < cap ? b : cap));
}

}  // namespace

// The rows as the device makes them, by the host: for lists whose copy and
// half-edge indices (20 bytes an edge beside the graph's 36) do not fit the
// device.
static dyg_status build_on_host(dyg_graph *G, uint32_t n, uint64_t m, const uint32_t *src,
                                const uint32_t *dst, const float *w, bool *bad) {
    for (uint64_t e = 0; e < m; ++e)
        if (src[e] >= n || dst[e] >= n || !(w[e] > 0.0f) || !std::isfinite(w[e])) {
            *bad = true;
            return DYG_EINVAL;
        }
    std::vector<uint64_t> row_ptr, fill;
    std::vector<uint32_t> col;
    std::vector<float> ww;
    try {
        row_ptr.assign((size_t)n + 1, 0);
        fill.resize(n);
        col.resize(2 * m + 1);
        ww.resize(2 * m + 1);
    } catch (const std::bad_alloc &) {
        set_error("host allocation failed");
        return DYG_ENOMEM;
    }
    for (uint64_t e = 0; e < m; ++e) {
        row_ptr[src[e] + 1]++;
        row_ptr[dst[e] + 1]++;
    }
    for (uint32_t v = 0; v < n; ++v) {
        row_ptr[v + 1] += row_ptr[v];
        fill[v] = row_ptr[v];
    }
    for (uint64_t e = 0; e < m; ++e) {
        const uint64_t ps = fill[src[e]]++;
        col[ps] = dst[e];
        ww[ps] = w[e];
        const uint64_t pd = fill[dst[e]]++;
        col[pd] = src[e];
        ww[pd] = w[e];
    }
    return upload_graph(G, n, row_ptr.data(), col.data(), ww.data());
}

dyg_status build_graph(dyg_graph *G, uint32_t n, uint64_t m, const uint32_t *src, const uint32_t *dst,
                       const float *w, bool *bad) {
    *bad = false;
    const uint64_t used = 2 * m + (uint64_t)G->slack * n;
    const uint64_t arena = used + (uint64_t)((double)(2 * m) * G->headroom) + 1024;
    if (arena >= 0xFFFFFFFFull) {
        set_error("graph too large for 32-bit slot offsets");
        return DYG_EINVAL;
    }
    G->g.n = n;
    G->g.arena_cap = arena;
    const size_t nn = n ? n : 1;
    if (dev_alloc(&G->g.desc, sizeof(uint2) * nn) != cudaSuccess ||
        dev_alloc(&G->g.cap, sizeof(uint32_t) * nn) != cudaSuccess ||
        dev_alloc(&G->g.slots, sizeof(uint2) * (size_t)arena) != cudaSuccess ||
        dev_alloc(&G->g.wts, sizeof(float) * (size_t)arena) != cudaSuccess) {
        cudaGetLastError();
        set_error("cudaMalloc of the graph arena failed");
        return DYG_ENOMEM;
    }
    Temps tmp;
    void *d_src, *d_dst, *d_w, *d_cnt, *d_idx;
    if (tmp.get(&d_src, sizeof(uint32_t) * m) != cudaSuccess ||
        tmp.get(&d_dst, sizeof(uint32_t) * m) != cudaSuccess ||
        tmp.get(&d_w, sizeof(float) * m) != cudaSuccess ||
        tmp.get(&d_cnt, sizeof(uint32_t) * nn) != cudaSuccess ||
        tmp.get(&d_idx, sizeof(uint32_t) * (size_t)(used + nn)) != cudaSuccess ||
        scan_ensure(G->ws, n, nullptr) != DYG_OK) {
        cudaGetLastError();
        set_error("");
        tmp.release();
        for (void *p : {(void *)G->g.desc, (void *)G->g.cap, (void *)G->g.slots, (void *)G->g.wts}) dev_free(p);
        G->g.desc = nullptr;
        G->g.cap = nullptr;
        G->g.slots = nullptr;
        G->g.wts = nullptr;
        return build_on_host(G, n, m, src, dst, w, bad);
    }
    cudaStream_t st = nullptr;
    unsigned long long *sc = ptr<unsigned long long>(G->ws.scalars);
    DYG_CUDA(cudaMemsetAsync(d_cnt, 0, sizeof(uint32_t) * nn, st));
    DYG_CUDA(cudaMemcpyAsync(d_src, src, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, st));
    DYG_CUDA(cudaMemcpyAsync(d_dst, dst, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, st));
    DYG_CUDA(cudaMemcpyAsync(d_w, w, sizeof(float) * m, cudaMemcpyHostToDevice, st));
    uint32_t *ds = (uint32_t *)d_src, *dd = (uint32_t *)d_dst, *cnt = (uint32_t *)d_cnt;
    uint32_t *idx = (uint32_t *)d_idx, *big = idx + used;
    if (m) {
        k_build_count<<<grid_of(m, 256), 256, 0, st>>>(ds, dd, (float *)d_w, (uint32_t)m, n, cnt, sc + S_ERR);
        count_launch();
        DYG_CUDA(cudaGetLastError());
        // nothing is placed by ids that were not checked
        DYG_TRY(read_scalars(G, st));
        if (G->ws.host_scalars[S_ERR]) {
            *bad = true;
            return DYG_EINVAL;
        }
    }
    if (n) {
        DYG_TRY(scan_op(G->ws, BuildScan{cnt, G->g.desc, G->g.cap, G->slack, sc + S_LONG, sc + S_TOP}, n,
                        st));
    }
    if (m) {
        const BuildList L{ds, dd, (float *)d_w};
        k_build_place<<<grid_of(m, 256), 256, 0, st>>>(ds, dd, (uint32_t)m, G->g.desc, cnt, idx, sc + S_ERR);
        count_launch();
        k_build_rows<<<grid_of(n, kBuildThreads), kBuildThreads, 0, st>>>(G->g, L, idx, big, sc + S_NBIG, sc + S_ERR);
        count_launch();
        k_build_big<<<num_sms() * 4, kBuildThreads, 0, st>>>(G->g, L, idx, big, sc + S_NBIG);
        count_launch();
        DYG_CUDA(cudaGetLastError());
        DYG_CUDA(cudaMemsetAsync(sc + S_NBIG, 0, sizeof(unsigned long long), st));
    }
    DYG_TRY(read_scalars(G, st));   // synchronizes; picks up a long row
    return check_scan(G);
}

// ----------------------------------------------------------------- export

namespace {

struct DegreeScan {
    const uint2 *desc;
    unsigned long long *row_ptr;   // n + 1
    uint32_t n;
    __device__ uint32_t load(uint32_t v) const { return desc[v].y; }
    __device__ void store(uint32_t v, uint32_t excl, uint32_t) const { row_ptr[v] = excl; }
    __device__ void last(uint32_t total) const { row_ptr[n] = total; }
};

__global__ void k_count_slots(const uint2 *desc, uint32_t n, unsigned long long *sum) {
    uint32_t mine = 0u;   // the slots of a graph fit 32 bits
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        mine += desc[v].y;
    mine = __reduce_add_sync(kFull, mine);
    if ((threadIdx.x & 31u) == 0u && mine) atomicAdd(sum, (unsigned long long)mine);
}

// Rows to their place in a CSR: a group of eight lanes per row, rows of a
// lattice being shorter than that; rows over kBigRow by the whole warp.
__global__ void __launch_bounds__(256)
k_export_rows(DevGraph g, const unsigned long long *row_ptr, uint32_t *col, float *w) {
    const uint32_t lane = threadIdx.x & 31u, sub = lane & 7u;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4u; v0 < g.n; v0 += 4u * warps) {
        const uint32_t v = v0 + (lane >> 3);
        const uint2 d = v < g.n ? g.desc[v] : make_uint2(0u, 0u);
        const unsigned long long o = v < g.n ? row_ptr[v] : 0ull;
        if (d.y <= kBigRow) {
#pragma unroll 4
            for (uint32_t j = sub; j < d.y; j += 8u) {
                col[o + j] = g.slots[d.x + j].x;
                w[o + j] = g.wts[d.x + j];
            }
        }
        unsigned todo = __ballot_sync(kFull, sub == 0u && d.y > kBigRow);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1u;
            const uint32_t off = __shfl_sync(kFull, d.x, src), deg = __shfl_sync(kFull, d.y, src);
            const unsigned long long to = __shfl_sync(kFull, o, src);
#pragma unroll 4
            for (uint32_t j = lane; j < deg; j += 32u) {
                col[to + j] = g.slots[off + j].x;
                w[to + j] = g.wts[off + j];
            }
        }
    }
}

}  // namespace

dyg_status count_slots_enqueue(dyg_graph *G, cudaStream_t st) {
    unsigned long long *sum = ptr<unsigned long long>(G->ws.scalars) + S_SLOTS;
    DYG_CUDA(cudaMemsetAsync(sum, 0, sizeof(unsigned long long), st));
    k_count_slots<<<grid_of(G->g.n, 256), 256, 0, st>>>(G->g.desc, G->g.n, sum);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

// The rows by the host from a copy of the arena, for when the device has no
// room for them twice.
static dyg_status export_on_host(dyg_graph *G, uint64_t *row_ptr, uint32_t *col, float *w, uint64_t slot_cap) {
    const uint32_t n = G->g.n;
    DYG_TRY(read_scalars(G, nullptr));
    const size_t top = (size_t)G->ws.host_scalars[S_TOP];
    std::vector<uint2> desc, slots;
    std::vector<float> wts;
    try {
        desc.resize(n);
        slots.resize(col ? top : 0);
        wts.resize(w ? top : 0);
    } catch (const std::bad_alloc &) {
        set_error("host allocation failed");
        return DYG_ENOMEM;
    }
    DYG_CUDA(cudaMemcpy(desc.data(), G->g.desc, sizeof(uint2) * n, cudaMemcpyDeviceToHost));
    if (!slots.empty()) DYG_CUDA(cudaMemcpy(slots.data(), G->g.slots, sizeof(uint2) * top, cudaMemcpyDeviceToHost));
    if (!wts.empty()) DYG_CUDA(cudaMemcpy(wts.data(), G->g.wts, sizeof(float) * top, cudaMemcpyDeviceToHost));
    uint64_t o = 0;
    for (uint32_t v = 0; v < n; ++v) {
        row_ptr[v] = o;
        for (uint32_t j = 0; j < desc[v].y && o + j < slot_cap; ++j) {
            if (col) col[o + j] = slots[desc[v].x + j].x;
            if (w) w[o + j] = wts[desc[v].x + j];
        }
        o += desc[v].y;
    }
    row_ptr[n] = o;
    return DYG_OK;
}

dyg_status export_graph(dyg_graph *G, uint64_t *row_ptr, uint32_t *col, float *w, uint64_t slot_cap) {
    const uint32_t n = G->g.n;
    row_ptr[0] = 0;
    if (n == 0) return DYG_OK;
    cudaStream_t st = nullptr;
    Temps tmp;
    void *d_rp, *d_col = nullptr, *d_w = nullptr;
    bool ok = tmp.get(&d_rp, sizeof(uint64_t) * ((size_t)n + 1)) == cudaSuccess;
    if (ok) {
        const dyg_status rc =
            scan_op(G->ws, DegreeScan{G->g.desc, (unsigned long long *)d_rp, n}, n, st);
        ok = rc == DYG_OK;
        if (!ok && rc != DYG_ENOMEM) return rc;
    }
    if (ok) {
        DYG_CUDA(cudaMemcpyAsync(row_ptr, d_rp, sizeof(uint64_t) * ((size_t)n + 1), cudaMemcpyDeviceToHost, st));
        DYG_TRY(read_scalars(G, st));
        DYG_TRY(check_scan(G));
        const uint64_t total = row_ptr[n], out = total < slot_cap ? total : slot_cap;
        if (!out || (!col && !w)) return DYG_OK;
        ok = tmp.get(&d_col, sizeof(uint32_t) * total) == cudaSuccess &&
             tmp.get(&d_w, sizeof(float) * total) == cudaSuccess;
        if (ok) {
            k_export_rows<<<grid_of((uint64_t)n * 8, 256), 256, 0, st>>>(
                G->g, (unsigned long long *)d_rp, (uint32_t *)d_col, (float *)d_w);
            count_launch();
            DYG_CUDA(cudaGetLastError());
            if (col) DYG_CUDA(cudaMemcpyAsync(col, d_col, sizeof(uint32_t) * out, cudaMemcpyDeviceToHost, st));
            if (w) DYG_CUDA(cudaMemcpyAsync(w, d_w, sizeof(float) * out, cudaMemcpyDeviceToHost, st));
            DYG_CUDA(cudaStreamSynchronize(st));
        }
    }
    if (ok) return DYG_OK;
    cudaGetLastError();
    set_error("");   // a scan's status words that did not fit either
    tmp.release();
    return export_on_host(G, row_ptr, col, w, slot_cap);
}

dyg_status grow_arena(dyg_graph *G, uint64_t min_cap, cudaStream_t st) {
    uint64_t cap = G->g.arena_cap + G->g.arena_cap / 2;
    if (cap < min_cap + min_cap / 4 + 1024) cap = min_cap + min_cap / 4 + 1024;
    if (cap >= 0xFFFFFFFFull) cap = 0xFFFFFFFEull;
    if (cap < min_cap) {
        set_error("arena would exceed 32-bit slot offsets");
        return DYG_ENOMEM;
    }
    uint2 *ns = nullptr;
    float *nw = nullptr;
    cudaError_t e = dev_alloc(&ns, sizeof(uint2) * (size_t)cap);
    if (e == cudaSuccess) e = dev_alloc(&nw, sizeof(float) * (size_t)cap);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (ns) dev_free(ns);
        set_error("cudaMalloc while growing the arena failed");
        return DYG_ENOMEM;
    }
    DYG_TRY(read_scalars(G, st));
    const unsigned long long top = G->ws.host_scalars[S_TOP];
    DYG_CUDA(cudaMemcpyAsync(ns, G->g.slots, sizeof(uint2) * (size_t)top, cudaMemcpyDeviceToDevice, st));
    DYG_CUDA(cudaMemcpyAsync(nw, G->g.wts, sizeof(float) * (size_t)top, cudaMemcpyDeviceToDevice, st));
    DYG_CUDA(cudaStreamSynchronize(st));
    dev_free(G->g.slots);
    dev_free(G->g.wts);
    G->g.slots = ns;
    G->g.wts = nw;
    G->g.arena_cap = cap;
    return DYG_OK;
}

// -------------------------------------------------------------- snapshots

namespace {
// n bytes (a multiple of 4) by the whole grid, 16 at a time, four loads per
// thread in flight; both pointers start on a 16-byte boundary.
__device__ __forceinline__ void copy_bytes(void *dst, const void *src, uint64_t n) {
    const uint4 *s = static_cast<const uint4 *>(src);
    uint4 *d = static_cast<uint4 *>(dst);
    const uint64_t n16 = n >> 4, step = (uint64_t)gridDim.x * blockDim.x;
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; i + 3u * step < n16; i += 4u * step) {
        const uint4 a = s[i], b = s[i + step], c = s[i + 2u * step], e = s[i + 3u * step];
        d[i] = a;
        d[i + step] = b;
        d[i + 2u * step] = c;
        d[i + 3u * step] = e;
    }
    for (; i < n16; i += step) d[i] = s[i];
    const uint32_t tail = (uint32_t)(n & 15u) >> 2;
    if (blockIdx.x == 0 && threadIdx.x < tail)
        static_cast<uint32_t *>(dst)[(n16 << 2) + threadIdx.x] =
            static_cast<const uint32_t *>(src)[(n16 << 2) + threadIdx.x];
}

// A graph's arrays up to its arena top, which stays on the device.  Bound by
// memory for large graphs and by its launch for small ones, where five copies,
// a memset and a host read of the top took 30 us.
__global__ void __launch_bounds__(256) k_copy_graph(DevGraph d, DevGraph s, unsigned long long *long_flag) {
    const uint64_t top = *s.top;
    copy_bytes(d.desc, s.desc, sizeof(uint2) * (uint64_t)s.n);
    copy_bytes(d.cap, s.cap, sizeof(uint32_t) * (uint64_t)s.n);
    copy_bytes(d.slots, s.slots, sizeof(uint2) * top);
    copy_bytes(d.wts, s.wts, sizeof(float) * top);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *d.top = top;
        *long_flag = 0ull;
    }
}
}  // namespace

dyg_status copy_graph_enqueue(dyg_graph *dst, const dyg_graph *src, cudaStream_t st) {
    const uint64_t bytes = 12ull * src->g.n + 12ull * src->g.arena_cap;   // the top is at most this
    const uint64_t want = (bytes + 256 * 64 - 1) / (256 * 64), cap = (uint64_t)num_sms() * 8;
    k_copy_graph<<<(unsigned)(want < 1 ? 1 : (want < cap ? want : cap)), 256, 0, st>>>(
        dst->g, src->g, ptr<unsigned long long>(dst->ws.scalars) + S_LONG);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    return DYG_OK;
}

// ---------------------------------------------------------- exclusive scan
namespace {
struct CopyScan {
    const uint32_t *in;
    uint32_t *out;
    __device__ uint32_t load(uint32_t i) const { return in[i]; }
    __device__ void store(uint32_t i, uint32_t excl, uint32_t) const { out[i] = excl; }
    __device__ void last(uint32_t) const {}
};
}  // namespace

dyg_status exclusive_scan_u32(Workspace &ws, const uint32_t *in, uint32_t *out, uint32_t m,
                              cudaStream_t st) {
    return scan_op(ws, CopyScan{in, out}, m, st);
}

// -------------------------------------------------------------- compaction

// Rows keep slack; a vertex with neither slots nor capacity (an unoccupied
// vertex of a pool graph) keeps none.
__global__ void k_new_caps(DevGraph g, uint32_t slack, uint32_t *caps) {
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= g.n) return;
    const uint32_t deg = g.desc[v].y;
    caps[v] = (deg == 0u && g.cap[v] == 0u) ? 0u : deg + slack;
}

// One warp per row: consecutive lanes copy consecutive slots into the new
// arena, four loads per lane issued before their stores (the new arena never
// overlaps the old one).  Lane 0 reads the descriptor and hands it to the
// warp before it rewrites it.
__global__ void k_move_rows(DevGraph g, uint2 *ns, float *nw, const uint32_t *off,
                            const uint32_t *caps) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < g.n; v += warps) {
        uint2 d = make_uint2(0u, 0u);
        if (lane == 0u) d = g.desc[v];
        d.x = __shfl_sync(kFull, d.x, 0);
        d.y = __shfl_sync(kFull, d.y, 0);
        const uint32_t o = off[v];
        for (uint32_t j0 = 0; j0 < d.y; j0 += 128u) {
            uint2 sv[4];
            float wv[4];
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u) {
                const uint32_t j = j0 + lane + 32u * u;
                if (j < d.y) {
                    sv[u] = g.slots[d.x + j];
                    wv[u] = g.wts[d.x + j];
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < 4u; ++u) {
                const uint32_t j = j0 + lane + 32u * u;
                if (j < d.y) {
                    ns[o + j] = sv[u];
                    nw[o + j] = wv[u];
                }
            }
        }
        if (lane == 0u) {
            g.desc[v] = make_uint2(o, d.y);
            g.cap[v] = caps[v];
        }
    }
}

dyg_status compact_graph(dyg_graph *G, cudaStream_t st) {
    Workspace &ws = G->ws;
    const uint32_t n = G->g.n;
    if (n == 0) return DYG_OK;
    DYG_TRY(ensure(ws.flags, sizeof(uint32_t) * (size_t)n));
    DYG_TRY(ensure(ws.pos, sizeof(uint32_t) * (size_t)n));
    const int th = 256;
    const int gr = (int)((n + th - 1) / th);
    k_new_caps<<<gr, th, 0, st>>>(G->g, G->slack, ptr<uint32_t>(ws.flags));
    count_launch();
    DYG_TRY(exclusive_scan_u32(ws, ptr<uint32_t>(ws.flags), ptr<uint32_t>(ws.pos), n, st));
    uint32_t last_off = 0, last_cap = 0;
    DYG_CUDA(cudaMemcpyAsync(&last_off, ptr<uint32_t>(ws.pos) + n - 1, 4, cudaMemcpyDeviceToHost, st));
    DYG_CUDA(cudaMemcpyAsync(&last_cap, ptr<uint32_t>(ws.flags) + n - 1, 4, cudaMemcpyDeviceToHost, st));
    DYG_TRY(read_scalars(G, st));
    DYG_TRY(check_scan(G));
    const uint64_t used = (uint64_t)last_off + last_cap;
    uint64_t cap = used + (uint64_t)((double)used * G->headroom) + 1024;
    if (cap < G->g.arena_cap / 2) cap = G->g.arena_cap / 2 > used ? G->g.arena_cap / 2 : cap;
    if (cap >= 0xFFFFFFFFull) cap = 0xFFFFFFFEull;
    uint2 *ns = nullptr;
    float *nw = nullptr;
    cudaError_t e = dev_alloc(&ns, sizeof(uint2) * (size_t)cap);
    if (e == cudaSuccess) e = dev_alloc(&nw, sizeof(float) * (size_t)cap);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (ns) dev_free(ns);
        set_error("cudaMalloc during compaction failed");
        return DYG_ENOMEM;
    }
    k_move_rows<<<num_sms() * 8, th, 0, st>>>(G->g, ns, nw, ptr<uint32_t>(ws.pos),
                                              ptr<uint32_t>(ws.flags));
    count_launch();
    DYG_CUDA(cudaGetLastError());
    unsigned long long top = used;
    DYG_CUDA(cudaMemcpyAsync(G->g.top, &top, sizeof(top), cudaMemcpyHostToDevice, st));
    DYG_CUDA(cudaStreamSynchronize(st));
    dev_free(G->g.slots);
    dev_free(G->g.wts);
    G->g.slots = ns;
    G->g.wts = nw;
    G->g.arena_cap = cap;
    return DYG_OK;
}

// ----------------------------------------------------------- vertex ranges
// A graph that holds many graphs at vertex offsets (the serving pool) loads,
// saves and clears one graph's rows at a time.

// One warp per vertex: row v0 + i goes to [out_off[i], out_off[i] + deg) of
// col / w, with columns made local (minus v0).
__global__ void k_gather_rows(DevGraph g, uint32_t v0, uint32_t n, const unsigned long long *out_off,
                              uint32_t *col, float *w) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n;
         i += (gridDim.x * blockDim.x) >> 5) {
        const uint2 d = g.desc[v0 + i];
        const unsigned long long o = out_off[i];
        for (uint32_t j = lane; j < d.y; j += 32u) {
            col[o + j] = g.slots[d.x + j].x - v0;
            w[o + j] = g.wts[d.x + j];
        }
    }
}

// One warp per vertex: row i of the staged CSR goes to the arena at
// top + rp[i] + slack * i, columns shifted by v0, with the correctly rounded
// 1/w beside each column.
__global__ void k_place_rows(DevGraph g, uint32_t v0, uint32_t n, unsigned long long top,
                             uint32_t slack, const unsigned long long *rp, const uint32_t *col,
                             const float *w, unsigned long long *long_flag) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n;
         i += (gridDim.x * blockDim.x) >> 5) {
        const unsigned long long a = rp[i];
        const uint32_t deg = (uint32_t)(rp[i + 1] - a);
        const unsigned long long off = top + a + (unsigned long long)slack * i;
        for (uint32_t j = lane; j < deg; j += 32u) {
            const float x = w[a + j];
            g.slots[off + j] = make_uint2(col[a + j] + v0, __float_as_uint(__frcp_rn(x)));
            g.wts[off + j] = x;
        }
        if (lane == 0u) {
            g.desc[v0 + i] = make_uint2((uint32_t)off, deg);
            g.cap[v0 + i] = deg + slack;
            if (deg > kBigRow) *long_flag = 1ull;
        }
    }
}

dyg_status load_range(dyg_graph *G, uint32_t v0, uint32_t n, const uint64_t *row_ptr,
                      const uint32_t *col, const float *w, cudaStream_t st) {
    if (n == 0) return DYG_OK;
    if ((uint64_t)v0 + n > G->g.n) {
        set_error("vertex range outside the graph");
        return DYG_EINVAL;
    }
    const uint64_t m = row_ptr[n];
    const uint64_t need = m + (uint64_t)G->slack * n;
    DYG_TRY(read_scalars(G, st));
    uint64_t top = G->ws.host_scalars[S_TOP];
    if (top + need > G->g.arena_cap) {
        // holes left by evicted graphs and moved rows go first
        DYG_TRY(compact_graph(G, st));
        DYG_TRY(read_scalars(G, st));
        top = G->ws.host_scalars[S_TOP];
        if (top + need > G->g.arena_cap) DYG_TRY(grow_arena(G, top + need, st));
    }
    if (top + need >= 0xFFFFFFFFull) {
        set_error("arena would exceed 32-bit slot offsets");
        return DYG_ENOMEM;
    }
    Workspace &ws = G->ws;
    DYG_TRY(ensure(ws.f_uid, sizeof(unsigned long long) * ((size_t)n + 1)));
    DYG_TRY(ensure(ws.cand_x, sizeof(uint32_t) * (m ? m : 1)));
    DYG_TRY(ensure(ws.cand_w, sizeof(float) * (m ? m : 1)));
    DYG_CUDA(cudaMemcpyAsync(ws.f_uid.p, row_ptr, sizeof(uint64_t) * ((size_t)n + 1),
                             cudaMemcpyHostToDevice, st));
    if (m) {
        DYG_CUDA(cudaMemcpyAsync(ws.cand_x.p, col, sizeof(uint32_t) * m, cudaMemcpyHostToDevice, st));
        DYG_CUDA(cudaMemcpyAsync(ws.cand_w.p, w, sizeof(float) * m, cudaMemcpyHostToDevice, st));
    }
    unsigned long long *sc = ptr<unsigned long long>(ws.scalars);
    const int gr = (int)std::min<uint64_t>(((uint64_t)n * 32 + 255) / 256, (uint64_t)num_sms() * 16);
    k_place_rows<<<gr, 256, 0, st>>>(G->g, v0, n, top, G->slack, ptr<unsigned long long>(ws.f_uid),
                                     ptr<uint32_t>(ws.cand_x), ptr<float>(ws.cand_w), sc + S_LONG);
    count_launch();
    DYG_CUDA(cudaGetLastError());
    const unsigned long long ntop = top + need;
    DYG_CUDA(cudaMemcpyAsync(G->g.top, &ntop, sizeof(ntop), cudaMemcpyHostToDevice, st));
    DYG_TRY(read_scalars(G, st));   // synchronizes; picks up a long row
    return DYG_OK;
}

dyg_status save_range(dyg_graph *G, uint32_t v0, uint32_t n, std::vector<uint64_t> &row_ptr,
                      std::vector<uint32_t> &col, std::vector<float> &w, cudaStream_t st) {
    row_ptr.assign((size_t)n + 1, 0);
    col.clear();
    w.clear();
    if (n == 0) return DYG_OK;
    std::vector<uint2> h_desc(n);
    DYG_CUDA(cudaMemcpyAsync(h_desc.data(), G->g.desc + v0, sizeof(uint2) * n, cudaMemcpyDeviceToHost, st));
    DYG_CUDA(cudaStreamSynchronize(st));
    std::vector<unsigned long long> off(n);
    for (uint32_t v = 0; v < n; ++v) {
        off[v] = row_ptr[v];
        row_ptr[v + 1] = row_ptr[v] + h_desc[v].y;
    }
    const uint64_t m = row_ptr[n];
    col.resize(m);
    w.resize(m);
    if (m == 0) return DYG_OK;
    Workspace &ws = G->ws;
    DYG_TRY(ensure(ws.f_uid, sizeof(unsigned long long) * n));
    DYG_TRY(ensure(ws.cand_x, sizeof(uint32_t) * m));
    DYG_TRY(ensure(ws.cand_w, sizeof(float) * m));
    DYG_CUDA(cudaMemcpyAsync(ws.f_uid.p, off.data(), sizeof(unsigned long long) * n,
                             cudaMemcpyHostToDevice, st));
    const int gr = (int)std::min<uint64_t>(((uint64_t)n * 32 + 255) / 256, (uint64_t)num_sms() * 16);
    k_gather_rows<<<gr, 256, 0, st>>>(G->g, v0, n, ptr<unsigned long long>(ws.f_uid),
                                      ptr<uint32_t>(ws.cand_x), ptr<float>(ws.cand_w));
    count_launch();
    DYG_CUDA(cudaGetLastError());
    DYG_CUDA(cudaMemcpyAsync(col.data(), ws.cand_x.p, sizeof(uint32_t) * m, cudaMemcpyDeviceToHost, st));
    DYG_CUDA(cudaMemcpyAsync(w.data(), ws.cand_w.p, sizeof(float) * m, cudaMemcpyDeviceToHost, st));
    DYG_CUDA(cudaStreamSynchronize(st));
    return DYG_OK;
}

dyg_status clear_range(dyg_graph *G, uint32_t v0, uint32_t n, cudaStream_t st) {
    if (n == 0) return DYG_OK;
    DYG_CUDA(cudaMemsetAsync(G->g.desc + v0, 0, sizeof(uint2) * n, st));
    DYG_CUDA(cudaMemsetAsync(G->g.cap + v0, 0, sizeof(uint32_t) * n, st));
    return DYG_OK;
}

}  // namespace dyg

extern "C" uint64_t dyg_kernel_launches(void) { return dyg::g_launches.load(); }
