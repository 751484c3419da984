// capi.cu -- the extern "C" boundary (include/dyg.h): graph handles and the
// incremental / decremental batch and stream entry points.
//
// The batch flows themselves are in pipeline.cu.  This file places the
// caller's arrays: host inputs of up to kPackMax bytes in all are packed into
// one page-locked block and copied once, results come back the same way, and
// device arrays are used where they are.
#include <math.h>
#include <string.h>

#include <string>

#include "dyg_internal.cuh"

namespace dyg {

static thread_local std::string g_last_error;

void set_error(const std::string &msg) { g_last_error = msg; }

dyg_status cuda_fail(cudaError_t e, const char *what, const char *file, int line) {
    cudaGetLastError();
    set_error(std::string(what) + " failed: " + cudaGetErrorString(e) + " (" + file + ":" +
              std::to_string(line) + ")");
    return DYG_ECUDA;
}

PtrPlace ptr_place(const void *p, int device) {
    if (!p) return kOnHost;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return kOnHost;
    }
    if (at.type == cudaMemoryTypeManaged) return kOnDevice;
    if (at.type == cudaMemoryTypeDevice) return at.device == device ? kOnDevice : kOnOtherDevice;
    return kOnHost;
}

dyg_status check_same_device(int device, const void *const *ptrs, const char *const *names,
                             int count) {
    for (int i = 0; i < count; ++i)
        if (ptrs[i] && ptr_place(ptrs[i], device) == kOnOtherDevice) {
            set_error(std::string(names[i]) + " is device memory of another GPU than the graph's (device " +
                      std::to_string(device) + ")");
            return DYG_EINVAL;
        }
    return DYG_OK;
}

namespace {

struct DeviceGuard {
    int prev = -1;
    bool changed = false;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) {
            changed = cudaSetDevice(dev) == cudaSuccess;
        }
        cudaGetLastError();
    }
    ~DeviceGuard() {
        if (changed) cudaSetDevice(prev);
    }
};

bool on_device(const void *p) {
    if (!p) return false;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

// The arrays of one call.  Where each lives is asked once.  Host inputs of up
// to kPackMax bytes together go to the device in one copy from pinned memory,
// and host results come back in one that the call's own wait covers: three
// pageable copies in and three out, each waited for by itself, were 45 of the
// 130 us of a 32-edge batch.  Larger arrays are copied one by one (staging
// them would cost the host a pass over memory that the copies overlap).
constexpr size_t kPackMax = 1u << 20;
constexpr size_t kScalarPinned = 256;   // bytes of a handle's pinned mirror
static_assert(kScalarBytes <= kScalarPinned, "the mirror holds scalars and counts");

struct InArray {
    const char *name;
    const void *p;
    size_t bytes;
    Buf *own;                   // device copy of a large array
    const void *dev = nullptr;  // where the kernels read it
    bool host = false;
};
struct OutArray {
    const char *name;
    void *p;
    size_t bytes;               // 0: not wanted by anyone
    Buf *own;
    void *dev = nullptr;
    bool host = false;          // the caller's array is host memory
    size_t at = 0;              // in the packed block
};

size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }

dyg_status ensure_pinned(Buf &b, size_t bytes) {
    if (b.bytes >= bytes) return DYG_OK;
    host_free(b.p, b.bytes);
    b = Buf{};
    size_t want = 4096;
    while (want < bytes) want *= 2;
    DYG_CUDA(host_alloc(&b.p, want));
    b.bytes = want;
    return DYG_OK;
}

dyg_status check_places(int device, InArray *in, int nin, OutArray *out, int nout) {
    auto place = [&](const void *p, const char *name, bool *host) {
        const PtrPlace w = ptr_place(p, device);
        *host = p && w == kOnHost;
        if (w != kOnOtherDevice) return DYG_OK;
        set_error(std::string(name) + " is device memory of another GPU than the graph's (device " +
                  std::to_string(device) + ")");
        return DYG_EINVAL;
    };
    for (int i = 0; i < nin; ++i) DYG_TRY(place(in[i].p, in[i].name, &in[i].host));
    for (int i = 0; i < nout; ++i) DYG_TRY(place(out[i].p, out[i].name, &out[i].host));
    return DYG_OK;
}

dyg_status stage_inputs(Workspace &ws, InArray *in, int nin, cudaStream_t st) {
    size_t total = 0;
    for (int i = 0; i < nin; ++i) {
        in[i].dev = in[i].p;
        if (in[i].host) total += align16(in[i].bytes);
    }
    if (total == 0) return DYG_OK;
    if (total > kPackMax) {
        for (int i = 0; i < nin; ++i) {
            if (!in[i].host) continue;
            DYG_TRY(ensure(*in[i].own, in[i].bytes));
            DYG_CUDA(cudaMemcpyAsync(in[i].own->p, in[i].p, in[i].bytes, cudaMemcpyHostToDevice, st));
            in[i].dev = in[i].own->p;
        }
        return DYG_OK;
    }
    // every call waits for its copies, so the pinned block is free again
    DYG_TRY(ensure_pinned(ws.pin_in, total));
    DYG_TRY(ensure(ws.io_in, total));
    size_t at = 0;
    for (int i = 0; i < nin; ++i) {
        if (!in[i].host) continue;
        memcpy(static_cast<char *>(ws.pin_in.p) + at, in[i].p, in[i].bytes);
        in[i].dev = static_cast<char *>(ws.io_in.p) + at;
        at += align16(in[i].bytes);
    }
    DYG_CUDA(cudaMemcpyAsync(ws.io_in.p, ws.pin_in.p, total, cudaMemcpyHostToDevice, st));
    return DYG_OK;
}

// Device places for the results: the caller's own where it is device memory.
// *packed gets the bytes of the block the others share, 0 if they are large.
dyg_status place_outputs(Workspace &ws, OutArray *out, int nout, size_t *packed) {
    size_t total = 0;
    for (int i = 0; i < nout; ++i) {
        out[i].dev = out[i].p && !out[i].host ? out[i].p : nullptr;
        if (out[i].dev || !out[i].bytes) continue;
        out[i].at = total;
        total += align16(out[i].bytes);
    }
    *packed = total <= kPackMax ? total : 0;
    if (*packed) DYG_TRY(ensure(ws.io_out, total));
    for (int i = 0; i < nout; ++i) {
        if (out[i].dev || !out[i].bytes) continue;
        if (*packed) {
            out[i].dev = static_cast<char *>(ws.io_out.p) + out[i].at;
        } else {
            DYG_TRY(ensure(*out[i].own, out[i].bytes));
            out[i].dev = out[i].own->p;
        }
    }
    return DYG_OK;
}

bool any_host(const OutArray *out, int nout) {
    for (int i = 0; i < nout; ++i)
        if (out[i].host) return true;
    return false;
}

// Host results to the caller: from the pinned block the call fetched, or by
// one copy each (*wait is set: the stream is to be waited for).
dyg_status deliver(Workspace &ws, const OutArray *out, int nout, size_t packed, cudaStream_t st,
                   bool *wait) {
    for (int i = 0; i < nout; ++i) {
        if (!out[i].host) continue;
        if (packed) {
            memcpy(out[i].p, static_cast<char *>(ws.pin_out.p) + out[i].at, out[i].bytes);
        } else {
            DYG_CUDA(cudaMemcpyAsync(out[i].p, out[i].dev, out[i].bytes, cudaMemcpyDeviceToHost, st));
            *wait = true;
        }
    }
    return DYG_OK;
}

// The recovered edges of a deletion call.  They are fetched with the other
// results as far as a call usually brings them (four per deletion); how many
// there are is only known after the wait.
struct RecordsOut {
    uint32_t *src, *dst;
    uint8_t *kind;
    uint64_t cap;
    bool host, any_host;        // all wanted arrays, any of them, are host memory
    uint64_t fetched = 0;
    size_t at = 0;              // of the fetched records in the pinned block
    bool wanted() const { return src || dst || kind; }
    dyg_status fetch(Workspace &ws, cudaStream_t st) {
        if (!fetched) return DYG_OK;
        char *pin = static_cast<char *>(ws.pin_out.p) + at;
        if (src) DYG_CUDA(cudaMemcpyAsync(pin, ws.rx2.p, 4 * fetched, cudaMemcpyDeviceToHost, st));
        if (dst) DYG_CUDA(cudaMemcpyAsync(pin + 4 * fetched, ws.ry2.p, 4 * fetched, cudaMemcpyDeviceToHost, st));
        if (kind) DYG_CUDA(cudaMemcpyAsync(pin + 8 * fetched, ws.rk2.p, fetched, cudaMemcpyDeviceToHost, st));
        return DYG_OK;
    }
    dyg_status deliver(Workspace &ws, uint64_t total, cudaStream_t st, bool *wait) {
        const uint64_t n = total < cap ? total : cap;
        if (!n || !wanted()) return DYG_OK;
        if (n <= fetched) {
            const char *pin = static_cast<const char *>(ws.pin_out.p) + at;
            if (src) memcpy(src, pin, 4 * n);
            if (dst) memcpy(dst, pin + 4 * fetched, 4 * n);
            if (kind) memcpy(kind, pin + 8 * fetched, n);
            return DYG_OK;
        }
        if (src) DYG_CUDA(cudaMemcpyAsync(src, ws.rx2.p, 4 * n, cudaMemcpyDefault, st));
        if (dst) DYG_CUDA(cudaMemcpyAsync(dst, ws.ry2.p, 4 * n, cudaMemcpyDefault, st));
        if (kind) DYG_CUDA(cudaMemcpyAsync(kind, ws.rk2.p, n, cudaMemcpyDefault, st));
        *wait |= any_host;
        return DYG_OK;
    }
};

// Pinned room for the packed results and the records to fetch: at most what
// the record buffers hold to begin with (four per deletion).
dyg_status prepare_fetch(Workspace &ws, size_t packed, RecordsOut *rec, uint64_t n) {
    size_t bytes = packed;
    if (rec && rec->wanted() && rec->host && packed) {
        uint64_t f = 4 * n + 64;
        if (f > rec->cap) f = rec->cap;
        if (9 * f <= kPackMax) {
            rec->fetched = f;
            rec->at = align16(packed);
            bytes = rec->at + 9 * f;
        }
    }
    return bytes ? ensure_pinned(ws.pin_out, bytes) : DYG_OK;
}

dyg_status check_params(const dyg_walk_params *p) {
    if (!p) {
        set_error("walk params are NULL");
        return DYG_EINVAL;
    }
    if (p->walkers == 0 || p->walkers % 32 != 0 || p->walkers > 1024) {
        set_error("walkers must be a positive multiple of 32 and <= 1024");
        return DYG_EINVAL;
    }
    if (p->max_steps < 1 || p->max_steps > 0x3FFFFF) {
        set_error("max_steps must be in [1, 4194303]");
        return DYG_EINVAL;
    }
    if (p->transition > DYG_TRANSITION_WEIGHTED) {
        set_error("unknown transition rule");
        return DYG_EINVAL;
    }
    if (p->heuristic_walkers > 1024) {
        set_error("heuristic_walkers must be <= 1024");
        return DYG_EINVAL;
    }
    return DYG_OK;
}

dyg_status check_ids(const uint32_t *v, size_t n, uint32_t nv, const char *what) {
    for (size_t i = 0; i < n; ++i)
        if (v[i] >= nv) {
            set_error(std::string(what) + "[" + std::to_string(i) + "] = " + std::to_string(v[i]) +
                      " is not a vertex (n = " + std::to_string(nv) + ")");
            return DYG_EINVAL;
        }
    return DYG_OK;
}

dyg_status check_weights(const float *w, size_t n) {
    for (size_t i = 0; i < n; ++i)
        if (!(w[i] > 0.0f) || !isfinite(w[i])) {
            set_error("weight[" + std::to_string(i) + "] is not finite and > 0");
            return DYG_EINVAL;
        }
    return DYG_OK;
}

dyg_status check_host_ids(const uint32_t *v, size_t n, uint32_t nv, const char *what) {
    return !v || on_device(v) ? DYG_OK : check_ids(v, n, nv, what);
}

dyg_status check_host_weights(const float *w, size_t n) {
    return !w || on_device(w) ? DYG_OK : check_weights(w, n);
}

// Host batches up to this size are checked on the host (the message names
// the entry); larger ones are staged first and checked by k_validate on the
// device, like device batches, instead of by a serial host loop.
constexpr uint32_t kHostCheckMax = 65536;

dyg_status check_device_errors(dyg_graph *G, cudaStream_t st) {
    DYG_TRY(read_scalars(G, st));
    const unsigned long long err = G->ws.host_scalars[S_ERR];
    if (err) {
        unsigned long long zero = 0;
        DYG_CUDA(cudaMemcpy(ptr<unsigned long long>(G->ws.scalars) + S_ERR, &zero, sizeof(zero),
                            cudaMemcpyHostToDevice));
        if (err & kErrVertex) {
            set_error("a batch endpoint is not a vertex of the graph");
            return DYG_EINVAL;
        }
        if (err & kErrWeight) {
            set_error("a batch weight is not finite and > 0");
            return DYG_EINVAL;
        }
        if (err & kErrScan) {
            set_error("a prefix scan tile timed out waiting for its predecessor");
            return DYG_ESTATE;
        }
        set_error("internal consistency check failed (device error bits " + std::to_string(err) + ")");
        return DYG_ESTATE;
    }
    return DYG_OK;
}

dyg_status graph_alloc_scalars(dyg_graph *G) {
    // counts follow the scalars, on the device and in the pinned mirror, so
    // that one copy reads both
    DYG_TRY(ensure(G->ws.scalars, kScalarBytes));
    DYG_CUDA(cudaMemset(G->ws.scalars.p, 0, kScalarBytes));
    G->ws.counts.p = ptr<unsigned long long>(G->ws.scalars) + S_NSCALARS;
    DYG_CUDA(host_alloc((void **)&G->ws.host_scalars, kScalarPinned));
    G->ws.host_counts = reinterpret_cast<uint32_t *>(G->ws.host_scalars + S_NSCALARS);
    G->g.top = ptr<unsigned long long>(G->ws.scalars) + S_TOP;
    G->counted = true;
    scratch_handles(G->device, 1);
    return DYG_OK;
}

void free_buf(Buf &b) {
    dev_free(b.p);
    b.p = nullptr;
    b.bytes = 0;
}

void free_graph(dyg_graph *G) {
    if (!G) return;
    DeviceGuard dg(G->device);
    cudaDeviceSynchronize();   // the blocks below may be handed out again at once
    if (G->counted) scratch_handles(G->device, -1);
    Workspace &ws = G->ws;
    Buf *bufs[] = {&ws.keys, &ws.flags, &ws.pos, &ws.f_src, &ws.f_dst, &ws.f_idx, &ws.f_uid,
                   &ws.f_w, &ws.found, &ws.path_v, &ws.path_s, &ws.path_len, &ws.rec_head, &ws.cand_x, &ws.cand_y,
                   &ws.cand_w, &ws.keep, &ws.htab_k, &ws.htab_v, &ws.scan_status,
                   &ws.s_src, &ws.s_dst, &ws.s_w, &ws.s_o1, &ws.s_o2, &ws.s_o3, &ws.rx2, &ws.ry2,
                   &ws.rk2, &ws.nxt, &ws.runs, &ws.rowcnt, &ws.rowhead, &ws.rowlist, &ws.blk, &ws.st_key,
                   &ws.st_cnt, &ws.st_val, &ws.st_pos, &ws.st_wapp, &ws.big, &ws.s_uid, &ws.scalars, &ws.io_in, &ws.io_out};
    for (Buf *b : bufs) free_buf(*b);
    host_free(ws.host_scalars, kScalarPinned);
    host_free(ws.pin_in.p, ws.pin_in.bytes);
    host_free(ws.pin_out.p, ws.pin_out.bytes);
    dev_free(G->g.desc);
    dev_free(G->g.cap);
    dev_free(G->g.slots);
    dev_free(G->g.wts);
    cudaGetLastError();
    delete G;
}

}  // namespace

dyg_status check_walk_params(const dyg_walk_params *p) { return check_params(p); }

dyg_status create_empty_graph(uint32_t n, uint64_t arena_slots, int device, uint32_t slack,
                              double headroom, dyg_graph **out) {
    *out = nullptr;
    if (arena_slots < 1024) arena_slots = 1024;
    if (arena_slots >= 0xFFFFFFFFull) {
        set_error("arena would exceed 32-bit slot offsets");
        return DYG_EINVAL;
    }
    DeviceGuard dg(device);
    dyg_graph *G = new dyg_graph();
    G->device = device;
    G->slack = slack;
    G->headroom = headroom;
    G->g.n = n;
    G->g.arena_cap = arena_slots;
    dyg_status rc = graph_alloc_scalars(G);
    if (rc == DYG_OK &&
        (dev_alloc(&G->g.desc, sizeof(uint2) * (size_t)(n ? n : 1)) != cudaSuccess ||
         dev_alloc(&G->g.cap, sizeof(uint32_t) * (size_t)(n ? n : 1)) != cudaSuccess ||
         dev_alloc(&G->g.slots, sizeof(uint2) * (size_t)arena_slots) != cudaSuccess ||
         dev_alloc(&G->g.wts, sizeof(float) * (size_t)arena_slots) != cudaSuccess)) {
        cudaGetLastError();
        set_error("cudaMalloc of a pool graph failed");
        rc = DYG_ENOMEM;
    }
    if (rc == DYG_OK && (cudaMemset(G->g.desc, 0, sizeof(uint2) * (size_t)(n ? n : 1)) != cudaSuccess ||
                         cudaMemset(G->g.cap, 0, sizeof(uint32_t) * (size_t)(n ? n : 1)) != cudaSuccess))
        rc = cuda_fail(cudaGetLastError(), "cudaMemset", __FILE__, __LINE__);
    // the first call on the graph may come on a stream that the default one
    // does not wait for
    if (rc == DYG_OK && cudaDeviceSynchronize() != cudaSuccess)
        rc = cuda_fail(cudaGetLastError(), "cudaDeviceSynchronize", __FILE__, __LINE__);
    if (rc != DYG_OK) {
        free_graph(G);
        return rc;
    }
    *out = G;
    return DYG_OK;
}

void destroy_graph(dyg_graph *G) {
    if (!G) return;
    {
        DeviceGuard dg(G->device);
        cudaDeviceSynchronize();
    }
    free_graph(G);
}

dyg_status device_errors(dyg_graph *G, cudaStream_t st) {
    return G->ws.host_scalars[S_ERR] ? check_device_errors(G, st) : DYG_OK;
}

}  // namespace dyg

using namespace dyg;

// ======================================================================= ABI

extern "C" {

const char *dyg_version(void) { return "dygrass_b200 0.1.0 (sm_100a)"; }

const char *dyg_last_error_string(void) { return g_last_error.c_str(); }

void dyg_walk_params_default(dyg_walk_params *p) {
    if (!p) return;
    p->threshold = 100.0f;
    p->walkers = 512;
    p->max_steps = 100;
    p->transition = DYG_TRANSITION_UNIFORM;
    p->heuristic_walkers = 16;
    p->flags = 0;
    p->seed = 20251203ull;
}

void dyg_graph_opts_default(dyg_graph_opts *o) {
    if (!o) return;
    o->slack_per_row = 2;
    o->reserved = 0;
    o->arena_headroom = 0.5;
    o->device = -1;
    o->pad = 0;
}

uint32_t dyg_reference_batch_size(uint32_t n) {
    const uint32_t b = (uint32_t)(((uint64_t)n + 9u) / 10u);
    return b ? b : 1u;
}

dyg_status dyg_graph_create_from_edges(uint32_t n_vertices, uint64_t n_edges, const uint32_t *src,
                                       const uint32_t *dst, const float *w,
                                       const dyg_graph_opts *opts, dyg_graph **out) {
    set_error("");
    if (!out || (n_edges && (!src || !dst || !w))) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    *out = nullptr;
    if (n_edges > 0x7FFFFFFFull) {
        set_error("too many edges");
        return DYG_EINVAL;
    }
    // like a batch's, long lists are checked on the device, as they are read
    if (n_edges <= kHostCheckMax) {
        DYG_TRY(check_ids(src, n_edges, n_vertices, "src"));
        DYG_TRY(check_ids(dst, n_edges, n_vertices, "dst"));
        DYG_TRY(check_weights(w, n_edges));
    }
    dyg_graph_opts o;
    dyg_graph_opts_default(&o);
    if (opts) o = *opts;
    int dev = o.device;
    if (dev < 0) DYG_CUDA(cudaGetDevice(&dev));
    DeviceGuard dg(dev);
    dyg_graph *G = new dyg_graph();
    G->device = dev;
    G->slack = o.slack_per_row;
    G->headroom = o.arena_headroom > 0 ? o.arena_headroom : 0.0;
    dyg_status rc = graph_alloc_scalars(G);
    bool bad = false;
    if (rc == DYG_OK) rc = build_graph(G, n_vertices, n_edges, src, dst, w, &bad);
    if (rc != DYG_OK) free_graph(G);
    if (bad) {
        // the message names the first entry that failed the device's check
        DYG_TRY(check_ids(src, n_edges, n_vertices, "src"));
        DYG_TRY(check_ids(dst, n_edges, n_vertices, "dst"));
        DYG_TRY(check_weights(w, n_edges));
        set_error("an edge is not valid");
    }
    if (rc != DYG_OK) return rc;
    *out = G;
    return DYG_OK;
}

dyg_status dyg_graph_create_from_csr(uint32_t n_vertices, const uint64_t *row_ptr,
                                     const uint32_t *col, const float *w,
                                     const dyg_graph_opts *opts, dyg_graph **out) {
    set_error("");
    if (!out || !row_ptr) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    *out = nullptr;
    const uint64_t m = row_ptr[n_vertices];
    if (m && (!col || !w)) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    if (row_ptr[0] != 0 || m > 0xFFFFFFFFull) {
        set_error("row_ptr must start at 0 and hold at most 2^32 - 1 slots");
        return DYG_EINVAL;
    }
    for (uint32_t v = 0; v < n_vertices; ++v)
        if (row_ptr[v + 1] < row_ptr[v]) {
            set_error("row_ptr must be non-decreasing");
            return DYG_EINVAL;
        }
    DYG_TRY(check_host_ids(col, m, n_vertices, "col"));
    DYG_TRY(check_host_weights(w, m));
    dyg_graph_opts o;
    dyg_graph_opts_default(&o);
    if (opts) o = *opts;
    int dev = o.device;
    if (dev < 0) DYG_CUDA(cudaGetDevice(&dev));
    DeviceGuard dg(dev);
    dyg_graph *G = new dyg_graph();
    G->device = dev;
    G->slack = o.slack_per_row;
    G->headroom = o.arena_headroom > 0 ? o.arena_headroom : 0.0;
    dyg_status rc = graph_alloc_scalars(G);
    if (rc == DYG_OK) rc = upload_graph(G, n_vertices, row_ptr, col, w);
    if (rc != DYG_OK) {
        free_graph(G);
        return rc;
    }
    *out = G;
    return DYG_OK;
}

dyg_status dyg_graph_copy_from(dyg_graph *dst, const dyg_graph *src, dyg_stream_t stream) {
    set_error("");
    if (!dst || !src || dst->g.n != src->g.n || dst->device != src->device) {
        set_error("copy_from needs two graphs with the same vertex count on one device");
        return DYG_EINVAL;
    }
    DeviceGuard dg(dst->device);
    cudaStream_t st = (cudaStream_t)stream;
    if (dst->g.arena_cap < src->g.arena_cap) {
        // the host needs src's top only when dst's arena might not hold it
        dyg_graph *s = const_cast<dyg_graph *>(src);
        DYG_TRY(read_scalars(s, st));
        if (dst->g.arena_cap < s->ws.host_scalars[S_TOP]) {
            uint2 *ns = nullptr;
            float *nw = nullptr;
            if (dev_alloc(&ns, sizeof(uint2) * (size_t)src->g.arena_cap) != cudaSuccess ||
                dev_alloc(&nw, sizeof(float) * (size_t)src->g.arena_cap) != cudaSuccess) {
                cudaGetLastError();
                if (ns) dev_free(ns);
                set_error("cudaMalloc in copy_from failed");
                return DYG_ENOMEM;
            }
            DYG_CUDA(cudaDeviceSynchronize());
            dev_free(dst->g.slots);
            dev_free(dst->g.wts);
            dst->g.slots = ns;
            dst->g.wts = nw;
            dst->g.arena_cap = src->g.arena_cap;
        }
    }
    if (dst != src) DYG_TRY(copy_graph_enqueue(dst, src, st));
    dst->slack = src->slack;
    dst->headroom = src->headroom;
    dst->long_rows = src->long_rows;
    dst->broken = src->broken;
    return DYG_OK;
}

dyg_status dyg_graph_clone(const dyg_graph *g, dyg_graph **out) {
    set_error("");
    if (!g || !out) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    DeviceGuard dg(g->device);
    dyg_graph *G = new dyg_graph();
    G->device = g->device;
    G->slack = g->slack;
    G->headroom = g->headroom;
    G->g.n = g->g.n;
    G->g.arena_cap = g->g.arena_cap;
    dyg_status rc = graph_alloc_scalars(G);
    if (rc == DYG_OK &&
        (dev_alloc(&G->g.desc, sizeof(uint2) * (size_t)(g->g.n ? g->g.n : 1)) != cudaSuccess ||
         dev_alloc(&G->g.cap, sizeof(uint32_t) * (size_t)(g->g.n ? g->g.n : 1)) != cudaSuccess ||
         dev_alloc(&G->g.slots, sizeof(uint2) * (size_t)g->g.arena_cap) != cudaSuccess ||
         dev_alloc(&G->g.wts, sizeof(float) * (size_t)g->g.arena_cap) != cudaSuccess)) {
        cudaGetLastError();
        set_error("cudaMalloc in clone failed");
        rc = DYG_ENOMEM;
    }
    if (rc == DYG_OK) rc = dyg_graph_copy_from(G, g, nullptr);
    if (rc == DYG_OK && cudaDeviceSynchronize() != cudaSuccess) rc = cuda_fail(cudaGetLastError(), "clone", __FILE__, __LINE__);
    if (rc != DYG_OK) {
        free_graph(G);
        return rc;
    }
    *out = G;
    return DYG_OK;
}

dyg_status dyg_graph_destroy(dyg_graph *g) {
    if (!g) return DYG_OK;
    {
        DeviceGuard dg(g->device);
        cudaDeviceSynchronize();
    }
    free_graph(g);
    return DYG_OK;
}

dyg_status dyg_graph_info(const dyg_graph *g, uint32_t *n_vertices, uint64_t *n_slots,
                          uint64_t *arena_used, uint64_t *arena_cap) {
    set_error("");
    if (!g) {
        set_error("NULL graph");
        return DYG_EINVAL;
    }
    DeviceGuard dg(g->device);
    dyg_graph *G = const_cast<dyg_graph *>(g);
    if (n_slots) DYG_TRY(count_slots_enqueue(G, nullptr));
    DYG_TRY(read_scalars(G, nullptr));
    if (n_vertices) *n_vertices = g->g.n;
    if (arena_used) *arena_used = G->ws.host_scalars[S_TOP];
    if (arena_cap) *arena_cap = g->g.arena_cap;
    if (n_slots) *n_slots = G->ws.host_scalars[S_SLOTS];
    return DYG_OK;
}

dyg_status dyg_graph_export(dyg_graph *g, uint64_t *row_ptr, uint32_t *col, float *w,
                            uint64_t slot_cap) {
    set_error("");
    if (!g || !row_ptr) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    DeviceGuard dg(g->device);
    DYG_CUDA(cudaDeviceSynchronize());
    DYG_TRY(export_graph(g, row_ptr, col, w, slot_cap));
    if (row_ptr[g->g.n] > slot_cap) {
        set_error("slot_cap smaller than the number of slots");
        return DYG_ERANGE;
    }
    return DYG_OK;
}

dyg_status dyg_graph_compact(dyg_graph *g, dyg_stream_t stream) {
    set_error("");
    if (!g) {
        set_error("NULL graph");
        return DYG_EINVAL;
    }
    DeviceGuard dg(g->device);
    return compact_graph(g, (cudaStream_t)stream);
}

dyg_status dyg_graph_counters(const dyg_graph *g, uint64_t *walker_moves, uint64_t *walks) {
    set_error("");
    if (!g) {
        set_error("NULL graph");
        return DYG_EINVAL;
    }
    DeviceGuard dg(g->device);
    dyg_graph *G = const_cast<dyg_graph *>(g);
    DYG_CUDA(cudaDeviceSynchronize());
    DYG_TRY(read_scalars(G, nullptr));
    if (walker_moves) *walker_moves = G->ws.host_scalars[S_MOVES];
    if (walks) *walks = G->ws.host_scalars[S_WALKS];
    return DYG_OK;
}

static dyg_status incremental_common(dyg_graph *H, dyg_graph *G, const uint32_t *src,
                                     const uint32_t *dst, const float *w, uint32_t n,
                                     uint32_t batch_size, uint64_t uid_base, const uint64_t *uids,
                                     const dyg_walk_params *p, int32_t *found_at,
                                     float *conductance, uint8_t *accepted, dyg_stream_t stream) {
    set_error("");
    if (!H || (n && (!src || !dst || !w))) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    DYG_TRY(check_params(p));
    if (G && (G == H || G->g.n != H->g.n || G->device != H->device)) {
        set_error("G and H must be two handles with the same vertex count and device");
        return DYG_EINVAL;
    }
    if (n == 0) return DYG_OK;
    DeviceGuard dg(H->device);
    cudaStream_t st = (cudaStream_t)stream;
    Workspace &ws = H->ws;
    InArray in[] = {{"src", src, sizeof(uint32_t) * (size_t)n, &ws.s_src},
                    {"dst", dst, sizeof(uint32_t) * (size_t)n, &ws.s_dst},
                    {"w", w, sizeof(float) * (size_t)n, &ws.s_w},
                    {"update_ids", uids, sizeof(uint64_t) * (size_t)n, &ws.s_uid}};
    OutArray out[] = {{"found_at", found_at, found_at ? sizeof(int32_t) * (size_t)n : 0, &ws.s_o1},
                      {"conductance", conductance, conductance ? sizeof(float) * (size_t)n : 0, &ws.s_o2},
                      {"accepted", accepted, accepted ? (size_t)n : 0, &ws.s_o3}};
    DYG_TRY(check_places(H->device, in, 4, out, 3));
    const bool host_check = n <= kHostCheckMax;
    if (host_check) {
        if (in[0].host) DYG_TRY(check_ids(src, n, H->g.n, "src"));
        if (in[1].host) DYG_TRY(check_ids(dst, n, H->g.n, "dst"));
        if (in[2].host) DYG_TRY(check_weights(w, n));
    }
    size_t packed = 0;
    DYG_TRY(stage_inputs(ws, in, 4, st));
    DYG_TRY(place_outputs(ws, out, 3, &packed));
    if (!any_host(out, 3)) packed = 0;
    DYG_TRY(prepare_fetch(ws, packed, nullptr, n));
    const std::function<dyg_status()> fetch = [&]() -> dyg_status {
        if (packed) DYG_CUDA(cudaMemcpyAsync(ws.pin_out.p, ws.io_out.p, packed, cudaMemcpyDeviceToHost, st));
        return DYG_OK;
    };
    const uint32_t B = batch_size ? batch_size : dyg_reference_batch_size(n);
    // inputs read in place from device memory were not checked on the host
    const bool dev_in = !host_check || !in[0].host || !in[1].host || !in[2].host;
    DYG_TRY(incremental_run(H, G, (const uint32_t *)in[0].dev, (const uint32_t *)in[1].dev,
                            (const float *)in[2].dev, n, B, uid_base,
                            (const unsigned long long *)in[3].dev, *p, (int32_t *)out[0].dev,
                            (float *)out[1].dev, (uint8_t *)out[2].dev, st, dev_in, nullptr, &fetch));
    if (H->ws.host_scalars[S_ERR]) DYG_TRY(check_device_errors(H, st));
    bool wait = false;
    DYG_TRY(deliver(ws, out, 3, packed, st, &wait));
    if (wait) DYG_CUDA(cudaStreamSynchronize(st));
    return DYG_OK;
}

dyg_status dyg_incremental_batch(dyg_graph *H, dyg_graph *G, const uint32_t *src,
                                 const uint32_t *dst, const float *w, uint32_t n,
                                 uint64_t first_update_id, const dyg_walk_params *p,
                                 int32_t *found_at, float *conductance, uint8_t *accepted,
                                 dyg_stream_t stream) {
    return incremental_common(H, G, src, dst, w, n, n ? n : 1, first_update_id, nullptr, p,
                              found_at, conductance, accepted, stream);
}

dyg_status dyg_incremental_stream(dyg_graph *H, dyg_graph *G, const uint32_t *src,
                                  const uint32_t *dst, const float *w, uint32_t n,
                                  uint32_t batch_size, const dyg_walk_params *p,
                                  int32_t *found_at, float *conductance, uint8_t *accepted,
                                  dyg_stream_t stream) {
    return incremental_common(H, G, src, dst, w, n, batch_size, 0, nullptr, p, found_at,
                              conductance, accepted, stream);
}

static dyg_status decremental_common(dyg_graph *G, dyg_graph *H, const uint32_t *src,
                                     const uint32_t *dst, uint32_t n, uint32_t batch_size,
                                     uint64_t uid_base, const uint64_t *uids,
                                     const dyg_walk_params *p, int32_t *status,
                                     float *conductance, uint32_t *rec_src, uint32_t *rec_dst,
                                     uint8_t *rec_kind, uint64_t rec_cap, uint64_t *n_rec,
                                     dyg_stream_t stream) {
    set_error("");
    if (!G || !H || (n && (!src || !dst))) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    DYG_TRY(check_params(p));
    if (G == H || G->g.n != H->g.n || G->device != H->device) {
        set_error("G and H must be two handles with the same vertex count and device");
        return DYG_EINVAL;
    }
    if (n_rec) *n_rec = 0;
    if (n == 0) return DYG_OK;
    DeviceGuard dg(G->device);
    cudaStream_t st = (cudaStream_t)stream;
    Workspace &ws = G->ws;
    InArray in[] = {{"src", src, sizeof(uint32_t) * (size_t)n, &ws.s_src},
                    {"dst", dst, sizeof(uint32_t) * (size_t)n, &ws.s_dst},
                    {"update_ids", uids, sizeof(uint64_t) * (size_t)n, &ws.s_uid}};
    // statuses and conductances are needed on the device even if not asked for
    OutArray out[] = {{"status", status, sizeof(int32_t) * (size_t)n, &ws.s_o1},
                      {"conductance", conductance, sizeof(float) * (size_t)n, &ws.s_o2}};
    OutArray recs[] = {{"rec_src", rec_src, 0, nullptr},
                       {"rec_dst", rec_dst, 0, nullptr},
                       {"rec_kind", rec_kind, 0, nullptr}};
    DYG_TRY(check_places(G->device, in, 3, out, 2));
    DYG_TRY(check_places(G->device, nullptr, 0, recs, 3));
    const bool host_check = n <= kHostCheckMax;
    if (host_check) {
        if (in[0].host) DYG_TRY(check_ids(src, n, G->g.n, "src"));
        if (in[1].host) DYG_TRY(check_ids(dst, n, G->g.n, "dst"));
    }
    RecordsOut rec{rec_src, rec_dst, rec_kind, rec_cap,
                   (!rec_src || recs[0].host) && (!rec_dst || recs[1].host) && (!rec_kind || recs[2].host),
                   any_host(recs, 3)};
    size_t packed = 0;
    DYG_TRY(stage_inputs(ws, in, 3, st));
    DYG_TRY(place_outputs(ws, out, 2, &packed));
    if (!any_host(out, 2)) packed = 0;
    DYG_TRY(prepare_fetch(ws, packed, &rec, n));
    const std::function<dyg_status()> fetch = [&]() -> dyg_status {
        if (packed) DYG_CUDA(cudaMemcpyAsync(ws.pin_out.p, ws.io_out.p, packed, cudaMemcpyDeviceToHost, st));
        return rec.fetch(ws, st);
    };
    const uint32_t B = batch_size ? batch_size : dyg_reference_batch_size(n);
    uint64_t total = 0;
    const bool dev_in = !host_check || !in[0].host || !in[1].host;
    G->last_rec = 0;
    DYG_TRY(decremental_run(G, H, (const uint32_t *)in[0].dev, (const uint32_t *)in[1].dev, n, B,
                            uid_base, (const unsigned long long *)in[2].dev, *p, (int32_t *)out[0].dev,
                            (float *)out[1].dev, &total, st, dev_in, nullptr, &fetch));
    G->last_rec = total;
    if (G->ws.host_scalars[S_ERR]) DYG_TRY(check_device_errors(G, st));
    bool wait = false;
    DYG_TRY(deliver(ws, out, 2, packed, st, &wait));
    DYG_TRY(rec.deliver(ws, total, st, &wait));
    if (wait) DYG_CUDA(cudaStreamSynchronize(st));
    if (n_rec) *n_rec = total;
    if (total > rec_cap && (rec_src || rec_dst || rec_kind)) {
        set_error("more recovered edges than rec_cap");
        return DYG_ERANGE;
    }
    return DYG_OK;
}

dyg_status dyg_decremental_batch(dyg_graph *G, dyg_graph *H, const uint32_t *src,
                                 const uint32_t *dst, uint32_t n, uint64_t first_update_id,
                                 const dyg_walk_params *p, int32_t *status, float *conductance,
                                 uint32_t *rec_src, uint32_t *rec_dst, uint8_t *rec_kind,
                                 uint64_t rec_cap, uint64_t *n_rec, dyg_stream_t stream) {
    return decremental_common(G, H, src, dst, n, n ? n : 1, first_update_id, nullptr, p, status,
                              conductance, rec_src, rec_dst, rec_kind, rec_cap, n_rec, stream);
}

dyg_status dyg_decremental_stream(dyg_graph *G, dyg_graph *H, const uint32_t *src,
                                  const uint32_t *dst, uint32_t n, uint32_t batch_size,
                                  const dyg_walk_params *p, int32_t *status, float *conductance,
                                  uint32_t *rec_src, uint32_t *rec_dst, uint8_t *rec_kind,
                                  uint64_t rec_cap, uint64_t *n_rec, dyg_stream_t stream) {
    return decremental_common(G, H, src, dst, n, batch_size, 0, nullptr, p, status, conductance,
                              rec_src, rec_dst, rec_kind, rec_cap, n_rec, stream);
}

dyg_status dyg_incremental_batch_ids(dyg_graph *H, dyg_graph *G, const uint32_t *src,
                                     const uint32_t *dst, const float *w,
                                     const uint64_t *update_ids, uint32_t n,
                                     const dyg_walk_params *p, int32_t *found_at,
                                     float *conductance, uint8_t *accepted, dyg_stream_t stream) {
    if (n && !update_ids) {
        set_error("NULL update_ids");
        return DYG_EINVAL;
    }
    return incremental_common(H, G, src, dst, w, n, n ? n : 1, 0, update_ids, p, found_at,
                              conductance, accepted, stream);
}

dyg_status dyg_decremental_batch_ids(dyg_graph *G, dyg_graph *H, const uint32_t *src,
                                     const uint32_t *dst, const uint64_t *update_ids, uint32_t n,
                                     const dyg_walk_params *p, int32_t *status,
                                     float *conductance, uint32_t *rec_src, uint32_t *rec_dst,
                                     uint8_t *rec_kind, uint64_t rec_cap, uint64_t *n_rec,
                                     dyg_stream_t stream) {
    if (n && !update_ids) {
        set_error("NULL update_ids");
        return DYG_EINVAL;
    }
    return decremental_common(G, H, src, dst, n, n ? n : 1, 0, update_ids, p, status, conductance,
                              rec_src, rec_dst, rec_kind, rec_cap, n_rec, stream);
}

dyg_status dyg_recovered_read(const dyg_graph *g, uint64_t first, uint64_t count,
                              uint32_t *rec_src, uint32_t *rec_dst, uint8_t *rec_kind) {
    set_error("");
    if (!g) {
        set_error("NULL graph");
        return DYG_EINVAL;
    }
    if (first > g->last_rec || count > g->last_rec - first) {
        set_error("records [" + std::to_string(first) + ", " + std::to_string(first + count) +
                  ") are not all among the last call's " + std::to_string(g->last_rec));
        return DYG_ERANGE;
    }
    if (count == 0) return DYG_OK;
    DeviceGuard dg(g->device);
    const Workspace &ws = g->ws;
    const void *ps[] = {rec_src, rec_dst, rec_kind};
    const char *nm[] = {"rec_src", "rec_dst", "rec_kind"};
    DYG_TRY(check_same_device(g->device, ps, nm, 3));
    if (rec_src)
        DYG_CUDA(cudaMemcpy(rec_src, ptr<uint32_t>(ws.rx2) + first, sizeof(uint32_t) * count,
                            cudaMemcpyDefault));
    if (rec_dst)
        DYG_CUDA(cudaMemcpy(rec_dst, ptr<uint32_t>(ws.ry2) + first, sizeof(uint32_t) * count,
                            cudaMemcpyDefault));
    if (rec_kind)
        DYG_CUDA(cudaMemcpy(rec_kind, ptr<uint8_t>(ws.rk2) + first, count, cudaMemcpyDefault));
    return DYG_OK;
}

uint32_t dyg_stream_default_chunk(uint32_t n_vertices) {
    return stream_default_chunk(n_vertices);
}

dyg_status dyg_stream_file(dyg_graph *G, dyg_graph *H, uint32_t op, const uint32_t *src,
                           const uint32_t *dst, const float *w, uint32_t n,
                           uint64_t first_update_id, uint32_t chunk, const dyg_walk_params *p,
                           int32_t *status, float *conductance, uint32_t *rec_src,
                           uint32_t *rec_dst, uint8_t *rec_kind, uint64_t rec_cap,
                           uint64_t *n_rec, dyg_stream_t stream) {
    set_error("");
    const bool ins = op == DYG_STREAM_INSERT;
    if (!G || !H || (n && (!src || !dst || (ins && !w)))) {
        set_error("NULL argument");
        return DYG_EINVAL;
    }
    if (op != DYG_STREAM_INSERT && op != DYG_STREAM_DELETE) {
        set_error("op must be DYG_STREAM_INSERT or DYG_STREAM_DELETE");
        return DYG_EINVAL;
    }
    DYG_TRY(check_params(p));
    if (G == H || G->g.n != H->g.n || G->device != H->device) {
        set_error("G and H must be two handles with the same vertex count and device");
        return DYG_EINVAL;
    }
    if (n_rec) *n_rec = 0;
    if (n == 0) return DYG_OK;
    DeviceGuard dg(G->device);
    cudaStream_t st = (cudaStream_t)stream;
    Workspace &ws = G->ws;
    InArray in[] = {{"src", src, sizeof(uint32_t) * (size_t)n, &ws.s_src},
                    {"dst", dst, sizeof(uint32_t) * (size_t)n, &ws.s_dst},
                    {"w", w, sizeof(float) * (size_t)n, &ws.s_w}};
    // statuses and conductances are needed on the device even if not asked for
    OutArray out[] = {{"status", status, sizeof(int32_t) * (size_t)n, &ws.s_o1},
                      {"conductance", conductance, sizeof(float) * (size_t)n, &ws.s_o2}};
    OutArray recs[] = {{"rec_src", rec_src, 0, nullptr},
                       {"rec_dst", rec_dst, 0, nullptr},
                       {"rec_kind", rec_kind, 0, nullptr}};
    // a deletion file's weights are not read, an insertion file has no records
    const int nin = ins ? 3 : 2;
    DYG_TRY(check_places(G->device, in, 3, out, 2));
    DYG_TRY(check_places(G->device, nullptr, 0, recs, 3));
    const bool host_check = n <= kHostCheckMax;
    if (host_check) {
        if (in[0].host) DYG_TRY(check_ids(src, n, G->g.n, "src"));
        if (in[1].host) DYG_TRY(check_ids(dst, n, G->g.n, "dst"));
        if (ins && in[2].host) DYG_TRY(check_weights(w, n));
    }
    RecordsOut rec{rec_src, rec_dst, rec_kind, rec_cap,
                   (!rec_src || recs[0].host) && (!rec_dst || recs[1].host) && (!rec_kind || recs[2].host),
                   any_host(recs, 3)};
    size_t packed = 0;
    DYG_TRY(stage_inputs(ws, in, nin, st));
    DYG_TRY(place_outputs(ws, out, 2, &packed));
    if (!any_host(out, 2)) packed = 0;
    DYG_TRY(prepare_fetch(ws, packed, ins ? nullptr : &rec, n));
    const std::function<dyg_status()> fetch = [&]() -> dyg_status {
        if (packed) DYG_CUDA(cudaMemcpyAsync(ws.pin_out.p, ws.io_out.p, packed, cudaMemcpyDeviceToHost, st));
        return rec.fetch(ws, st);
    };
    uint64_t total = 0;
    const bool dev_in = !host_check || !in[0].host || !in[1].host || (ins && !in[2].host);
    if (!ins) G->last_rec = 0;
    DYG_TRY(stream_file_run(G, H, op, (const uint32_t *)in[0].dev, (const uint32_t *)in[1].dev,
                            ins ? (const float *)in[2].dev : nullptr, n, first_update_id, chunk, *p,
                            (int32_t *)out[0].dev, (float *)out[1].dev, &total, st, dev_in, &fetch));
    if (!ins) G->last_rec = total;
    if (G->ws.host_scalars[S_ERR]) DYG_TRY(check_device_errors(G, st));
    if (H->ws.host_scalars[S_ERR]) DYG_TRY(check_device_errors(H, st));
    bool wait = false;
    DYG_TRY(deliver(ws, out, 2, packed, st, &wait));
    if (!ins) DYG_TRY(rec.deliver(ws, total, st, &wait));
    if (wait) DYG_CUDA(cudaStreamSynchronize(st));
    if (n_rec) *n_rec = total;
    if (total > rec_cap && (rec_src || rec_dst || rec_kind)) {
        set_error("more recovered edges than rec_cap");
        return DYG_ERANGE;
    }
    return DYG_OK;
}

}  // extern "C"
