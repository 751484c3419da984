// gridsync.cuh -- barriers and ordered block ranges for the kernels that run
// a whole row update in one launch.
//
// A batch's commit is a chain of short passes, each needing the one before it
// to be complete.  As separate launches a pass of a few thousand entries
// costs 4-6 us, nearly all of it launch and drain; as phases of one launch
// separated by a barrier it costs the barrier and its own loads.  Measured on
// whole calls: 64 deletions with recovery, 24 launches -> 4, 301 -> 223 us;
// 1,000 insertions in ten batches 652 -> 424 us; 297,000 deletions of a 100^3
// mesh in ten batches 4.79 -> 3.82 ms.
//
// A list that one block holds needs no more than its own barrier.  Up to 16
// blocks are launched as one thread-block cluster, scheduled together by the
// hardware and meeting at its barrier: 10 us a launch less than a cooperative
// grid of as many blocks (the thirteen batches of 4,999 insertions and 7,777
// deletions on a 37 x 41 x 29 mesh: 1.58 -> 1.44 ms).  Larger grids are
// launched cooperatively; their barrier counts arrivals on one word and
// publishes a generation on another, both in the owning graph's scalars.  All
// blocks of such a grid are resident, so a waiting block's peers run; the wait
// is bounded all the same, and a block that gives up raises kErrBarrier, halts
// the call (every later launch of it returns at once) and leaves.  What the
// kernel was doing stays half done: read_scalars2 reports it as DYG_ESTATE and
// marks the graphs (see recover_workspace).
//
// A block may give up while others of its grid go on to the next phase (the
// late arrival that it did not wait for opens the barrier), so the halt word
// can change under a running phase.  A kernel that asks whether *it* halted
// therefore compares the word with its own code; the word is only set when it
// is zero, so that such a code stays.
#pragma once

#include <atomic>

#include <type_traits>

#include "dyg_internal.cuh"

namespace dyg {

// Two blocks of this size an SM leave 64 registers a thread: k_append spills 24 to
// 36 bytes, k_recover 36, k_delete 8.
constexpr uint32_t kOpThreads = 512;

struct GridBar {
    uint32_t *count, *gen;
    unsigned long long *err, *halt;
    uint32_t limit;   // reads of the generation word before a block gives up
    bool cluster;     // the grid is one thread-block cluster
};

struct NoWork {
    __device__ void operator()() const {}
};

// Every thread of the cluster arrives and waits; writes made before are
// visible after, in global memory as well.  Not the .aligned forms: a phase
// ends in loops of different lengths and in branches of one thread, and
// nothing makes the lanes of a warp come back together before they get here.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// The last block to arrive runs `last` (one thread) before any block leaves.
// Writes made before the barrier by any thread of the grid are visible after
// it.  False: the wait ran out.  Every thread of every block calls it.
template <class F>
__device__ __forceinline__ bool grid_sync(const GridBar &b, F last) {
    __shared__ uint32_t s_ok;
    if (b.cluster) {
        cluster_sync();
        if (!std::is_same<F, NoWork>::value) {
            if (blockIdx.x == 0u && threadIdx.x == 0u) last();
            cluster_sync();
        }
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t ok = 1u;
        if (gridDim.x == 1u) {
            last();
        } else {
            volatile uint32_t *vg = b.gen;
            const uint32_t g = *vg;   // cannot advance before this block arrives
            __threadfence();
            if (atomicAdd(b.count, 1u) == gridDim.x - 1u) {
                __threadfence();
                last();
                *(volatile uint32_t *)b.count = 0u;
                __threadfence();
                atomicAdd(b.gen, 1u);
            } else {
                uint32_t spins = 0;
                while (*vg == g) {
                    if (++spins > 4096u) __nanosleep(256);
                    if (spins > b.limit) {
                        atomicOr(b.err, (unsigned long long)kErrBarrier);
                        atomicCAS(b.halt, 0ull, halt_code(0, (uint32_t)kHaltBroken, 0));
                        ok = 0u;
                        break;
                    }
                }
            }
            __threadfence();
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0u;
}
__device__ __forceinline__ bool grid_sync(const GridBar &b) {
    return grid_sync(b, NoWork{});
}

// This block's contiguous share of [0, m): whole warps, in block order, so
// that per-block counts scan to positions in list order.
__device__ __forceinline__ uint2 block_range(uint32_t m) {
    const uint32_t per = (uint32_t)(((uint64_t)m + gridDim.x - 1u) / gridDim.x + 31u) & ~31u;
    const uint64_t lo = (uint64_t)per * blockIdx.x;
    if (lo >= m) return make_uint2(m, m);
    return make_uint2((uint32_t)lo, (uint32_t)min((uint64_t)m, lo + per));
}

// Exclusive prefix of v over the block's threads; *total gets the sum.
// s_warp holds kOpThreads / 32 + 1 words.  Every thread calls it.
__device__ __forceinline__ uint32_t block_excl(uint32_t v, uint32_t *s_warp, uint32_t *total) {
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31u) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0u) {
        const uint32_t w = lane < nw ? s_warp[lane] : 0u;
        uint32_t x = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, x, o);
            if (lane >= (uint32_t)o) x += t;
        }
        if (lane < nw) s_warp[lane] = x - w;
        if (lane == nw - 1u) s_warp[nw] = x;
    }
    __syncthreads();
    const uint32_t r = s_warp[wid] + incl - v;
    *total = s_warp[nw];
    __syncthreads();   // s_warp may be written again
    return r;
}

// Sum of v over the block.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *s_warp) {
    uint32_t total;
    block_excl(v, s_warp, &total);
    return total;
}

// Sums of the per-block words vals[0, blockIdx.x) and vals[0, gridDim.x).
__device__ __forceinline__ uint2 blocks_before(const uint32_t *vals, uint32_t *s_warp) {
    uint32_t before = 0u, all = 0u;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
        const uint32_t v = __ldcg(vals + b);
        all += v;
        if (b < blockIdx.x) before += v;
    }
    const uint32_t x = block_sum(before, s_warp);
    return make_uint2(x, block_sum(all, s_warp));
}

// Most blocks of a one-launch kernel (the per-block words are sized for it).
constexpr uint32_t kOpBlocksMax = 1024;

// Most blocks of a grid that is launched as one cluster (16 needs the opt-in
// that launch_phases makes).
constexpr uint32_t kClusterMax = 16;

// Launches Kernel(args..., bar) with `want` blocks of kOpThreads: a single
// block as it is; up to kClusterMax blocks as one cluster, whose blocks are
// scheduled together and meet at the hardware's barrier; more of them
// cooperatively, no more than fit the device at once.
template <auto Kernel, class... A>
dyg_status launch_phases(uint32_t want, cudaStream_t st, GridBar bar, const A &...args) {
    count_launch();
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kOpThreads);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    cfg.attrs = &at;
    // the largest cluster of this kernel that the device can place, asked for
    // (and allowed, which a context keeps) once in each device's context
    constexpr int kDevs = 64;
    static std::atomic<unsigned long long> placed[kDevs];   // context, 1 + the size; 0: not asked yet
    uint32_t cluster_max = 0;
    int dev = -1;
    if (want > 1u && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kDevs) {
        const unsigned long long ctx = current_context_id() << 8;
        unsigned long long known = placed[dev].load(std::memory_order_acquire);
        if (!known || (known & ~0xFFull) != ctx) {
            cudaLaunchConfig_t c{};
            c.gridDim = dim3(kClusterMax);
            c.blockDim = dim3(kOpThreads);
            int most = 0;
            if (cudaFuncSetAttribute(Kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                cudaOccupancyMaxPotentialClusterSize(&most, Kernel, &c) != cudaSuccess || most < 0) {
                cudaGetLastError();
                most = 0;
            }
            known = ctx | (1u + (most < (int)kClusterMax ? (uint32_t)most : kClusterMax));
            placed[dev].store(known, std::memory_order_release);
        }
        cluster_max = (uint32_t)(known & 0xFFull) - 1u;
    }
    uint32_t k = 2u;
    while (k < want) k <<= 1;
    if (want <= 1u) {
        cfg.gridDim = dim3(1);
    } else if (k <= cluster_max) {
        cfg.gridDim = dim3(k);
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = k;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.numAttrs = 1;
        bar.cluster = true;
    } else {
        static const int per_sm = [] {
            int nb = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, Kernel, kOpThreads, 0);
            return nb < 1 ? 1 : nb;
        }();
        uint32_t fit = (uint32_t)per_sm * (uint32_t)num_sms();
        if (fit > kOpBlocksMax) fit = kOpBlocksMax;
        cfg.gridDim = dim3(want < fit ? want : fit);
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        cfg.numAttrs = 1;
    }
    DYG_CUDA(cudaLaunchKernelEx(&cfg, Kernel, args..., bar));
    return DYG_OK;
}

// Blocks for a list of m entries.  One entry per thread, but on a graph with
// hub rows the list is spread over every SM, a warp's worth of entries per
// block at least: a block rewrites its entries' hub rows one after another.
inline uint32_t op_blocks(uint64_t m, bool hubs) {
    uint64_t b = (m + kOpThreads - 1) / kOpThreads;
    if (hubs) {
        const uint64_t spread = (m + 31) / 32, sms = (uint64_t)num_sms();
        const uint64_t s = spread < sms ? spread : sms;
        if (b < s) b = s;
    }
    return b < 1 ? 1u : (b > kOpBlocksMax ? kOpBlocksMax : (uint32_t)b);
}

}  // namespace dyg
