// sort_common.cuh -- device-wide exclusive scan and per-bucket key sort shared
// by the drop-in intersection operator (isect.cu) and the fused multi-view
// render path (scene.cu).
#pragma once

#include <cooperative_groups.h>

#include "bucket_math.h"
#include "ubs_common.cuh"

namespace ubs {

constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_TILE = SCAN_ITEMS * SCAN_THREADS;
constexpr int WARP_SEG = 1024;  // longest bucket sorted by one warp in registers
constexpr int SMALL_SEG = 4096; // longest bucket sorted by one CTA in shared memory
constexpr int BIG_THREADS = 512;
constexpr int MERGE_ITEMS = 8;
constexpr int EMIT_ROUNDS = 4; // (entry, tile) rounds of 32 whose cursor atomics overlap

// ------------------------------------------------------------------- scan
// Exclusive scan of int32 counts.  Per block: SCAN_TILE items; block-local
// prefixes go to out, block totals to block_sums; a single block scans the
// totals, a last pass adds them.  OutT is int32_t or int64_t.
template <typename OutT>
__global__ void __launch_bounds__(SCAN_THREADS) scan_blocks_kernel(const int32_t *__restrict__ in,
                                                                  OutT *__restrict__ out,
                                                                  int64_t n,
                                                                  int64_t *__restrict__ sums) {
    __shared__ int64_t warp_tot[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)tid * SCAN_ITEMS;
    int64_t v[SCAN_ITEMS];
    int64_t run = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int64_t x = (base + k < n) ? (int64_t)in[base + k] : 0;
        v[k] = run;
        run += x;
    }
    // inclusive warp scan of thread totals
    int64_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int64_t w = warp_tot[lane];
        int64_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        warp_tot[lane] = wi - w; // exclusive
        if (lane == 31) sums[blockIdx.x] = wi;
    }
    __syncthreads();
    const int64_t off = warp_tot[warp] + (inc - run);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k)
        if (base + k < n) out[base + k] = scan_value<OutT>(v[k] + off);
}

static __global__ void __launch_bounds__(SCAN_THREADS) scan_sums_kernel(int64_t *sums, int64_t nblocks,
                                                                 int64_t *total) {
    __shared__ int64_t warp_tot[32];
    __shared__ int64_t carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int64_t base = 0; base < nblocks; base += SCAN_THREADS) {
        const int64_t i = base + tid;
        const int64_t x = i < nblocks ? sums[i] : 0;
        int64_t inc = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) warp_tot[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const int64_t w = warp_tot[lane];
            int64_t wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += y;
            }
            warp_tot[lane] = wi - w;
        }
        __syncthreads();
        const int64_t c0 = carry;
        if (i < nblocks) sums[i] = c0 + warp_tot[warp] + inc - x;
        __syncthreads();
        if (tid == SCAN_THREADS - 1) carry = c0 + warp_tot[warp] + inc;
        __syncthreads();
    }
    if (tid == 0) *total = carry;
}

template <typename OutT>
__global__ void scan_add_kernel(OutT *out, int64_t n, const int64_t *__restrict__ sums) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = scan_value<OutT>((int64_t)out[i] + sums[i / SCAN_TILE]);
}

template <typename OutT>
inline int device_exclusive_scan(const int32_t *in, OutT *out, int64_t n, int64_t *sums,
                                 int64_t *total, cudaStream_t st) {
    if (n == 0) {
        if (cudaMemsetAsync(total, 0, 8, st) != cudaSuccess) return check_launch("scan memset");
        return UBS_OK;
    }
    const int64_t nblocks = (n + SCAN_TILE - 1) / SCAN_TILE;
    UBS_TIMED("scan", st,
              scan_blocks_kernel<OutT><<<(unsigned)nblocks, SCAN_THREADS, 0, st>>>(in, out, n,
                                                                                  sums);
              scan_sums_kernel<<<1, SCAN_THREADS, 0, st>>>(sums, nblocks, total);
              if (nblocks > 1) scan_add_kernel<OutT><<<grid_for(n, 256), 256, 0, st>>>(out, n,
                                                                                       sums));
    ::ubs::note_launch(nblocks > 1 ? 3 : 2);
    return check_launch("exclusive scan");
}


// ------------------------------------------------------------ bucket sort
// Buckets hold unique 64-bit keys (depth bits << 32 | flatten index), so any
// correct sort yields the reference's stable order.  Writer::operator()(key,
// sorted position, bucket) stores one sorted entry.  The intersection count
// is read on the device when T_dev is given (clamped to the key capacity
// cap), else it is cap, so no host round trip is needed.

__device__ __forceinline__ void bucket_range(const int32_t *offsets, int64_t bkt, int64_t n_buckets,
                                             int64_t T, int64_t &lo, int64_t &hi) {
    bucket_bounds(offsets[bkt], bkt + 1 < n_buckets ? offsets[bkt + 1] : INT32_MAX, T, lo, hi);
}

// Warp-flattened emission of sort keys: every lane holds the tile rectangle
// of one (view, primitive) entry -- n tiles, bw columns, row pitch `pitch`,
// cursor of its first tile `cur` -- and the warp walks the concatenation of
// the 32 rectangles 32 (entry, tile) pairs per round, so its rounds follow the
// warp's total tile count rather than its largest entry and the cursor
// atomics of a round are independent.  Each pair takes the next slot of its
// tile's cursor and stores the entry's key there (slots past `cap` set the
// overflow bit instead).
__device__ __forceinline__ void warp_emit_rects(uint32_t n, uint32_t bw, uint32_t pitch,
                                                int32_t *cur, uint64_t key, int lane,
                                                uint64_t *__restrict__ keys, int64_t cap,
                                                uint32_t *status) {
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    // pair j of the flattened list: the cursor of its tile and its entry's key
    auto locate = [&](uint32_t j, int32_t *&slot, uint64_t &k) {
        int owner = 0; // first lane whose inclusive count exceeds j
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
            const uint32_t c = __shfl_sync(0xffffffffu, incl, owner + step - 1);
            if (c <= j) owner += step;
        }
        const uint32_t o_incl = __shfl_sync(0xffffffffu, incl, owner);
        const uint32_t o_n = __shfl_sync(0xffffffffu, n, owner);
        const uint32_t o_bw = __shfl_sync(0xffffffffu, bw, owner);
        const uint32_t o_pitch = __shfl_sync(0xffffffffu, pitch, owner);
        k = __shfl_sync(0xffffffffu, key, owner);
        int32_t *o_cur = reinterpret_cast<int32_t *>(
            __shfl_sync(0xffffffffu, reinterpret_cast<uintptr_t>(cur), owner));
        const uint32_t local = j - (o_incl - o_n);
        const uint32_t ry = local / o_bw, rx = local - ry * o_bw;
        slot = o_cur + (int64_t)ry * o_pitch + rx;
    };
    // EMIT_ROUNDS rounds per iteration: all their cursor atomics are in
    // flight before any of them stores its key
    for (uint32_t base = 0; base < total; base += 32 * EMIT_ROUNDS) {
        int32_t *sl[EMIT_ROUNDS];
        uint64_t kk[EMIT_ROUNDS];
        int32_t pos[EMIT_ROUNDS];
#pragma unroll
        for (int r = 0; r < EMIT_ROUNDS; ++r)
            if (base + 32 * r < total) locate(base + 32 * r + lane, sl[r], kk[r]); // uniform
#pragma unroll
        for (int r = 0; r < EMIT_ROUNDS; ++r)
            pos[r] = base + 32 * r + lane < total ? atomicAdd(sl[r], 1) : -1;
#pragma unroll
        for (int r = 0; r < EMIT_ROUNDS; ++r) {
            if (base + 32 * r + lane < total) {
                if (pos[r] >= 0 && pos[r] < cap) keys[pos[r]] = kk[r];
                else atomicOr(status, DEV_ERR_OVERFLOW);
            }
        }
    }
}

// Heaviest-first order of the buckets for the blend (longest-processing-time
// scheduling): one CTA counting-sorts the buckets by record count into
// ORDER_BINS bins of 4 records (descending; counts >= 4 * ORDER_BINS share the
// first bin).  Order within a bin is arbitrary, which only changes the launch
// order of the blend's CTAs, never a result.
constexpr int ORDER_BINS = 1024;
static __global__ void __launch_bounds__(1024) bucket_order_kernel(const int32_t *__restrict__ offsets,
                                                            const int64_t *T_dev, int64_t cap,
                                                            int32_t n_buckets,
                                                            int32_t *__restrict__ order) {
    __shared__ int32_t bins[ORDER_BINS];
    __shared__ int32_t warp_tot[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t T = T_dev ? imin64(*T_dev, cap) : cap;
    for (int i = tid; i < ORDER_BINS; i += blockDim.x) bins[i] = 0;
    __syncthreads();
    auto bin_of = [&](int32_t b) {
        int64_t lo, hi;
        bucket_range(offsets, b, n_buckets, T, lo, hi);
        const int64_t c = (hi - lo) >> 2;
        return ORDER_BINS - 1 - (int)(c < ORDER_BINS - 1 ? c : ORDER_BINS - 1);
    };
    for (int32_t b = tid; b < n_buckets; b += blockDim.x) atomicAdd(&bins[bin_of(b)], 1);
    __syncthreads();
    // exclusive scan of the 1024 bins (one per thread)
    const int v = tid < ORDER_BINS ? bins[tid] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int t = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        warp_tot[lane] = t; // inclusive
    }
    __syncthreads();
    if (tid < ORDER_BINS) bins[tid] = x - v + (wid ? warp_tot[wid - 1] : 0);
    __syncthreads();
    for (int32_t b = tid; b < n_buckets; b += blockDim.x) order[atomicAdd(&bins[bin_of(b)], 1)] = b;
}

// Both per-bucket passes of a frame with at most SCAN_ORDER_MAX buckets, in one
// launch of one cluster: the exclusive scan of the bucket counts (bucket
// offsets, int32, and the intersection total) and the heaviest-first bucket
// order of bucket_order_kernel (a counting sort by record count).
// The counts come in R replicas ([R][n], replica-major: the atomics of a
// bucket spread over R lines).  Every CTA folds, scans and bins a contiguous
// part of the buckets; the CTAs exchange their sums and histograms through
// distributed shared memory.  cursor[r n + b] receives the start of replica
// r's sub-range of bucket b (its bucket offset plus the counts of replicas
// 0 .. r - 1).  One CTA took 24 us for the 8,160 buckets of a 1080p frame and
// 111 us for 30,000.
// host (optional, memory the host reads): the total and the status word.
// order and cursor are optional too: without them this is the scan alone.
constexpr int SCAN_CTAS = 8;                    // cluster size above SCAN_SMALL buckets
constexpr int SCAN_SMALL = 1024;                // up to here one CTA
constexpr int SCAN_PER = 8;                     // buckets per thread at most
constexpr int SCAN_ORDER_MAX = SCAN_CTAS * 1024 * SCAN_PER;
template <int R>
__global__ void __launch_bounds__(1024) bucket_scan_order_kernel(
    const int32_t *__restrict__ counts, int32_t n, int32_t *__restrict__ offsets,
    int64_t *__restrict__ total, int32_t *__restrict__ order, int32_t *__restrict__ cursor,
    const uint32_t *status, volatile int64_t *host) {
    namespace cg = cooperative_groups;
    static_assert(ORDER_BINS == 1024, "one bin per thread");
    __shared__ int32_t cnt[1024 * SCAN_PER];
    __shared__ int32_t bins[ORDER_BINS], pos[ORDER_BINS];
    __shared__ int64_t wtot[32], cta_sum;
    __shared__ int32_t btot[32];
    const cg::cluster_group cluster = cg::this_cluster();
    const int G = gridDim.x, rank = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int chunk = (n + G - 1) / G;
    const int c0 = min(n, rank * chunk), m = min(n - c0, chunk);
    auto bin_of = [](int32_t c) {
        const int32_t q = c >> 2;
        return ORDER_BINS - 1 - (q < ORDER_BINS - 1 ? q : ORDER_BINS - 1);
    };
    bins[tid] = 0;
    __syncthreads();
    for (int i = tid; i < m; i += 1024) {
        int32_t c = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) c += counts[(int64_t)r * n + c0 + i];
        cnt[i] = c;
        atomicAdd(&bins[bin_of(c)], 1);
    }
    __syncthreads();
    // scan of this part, a run of consecutive buckets per thread
    const int per = (m + 1023) / 1024;
    int32_t c[SCAN_PER];
    int64_t run = 0;
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) {
        const int i = tid * per + k;
        c[k] = k < per && i < m ? cnt[i] : -1;
        run += max(c[k], 0);
    }
    int64_t inc = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wtot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int64_t w = wtot[lane];
        int64_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        wtot[lane] = wi - w; // exclusive
        if (lane == 31) cta_sum = wi;
    }
    cluster.sync(); // every CTA's sum and histogram are complete
    int64_t off = wtot[wid] + inc - run, all = 0;
    int32_t before = 0, in_bin = 0; // of bin tid: in lower CTAs, in all
    for (int g = 0; g < G; ++g) {
        const int64_t s = *cluster.map_shared_rank(&cta_sum, g);
        const int32_t h = cluster.map_shared_rank(bins, g)[tid];
        if (g < rank) {
            off += s;
            before += h;
        }
        all += s;
        in_bin += h;
    }
    if (rank == 0 && tid == 0) {
        *total = all;
        if (host) {
            host[1] = (int64_t)*status;
            host[0] = all;
        }
    }
#pragma unroll
    for (int k = 0; k < SCAN_PER; ++k) {
        if (c[k] >= 0) cnt[tid * per + k] = bucket_start(off);
        off += max(c[k], 0);
    }
    // heaviest-first order: exclusive scan of the bins, then a scatter
    int x = in_bin;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) btot[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int t = btot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        btot[lane] = t; // inclusive
    }
    __syncthreads();
    pos[tid] = x - in_bin + (wid ? btot[wid - 1] : 0) + before;
    __syncthreads();
    if (order) {
#pragma unroll
        for (int k = 0; k < SCAN_PER; ++k)
            if (c[k] >= 0) order[atomicAdd(&pos[bin_of(c[k])], 1)] = c0 + tid * per + k;
    }
    for (int i = tid; i < m; i += 1024) {
        int32_t o = cnt[i];
        offsets[c0 + i] = o;
        if (!cursor) continue;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            cursor[(int64_t)r * n + c0 + i] = o;
            o = bucket_start((int64_t)o + counts[(int64_t)r * n + c0 + i]);
        }
    }
    cluster.sync(); // no CTA leaves while another reads its histogram
}

template <int R>
inline int launch_bucket_scan_order(const int32_t *counts, int32_t n, int32_t *offsets,
                                    int64_t *total, int32_t *order, int32_t *cursor,
                                    const uint32_t *status, int64_t *host, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    const unsigned g = n <= SCAN_SMALL ? 1 : SCAN_CTAS;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = g;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = g;
    cfg.blockDim = 1024;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    UBS_TIMED("bucket_scan_order", st,
              cudaLaunchKernelEx(&cfg, bucket_scan_order_kernel<R>, counts, n, offsets, total,
                                 order, cursor, status, (volatile int64_t *)host));
    note_launch();
    return check_launch("bucket_scan_order");
}

// Larger frames (more than SCAN_ORDER_MAX buckets): the replicas' sums ...
template <int R>
__global__ void fold_replicas_kernel(const int32_t *__restrict__ counts, int64_t n,
                                     int32_t *__restrict__ totals) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    int32_t c = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) c += counts[r * n + b];
    totals[b] = c;
}
// ... and, after their exclusive scan, the replicas' cursors.
template <int R>
__global__ void replica_cursors_kernel(const int32_t *__restrict__ counts, int32_t n,
                                       const int32_t *__restrict__ offsets,
                                       int32_t *__restrict__ cursor) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    int32_t off = offsets[b];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        cursor[(int64_t)r * n + b] = off;
        off = bucket_start((int64_t)off + counts[(int64_t)r * n + b]);
    }
}

// Bitonic sort of the 32 * E keys of a warp held E per lane in registers,
// blocked (element i = lane * E + e): exchange distances below E stay inside
// a lane, larger ones are lane-xor shuffles.  The network runs in two phases
// so that no compare-exchange recomputes its direction:
//   * stages k < E sort runs inside a lane: distances and directions are
//     compile-time (element e of a run of k ascends when e & k == 0);
//   * stages k >= E: the direction of all E elements of a lane is the same,
//     ((lane * E) & k) == 0, one predicate per stage; the stage loop runs at
//     run time with one unrolled body per in-lane distance, which keeps the
//     code small enough for the instruction cache.
// The network is the same as the textbook bitonic sort, so the result is.
template <int E, int J, int K>
__device__ __forceinline__ void bitonic_run_pass(uint64_t (&v)[E]) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int p = e ^ J;
        if (p > e) {
            const uint64_t a = v[e], b = v[p];
            const bool sw = ((e & K) == 0) ? (a > b) : (a < b);
            v[e] = sw ? b : a;
            v[p] = sw ? a : b;
        }
    }
}
template <int E, int K, int J> struct BitonicRunStage {
    static __device__ __forceinline__ void run(uint64_t (&v)[E]) {
        bitonic_run_pass<E, J, K>(v);
        BitonicRunStage<E, K, J / 2>::run(v);
    }
};
template <int E, int K> struct BitonicRunStage<E, K, 0> {
    static __device__ __forceinline__ void run(uint64_t (&)[E]) {}
};
template <int E, int K> struct BitonicRuns { // stages K, 2K, .. < E
    static __device__ __forceinline__ void run(uint64_t (&v)[E]) {
        BitonicRunStage<E, K, K / 2>::run(v);
        BitonicRuns<E, (2 * K < E ? 2 * K : 0)>::run(v);
    }
};
template <int E> struct BitonicRuns<E, 0> {
    static __device__ __forceinline__ void run(uint64_t (&)[E]) {}
};

// One in-lane pass of distance J with the lane's direction `up`.
template <int E, int J>
__device__ __forceinline__ void bitonic_in_lane(uint64_t (&v)[E], bool up) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int p = e ^ J;
        if (p > e) {
            const uint64_t a = v[e], b = v[p];
            const bool sw = (a > b) == up;
            v[e] = sw ? b : a;
            v[p] = sw ? a : b;
        }
    }
}

template <int E>
__device__ __forceinline__ void warp_bitonic(uint64_t (&v)[E], int lane) {
    constexpr int N = 32 * E;
    BitonicRuns<E, (E >= 4 ? 2 : 0)>::run(v); // k = 2 .. E / 2 inside the lane
#pragma unroll 1
    for (int k = E >= 2 ? E : 2; k <= N; k <<= 1) {
        const bool up = ((lane * E) & k) == 0;
#pragma unroll 1
        for (int j = k >> 1; j >= E; j >>= 1) { // across lanes
            const int lj = j / E;
            const bool keep_min = ((lane & lj) == 0) == up;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint64_t o = __shfl_xor_sync(0xffffffffu, v[e], lj);
                v[e] = (keep_min == (o < v[e])) ? o : v[e];
            }
        }
        // inside a lane: distances E / 2 .. 1
        if (E >= 32) bitonic_in_lane<E, (E >= 32 ? 16 : 1)>(v, up);
        if (E >= 16) bitonic_in_lane<E, (E >= 16 ? 8 : 1)>(v, up);
        if (E >= 8) bitonic_in_lane<E, (E >= 8 ? 4 : 1)>(v, up);
        if (E >= 4) bitonic_in_lane<E, (E >= 4 ? 2 : 1)>(v, up);
        if (E >= 2) bitonic_in_lane<E, 1>(v, up);
    }
}

// The same network on 32-bit values: a compare-exchange is one minimum or
// maximum per value instead of a 64-bit comparison and two selects.
template <int E, int J>
__device__ __forceinline__ void bitonic32_in_lane(uint32_t (&v)[E], bool up) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int p = e ^ J;
        if (p > e) {
            const uint32_t a = v[e], b = v[p];
            v[e] = up ? min(a, b) : max(a, b);
            v[p] = up ? max(a, b) : min(a, b);
        }
    }
}
template <int E, int K, int J> struct Bitonic32RunStage {
    static __device__ __forceinline__ void run(uint32_t (&v)[E]) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int p = e ^ J;
            if (p > e) {
                const uint32_t a = v[e], b = v[p];
                v[e] = (e & K) == 0 ? min(a, b) : max(a, b);
                v[p] = (e & K) == 0 ? max(a, b) : min(a, b);
            }
        }
        Bitonic32RunStage<E, K, J / 2>::run(v);
    }
};
template <int E, int K> struct Bitonic32RunStage<E, K, 0> {
    static __device__ __forceinline__ void run(uint32_t (&)[E]) {}
};
template <int E, int K> struct Bitonic32Runs {
    static __device__ __forceinline__ void run(uint32_t (&v)[E]) {
        Bitonic32RunStage<E, K, K / 2>::run(v);
        Bitonic32Runs<E, (2 * K < E ? 2 * K : 0)>::run(v);
    }
};
template <int E> struct Bitonic32Runs<E, 0> {
    static __device__ __forceinline__ void run(uint32_t (&)[E]) {}
};
// The passes of stage k whose distances stay inside a warp (from j down).
template <int E>
__device__ __forceinline__ void bitonic32_in_warp(uint32_t (&v)[E], int lane, int j, bool up) {
#pragma unroll 1
    for (; j >= E; j >>= 1) { // across lanes
        const int lj = j / E;
        const bool keep_min = ((lane & lj) == 0) == up;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const uint32_t o = __shfl_xor_sync(0xffffffffu, v[e], lj);
            v[e] = keep_min ? min(v[e], o) : max(v[e], o);
        }
    }
    if (E >= 32) bitonic32_in_lane<E, (E >= 32 ? 16 : 1)>(v, up);
    if (E >= 16) bitonic32_in_lane<E, (E >= 16 ? 8 : 1)>(v, up);
    if (E >= 8) bitonic32_in_lane<E, (E >= 8 ? 4 : 1)>(v, up);
    if (E >= 4) bitonic32_in_lane<E, (E >= 4 ? 2 : 1)>(v, up);
    if (E >= 2) bitonic32_in_lane<E, 1>(v, up);
}
// Sorts the values of W warps, E per thread (thread t of the W warps holds
// elements t E ..); xch: shared memory of W 32 E values (W > 1, whose warps are
// the whole CTA).
template <int E, int W>
__device__ __forceinline__ void bitonic32(uint32_t (&v)[E], int t, uint32_t *xch) {
    constexpr int N = 32 * E;
    Bitonic32Runs<E, (E >= 4 ? 2 : 0)>::run(v);
#pragma unroll 1
    for (int k = E >= 2 ? E : 2; k <= N; k <<= 1)
        bitonic32_in_warp<E>(v, t & 31, k >> 1, ((t * E) & k) == 0);
    if (W > 1) {
#pragma unroll 1
        for (int k = 2 * N; k <= W * N; k <<= 1) {
            const bool up = ((t * E) & k) == 0;
#pragma unroll 1
            for (int j = k >> 1; j >= N; j >>= 1) { // across warps
                const int tj = j / E;
                const bool keep_min = ((t & tj) == 0) == up;
                __syncthreads();
#pragma unroll
                for (int e = 0; e < E; ++e) xch[e * 32 * W + t] = v[e];
                __syncthreads();
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const uint32_t o = xch[e * 32 * W + (t ^ tj)];
                    v[e] = keep_min ? min(v[e], o) : max(v[e], o);
                }
            }
            bitonic32_in_warp<E>(v, t & 31, N >> 1, up);
        }
    }
}

// Shared memory of one warp's sort: its keys and their order.
constexpr int ORDER_PITCH(int E) { return E + 2; } // 16-bit slots per lane, odd in words
constexpr size_t WARP_SORT_SMEM = WARP_SEG * sizeof(uint64_t) + 32 * ORDER_PITCH(32) * 2;

// Sorts n <= 32 E W unique keys src[0..n) with W warps (one warp, or all of a
// CTA's) and hands each to put(position, key).  sk (32 E W keys), si (32 W
// ORDER_PITCH(E) indices) and, for W > 1, xch are shared memory; src may be
// where put stores.
// The network runs on 32-bit composites: the depth bits above the smallest of
// the bucket (the entry bits where all depths are equal), shifted so that they
// leave room for the key's index among the n (a 1080p bucket of 500 keys keeps
// depth to 1 or 2 units in the last place).  Keys that agree in the bits kept
// come out in index order, so odd-even rounds on the index list exchange
// neighbours out of order until one finds none (nearly always the first or the
// second).  Returns false where that does not end soon -- many keys of a few
// depths -- with sk holding the keys as they came and put not called.
template <int E, int W, typename Put>
__device__ __forceinline__ bool sort_keys32(const uint64_t *src, int n, int t, uint64_t *sk,
                                            uint16_t *si, uint32_t *xch, Put put) {
    constexpr int T = 32 * W, N = T * E, P = ORDER_PITCH(E);
    constexpr int IB = N <= 32 ? 5 : N <= 64 ? 6 : N <= 128 ? 7 : N <= 256 ? 8 : N <= 512 ? 9
                       : N <= 1024 ? 10 : N <= 2048 ? 11 : 12;
    auto sync = []() {
        if (W > 1) __syncthreads();
        else __syncwarp();
    };
    auto any = [](bool b) {
        return W > 1 ? __syncthreads_or(b) != 0 : __any_sync(0xffffffffu, b) != 0;
    };
    __shared__ uint32_t range[W > 1 ? 2 * W : 1];
    // smallest and largest value over the keys
    auto span = [&](const uint32_t (&c)[E], uint32_t &lo, uint32_t &hi) {
        lo = ~0u;
        hi = 0u;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (e * T + t < n) {
                lo = min(lo, c[e]);
                hi = max(hi, c[e]);
            }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (W > 1) {
            __syncthreads();
            if ((t & 31) == 0) {
                range[t >> 5] = lo;
                range[W + (t >> 5)] = hi;
            }
            __syncthreads();
#pragma unroll
            for (int w = 0; w < W; ++w) {
                lo = min(lo, range[w]);
                hi = max(hi, range[W + w]);
            }
        }
    };
    uint32_t c[E], lo, hi;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = e * T + t;
        c[e] = 0u;
        if (i < n) {
            const uint64_t k = src[i];
            sk[i] = k;
            c[e] = (uint32_t)(k >> 32);
        }
    }
    span(c, lo, hi);
    if (lo == hi) { // the same in every thread
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (e * T + t < n) c[e] = (uint32_t)sk[e * T + t];
        span(c, lo, hi);
    }
    const int shift = max(0, IB - __clz(hi - lo));
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = e * T + t;
        c[e] = i < n ? ((c[e] - lo) >> shift) << IB | (uint32_t)i : ~0u;
    }
    bitonic32<E, W>(c, t, xch);
#pragma unroll
    for (int e = 0; e < E; ++e) si[t * P + e] = (uint16_t)(c[e] & (N - 1));
    sync();
    auto slot = [](int p) { return p / E * P + p % E; };
    // odd-even rounds: one without an exchange shows that the sequence is sorted
    bool sorted = false;
#pragma unroll 1
    for (int round = 0; round < 6 && !sorted; ++round) {
        bool swapped = false;
#pragma unroll 1
        for (int odd = 0; odd < 2; ++odd) {
#pragma unroll 4
            for (int p = 2 * t + odd; p + 1 < n; p += 2 * T) {
                const uint16_t a = si[slot(p)], b = si[slot(p + 1)];
                if (sk[a] > sk[b]) {
                    si[slot(p)] = b;
                    si[slot(p + 1)] = a;
                    swapped = true;
                }
            }
            if (W == 1 || !odd) sync(); // any() is the barrier of several warps
        }
        sorted = !any(swapped);
    }
    if (!sorted) return false;
#pragma unroll 4
    for (int p = t; p < n; p += T) put(p, sk[si[slot(p)]]);
    return true;
}

// One warp: the above, and the 64-bit network where it gives up.
template <int E, typename Put>
__device__ __forceinline__ void warp_sort_keys(const uint64_t *src, int n, int lane, uint64_t *sk,
                                               uint16_t *si, Put put) {
    if (sort_keys32<E, 1>(src, n, lane, sk, si, nullptr, put)) return;
    uint64_t v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = lane * E + e;
        v[e] = i < n ? sk[i] : ~0ull;
    }
    warp_bitonic<E>(v, lane);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = lane * E + e;
        if (i < n) put(i, v[e]);
    }
}

// One warp per bucket for buckets of at most WARP_SEG keys; longer buckets go
// to the device-side lists: mid (<= SMALL_SEG) from the front of `lists`, big
// from the back.  counters = {n_big, n_mid}.
constexpr int SORT_WARPS = 4;
template <typename Writer>
__global__ void __launch_bounds__(SORT_WARPS * 32, 5) bucket_sort_warp_kernel(
    int64_t n_buckets, const int32_t *__restrict__ offsets, const int64_t *T_dev, int64_t cap,
    const uint64_t *keys, int32_t *lists, int32_t *counters, Writer w) {
    __shared__ __align__(16) unsigned char sm[SORT_WARPS][WARP_SORT_SMEM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t bkt = (int64_t)blockIdx.x * SORT_WARPS + warp;
    if (bkt >= n_buckets) return;
    const int64_t T = T_dev ? imin64(*T_dev, cap) : cap;
    int64_t lo, hi;
    bucket_range(offsets, bkt, n_buckets, T, lo, hi);
    const int64_t n = hi - lo;
    if (n <= 0) return;
    if (n > WARP_SEG) {
        if (lane == 0) {
            if (n > SMALL_SEG) lists[n_buckets - 1 - atomicAdd(&counters[0], 1)] = (int32_t)bkt;
            else lists[atomicAdd(&counters[1], 1)] = (int32_t)bkt;
        }
        return;
    }
    const int m = (int)n;
    uint64_t *sk = reinterpret_cast<uint64_t *>(sm[warp]);
    uint16_t *si = reinterpret_cast<uint16_t *>(sk + WARP_SEG);
    auto put = [&](int p, uint64_t k) { w(k, lo + p, bkt); };
    if (m <= 32) warp_sort_keys<1>(keys + lo, m, lane, sk, si, put);
    else if (m <= 64) warp_sort_keys<2>(keys + lo, m, lane, sk, si, put);
    else if (m <= 128) warp_sort_keys<4>(keys + lo, m, lane, sk, si, put);
    else if (m <= 256) warp_sort_keys<8>(keys + lo, m, lane, sk, si, put);
    else if (m <= 512) warp_sort_keys<16>(keys + lo, m, lane, sk, si, put);
    else warp_sort_keys<32>(keys + lo, m, lane, sk, si, put);
}

// merge path: number of elements taken from a for output diagonal d
__device__ __forceinline__ int64_t merge_split(const uint64_t *a, int64_t na, const uint64_t *b,
                                               int64_t nb, int64_t d) {
    int64_t lo = d > nb ? d - nb : 0, hi = d < na ? d : na;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (a[mid] < b[d - 1 - mid]) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// In-place bitonic sort of s[0..n2) (n2 a power of two) by the whole CTA.
__device__ __forceinline__ void block_bitonic(uint64_t *s, int n2) {
    for (int k = 2; k <= n2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < n2; i += blockDim.x) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const uint64_t a = s[i], b = s[ixj];
                    const bool up = (i & k) == 0;
                    if ((a > b) == up) {
                        s[i] = b;
                        s[ixj] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// Buckets of WARP_SEG < n <= SMALL_SEG keys (the mid list): a fixed grid walks
// the device-side list with one CTA of MID_WARPS warps per bucket, whose
// threads run the 32-bit network together, 16 or 32 values each.
constexpr int MID_WARPS = 4;
constexpr size_t MID_SMEM = SMALL_SEG * (sizeof(uint64_t) + sizeof(uint32_t)) +
                            MID_WARPS * 32 * ORDER_PITCH(32) * sizeof(uint16_t);
template <typename Writer>
__global__ void __launch_bounds__(MID_WARPS * 32, 4) bucket_sort_mid_kernel(
    int64_t n_buckets, const int32_t *__restrict__ offsets, const int64_t *T_dev, int64_t cap,
    const uint64_t *keys, const int32_t *lists, const int32_t *counters, Writer w) {
    extern __shared__ __align__(16) uint64_t mid_keys[]; // keys, exchange buffer, order
    uint32_t *xch = reinterpret_cast<uint32_t *>(mid_keys + SMALL_SEG);
    uint16_t *si = reinterpret_cast<uint16_t *>(xch + SMALL_SEG);
    const int n_mid = counters[1];
    const int64_t T = T_dev ? imin64(*T_dev, cap) : cap;
    for (int item = blockIdx.x; item < n_mid; item += gridDim.x) {
        __syncthreads();
        const int64_t bkt = lists[item];
        int64_t lo, hi;
        bucket_range(offsets, bkt, n_buckets, T, lo, hi);
        const int n = (int)(hi - lo);
        auto put = [&](int p, uint64_t k) { w(k, lo + p, bkt); };
        const bool done =
            n <= 2048 ? sort_keys32<16, MID_WARPS>(keys + lo, n, threadIdx.x, mid_keys, si, xch, put)
                      : sort_keys32<32, MID_WARPS>(keys + lo, n, threadIdx.x, mid_keys, si, xch, put);
        if (done) continue; // the same in every thread
        int n2 = 2048;
        while (n2 < n) n2 <<= 1;
        for (int i = n + threadIdx.x; i < n2; i += blockDim.x) mid_keys[i] = ~0ull;
        __syncthreads();
        block_bitonic(mid_keys, n2);
        for (int i = threadIdx.x; i < n; i += blockDim.x) put(i, mid_keys[i]);
    }
}

// Long buckets (their number is known only on the device): a fixed grid walks
// the device-side list; the warps of a CTA sort runs of WARP_SEG keys in
// place, which the CTA merges pairwise in global memory (keys <-> scratch).
constexpr int BIG_WARPS = BIG_THREADS / 32;
constexpr size_t BIG_SMEM = BIG_WARPS * WARP_SORT_SMEM;
template <typename Writer>
__global__ void __launch_bounds__(BIG_THREADS) bucket_sort_big_kernel(
    int64_t n_buckets, const int32_t *__restrict__ offsets, const int64_t *T_dev, int64_t cap,
    uint64_t *keys, uint64_t *scratch, const int32_t *lists, const int32_t *counters, Writer w) {
    extern __shared__ __align__(16) unsigned char big_sm[];
    const int n_big = counters[0];
    const int64_t T = T_dev ? imin64(*T_dev, cap) : cap;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t *sk = reinterpret_cast<uint64_t *>(big_sm + warp * WARP_SORT_SMEM);
    uint16_t *si = reinterpret_cast<uint16_t *>(sk + WARP_SEG);
    for (int item = blockIdx.x; item < n_big; item += gridDim.x) {
        __syncthreads();
        const int64_t bkt = lists[n_buckets - 1 - item];
        int64_t lo, hi;
        bucket_range(offsets, bkt, n_buckets, T, lo, hi);
        const int64_t n = hi - lo;
        uint64_t *src = keys + lo, *dst = scratch + lo;
        for (int64_t c0 = (int64_t)warp * WARP_SEG; c0 < n; c0 += (int64_t)BIG_WARPS * WARP_SEG) {
            __syncwarp();
            warp_sort_keys<32>(src + c0, (int)imin64(WARP_SEG, n - c0), lane, sk, si,
                               [&](int p, uint64_t k) { src[c0 + p] = k; });
        }
        __syncthreads();
        for (int64_t width = WARP_SEG; width < n; width <<= 1) {
            for (int64_t r0 = 0; r0 < n; r0 += 2 * width) {
                const int64_t na = imin64(width, n - r0);
                const int64_t nb = imin64(width, n - r0 - na);
                const uint64_t *A = src + r0, *Bv = src + r0 + na;
                uint64_t *O = dst + r0;
                const int64_t total = na + nb;
                for (int64_t o0 = (int64_t)threadIdx.x * MERGE_ITEMS; o0 < total;
                     o0 += (int64_t)blockDim.x * MERGE_ITEMS) {
                    int64_t ia = merge_split(A, na, Bv, nb, o0);
                    int64_t ib = o0 - ia;
                    const int64_t oend = imin64(total, o0 + MERGE_ITEMS);
                    for (int64_t o = o0; o < oend; ++o) {
                        const bool take_a = ib >= nb || (ia < na && A[ia] < Bv[ib]);
                        O[o] = take_a ? A[ia++] : Bv[ib++];
                    }
                }
            }
            __syncthreads();
            uint64_t *t = src;
            src = dst;
            dst = t;
        }
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x) w(src[i], lo + i, bkt);
    }
}

// Launches the per-bucket sort: buckets of <= WARP_SEG keys one warp each in
// registers, <= SMALL_SEG one CTA each in shared memory, longer ones merged on
// a fixed grid.  lists ([n_buckets]) and counters ([2], zeroed here unless they
// are already) are scratch.
template <typename Writer>
inline int launch_bucket_sort(int64_t n_buckets, const int32_t *offsets, const int64_t *T_dev,
                              int64_t cap, uint64_t *keys, uint64_t *scratch, int32_t *lists,
                              int32_t *counters, Writer w, cudaStream_t st,
                              bool zeroed = false) {
    if (n_buckets <= 0 || cap <= 0) return UBS_OK;
    if (!zeroed && cudaMemsetAsync(counters, 0, 8, st) != cudaSuccess) return check_launch("sort memset");
    UBS_TIMED("bucket_sort_warp", st,
              bucket_sort_warp_kernel<Writer>
              <<<grid_for(n_buckets, SORT_WARPS), SORT_WARPS * 32, 0, st>>>(
                  n_buckets, offsets, T_dev, cap, keys, lists, counters, w));
    note_launch();
    if (cap > WARP_SEG) {
        const int64_t max_mid = cap / (WARP_SEG + 1);
        const unsigned grid = (unsigned)imin64(imin64(max_mid, n_buckets), 152 * 8);
        if (cudaFuncSetAttribute(bucket_sort_mid_kernel<Writer>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)MID_SMEM) != cudaSuccess)
            return check_launch("bucket_sort_mid attribute");
        UBS_TIMED("bucket_sort_mid", st,
                  bucket_sort_mid_kernel<Writer><<<grid, MID_WARPS * 32, MID_SMEM, st>>>(
                      n_buckets, offsets, T_dev, cap, keys, lists, counters, w));
        note_launch();
    }
    if (cap > SMALL_SEG) {
        const int64_t max_big = cap / (SMALL_SEG + 1);
        const unsigned grid = (unsigned)imin64(imin64(max_big, n_buckets), 152);
        if (grid > 0) {
            if (cudaFuncSetAttribute(bucket_sort_big_kernel<Writer>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)BIG_SMEM) != cudaSuccess)
                return check_launch("bucket_sort_big attribute");
            UBS_TIMED("bucket_sort_big", st,
                      bucket_sort_big_kernel<Writer><<<grid, BIG_THREADS, BIG_SMEM, st>>>(
                          n_buckets, offsets, T_dev, cap, keys, scratch, lists, counters, w));
            note_launch();
        }
    }
    return check_launch("bucket sort");
}

} // namespace ubs
