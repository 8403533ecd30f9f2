// One-sweep LSD radix sort of 64-bit Morton codes with 32-bit slot indices.
//
// Replaces the reference's recursiveParallelMortonSort / mortonSort
// (src/NBody/Simulation/Solvers/MortonSort.h:75-88, 141-183: MSB partition then boost spreadsort).
// The reference leaves the order of equal codes unspecified; this sort is stable, so equal codes
// keep their input order (input index order on a fresh set of bodies).
//
// Design (one-sweep, decoupled look-back), above kSmallSort keys:
//   - the Morton kernel already counted all eight 8-bit digit histograms;
//   - each of the 8 passes is ONE kernel: a block takes the next tile (atomic ticket), ranks its
//     4096 keys by digit with warp ballots (stable), publishes its per-digit counts, looks
//     back over earlier tiles' published counts (four at a time) for its global digit offsets, stages
//     the tile in shared memory in digit order and writes it out in runs of equal digits. The
//     exclusive prefix of the pass's histogram is a scan of 256 counts in every block.
// Per pass each key is read once and written once: 12 B read + 12 B written per body.
// Every look-back wait is bounded by a 2 s timer; on expiry the kernel sets an error bit that the
// host reports, and carries on without hanging the device.
// Up to kSmallSort keys are sorted by one cluster of blocks, all passes in one kernel.
#include <utility>

#include <cooperative_groups.h>

#include "nb_internal.cuh"

namespace cg = cooperative_groups;

namespace nbg {

namespace {

constexpr int kThreads = 512;
constexpr int kItems = 8;
constexpr int kTile = kSortTileKeys;
static_assert(kThreads * kItems == kTile, "one tile is kItems keys per thread");
constexpr int kWarps = kThreads / 32;
constexpr int kPasses = kSortPasses;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1;
constexpr int kLook = 4;  // tiles looked back over at a time
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The lanes that hold the same 8-bit digit (bits above are ignored): eight ballots. __match_any_sync takes
// time with the number of distinct values, here nearly one per lane: a one-sweep pass over 2^20 keys
// took 21.5 us with it, 20.4 us with ballots, the cluster sort of 10,000 keys 53 and 43 us.
__device__ __forceinline__ uint32_t same_digit(uint32_t d) {
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t set = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? set : ~set;
    }
    return peers;
}

__device__ __forceinline__ uint32_t load_volatile(const uint32_t *p) { return *(const volatile uint32_t *) p; }
__device__ __forceinline__ void store_volatile(uint32_t *p, uint32_t v) { *(volatile uint32_t *) p = v; }

// All 8 passes over at most kCluster x kClusterThreads x K keys by one cluster of eight blocks, keys in
// registers. Per pass every block ranks its keys, the blocks read each other's digit counts and
// store their keys straight into the shared memory of the block that holds their new position
// (distributed shared memory): two cluster barriers per pass instead of a kernel with its look-back.
// Latency bound. 1,023 keys: 49 us in eight one-sweep launches before, 20 us now; 10,000 keys: 68 and
// 37 us (43 us when keys went straight from their lanes to scattered places of the other blocks). One
// block of 1,024 threads instead of the cluster: 28 and 143 us.
constexpr int kCluster = 8;
constexpr int kClusterThreads = 512;
constexpr int kClusterWarps = kClusterThreads / 32;

template<int K>
struct ClusterSmem {
    uint64_t keys[kClusterThreads * K];
    uint32_t vals[kClusterThreads * K];
    uint64_t stage_keys[kClusterThreads * K];  // the block's keys in digit order
    uint32_t stage_vals[kClusterThreads * K];
    uint32_t hist[kClusterWarps][256];  // per warp: digit counts, then its keys' places in the block
    uint32_t count[256];                // the block's digit counts, read by the other blocks
    uint32_t shift[256];                // per digit: place in the cluster minus place in the block
    uint32_t total[8];
};

template<int K>
__global__ void __launch_bounds__(kClusterThreads) __cluster_dims__(kCluster, 1, 1)
    cluster_sort_kernel(const uint64_t *keys_in, uint64_t *keys_out, uint32_t *vals_out, int n) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem<K> &S = *reinterpret_cast<ClusterSmem<K> *>(smem_raw);
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int kBlockKeys = kClusterThreads * K;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int) cluster.block_rank();
    const uint32_t lt = lanemask_lt();
    // Padding keys are all ones and come last; ties keep the input order, so they stay last.
    uint64_t k[K];
    uint32_t v[K], r[K];
#pragma unroll
    for (int it = 0; it < K; ++it) {
        const int i = rank * kBlockKeys + (warp * K + it) * 32 + lane;
        k[it] = i < n ? keys_in[i] : ~0ull;
        v[it] = (uint32_t) i;
    }
    for (int shift = 0; shift < 64; shift += 8) {
        for (int i = tid; i < kClusterWarps * 256; i += kClusterThreads) (&S.hist[0][0])[i] = 0;
        __syncthreads();
#pragma unroll
        for (int it = 0; it < K; ++it) {
            const uint32_t d = (uint32_t) (k[it] >> shift) & 255u;
            const uint32_t peers = same_digit(d);
            const int leader = 31 - __clz(peers);
            uint32_t before = 0;
            if (lane == leader) {
                before = S.hist[warp][d];
                S.hist[warp][d] = before + __popc(peers);
            }
            before = __shfl_sync(0xffffffffu, before, leader);
            r[it] = before + __popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        uint32_t c[kClusterWarps];
        uint32_t sum = 0;
        if (tid < 256) {
#pragma unroll
            for (int w = 0; w < kClusterWarps; ++w) c[w] = S.hist[w][tid];
#pragma unroll
            for (int w = 0; w < kClusterWarps; ++w) sum += c[w];
            S.count[tid] = sum;
        }
        cluster.sync();
        // one scan over the digits for both: the cluster's counts (upper half) and the block's
        uint32_t packed = 0, before = 0, incl = 0;
        if (tid < 256) {
#pragma unroll
            for (int b = 0; b < kCluster; ++b) {
                const uint32_t x = *cluster.map_shared_rank(&S.count[tid], b);
                packed += x << 16;
                if (b < rank) before += x;
            }
            packed += sum;
            incl = packed;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) S.total[warp] = incl;
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t run = incl - packed;
#pragma unroll
            for (int w = 0; w < 8; ++w) run += w < warp ? S.total[w] : 0u;
            uint32_t place = run & 0xffffu;
            S.shift[tid] = (run >> 16) + before - place;
#pragma unroll
            for (int w = 0; w < kClusterWarps; ++w) {
                S.hist[w][tid] = place;
                place += c[w];
            }
        }
        __syncthreads();
        // in digit order within the block first, so that neighbouring threads store to neighbouring
        // places of the other blocks: single stores to scattered ones took most of a pass
#pragma unroll
        for (int it = 0; it < K; ++it) {
            const uint32_t at = S.hist[warp][(uint32_t) (k[it] >> shift) & 255u] + r[it];
            S.stage_keys[at] = k[it];
            S.stage_vals[at] = v[it];
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < K; ++it) {
            const int i = it * kClusterThreads + tid;
            const uint64_t key = S.stage_keys[i];
            const uint32_t pos = i + S.shift[(uint32_t) (key >> shift) & 255u];
            const unsigned to = pos / kBlockKeys, at = pos % kBlockKeys;
            *cluster.map_shared_rank(&S.keys[at], to) = key;
            *cluster.map_shared_rank(&S.vals[at], to) = S.stage_vals[i];
        }
        cluster.sync();
#pragma unroll
        for (int it = 0; it < K; ++it) {
            k[it] = S.keys[(warp * K + it) * 32 + lane];
            v[it] = S.vals[(warp * K + it) * 32 + lane];
        }
    }
#pragma unroll
    for (int it = 0; it < K; ++it) {
        const int i = rank * kBlockKeys + (warp * K + it) * 32 + lane;
        if (i < n) {
            keys_out[i] = k[it];
            vals_out[i] = v[it];
        }
    }
}
static_assert(kCluster * kClusterThreads * 4 == kSmallSort, "the cluster sort's largest form");

template<int K>
cudaError_t launch_cluster_sort(const uint64_t *keys_in, uint64_t *keys_out, uint32_t *vals_out, int n, cudaStream_t s) {
    static bool ready[64] = {false};
    constexpr size_t smem = sizeof(ClusterSmem<K>);
    int device = 0;
    cudaGetDevice(&device);
    if (device < 0 || device >= 64) device = 0;
    if (!ready[device]) {
        const cudaError_t e = cudaFuncSetAttribute(cluster_sort_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        if (e != cudaSuccess) return e;
        ready[device] = true;
    }
    cluster_sort_kernel<K><<<kCluster, kClusterThreads, smem, s>>>(keys_in, keys_out, vals_out, n);
    return cudaPeekAtLastError();
}

struct TileSmem {
    uint64_t keys[kTile];
    uint32_t vals[kTile];
    uint32_t whist[kWarps][256];
    uint32_t start[256];
    int32_t base[256];
    uint32_t warp_tot[kWarps], digit_tot[kWarps];
    uint32_t tile;
};

__global__ void __launch_bounds__(kThreads, 2) onesweep_kernel(const uint64_t *__restrict__ keys_in,
                                                            const uint32_t *__restrict__ vals_in,
                                                            uint64_t *__restrict__ keys_out,
                                                            uint32_t *__restrict__ vals_out, int64_t n, int pass,
                                                            const uint32_t *__restrict__ hist,
                                                            uint32_t *__restrict__ lookback,
                                                            uint32_t *__restrict__ tile_counter,
                                                            uint32_t *__restrict__ err,
                                                            unsigned long long wait_limit_ns) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileSmem &S = *reinterpret_cast<TileSmem *>(smem_raw);
    uint64_t *s_keys = S.keys;
    uint32_t *s_vals = S.vals;
    uint32_t(*s_whist)[256] = S.whist;
    uint32_t *s_start = S.start, *s_warp_tot = S.warp_tot, *s_digit_tot = S.digit_tot;
    int32_t *s_base = S.base;
    uint32_t &s_tile = S.tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int num_tiles = gridDim.x;
    const bool first = (pass == 0);
    const int shift = 8 * pass;

    if (tid == 0) s_tile = atomicAdd(&tile_counter[pass], 1u);
    for (int i = tid; i < kWarps * 256; i += kThreads) (&s_whist[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t base = tile * kTile;

    const uint32_t digit_count = tid < 256 ? hist[pass * 256 + tid] : 0u;
    if (__syncthreads_or(tid < 256 && (int64_t) digit_count == n)) {
        // Every key has the same digit in this pass: the stable result is the input order.
        for (int i = tid; i < kTile; i += kThreads) {
            int64_t idx = base + i;
            if (idx < n) {
                keys_out[idx] = keys_in[idx];
                vals_out[idx] = first ? (uint32_t) idx : vals_in[idx];
            }
        }
        return;
    }

    // Warp-striped load: item it of lane l in warp w is key base + w*256 + it*32 + l, so that
    // ranking items in (it, lane) order within a warp and warps in order keeps the sort stable.
    uint64_t k[kItems];
    uint32_t v[kItems], rank[kItems], dig[kItems];
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        int64_t idx = base + warp * 32 * kItems + it * 32 + lane;
        bool valid = idx < n;
        k[it] = valid ? keys_in[idx] : ~0ull;
        v[it] = valid ? (first ? (uint32_t) idx : vals_in[idx]) : 0u;
        dig[it] = valid ? (uint32_t) ((k[it] >> shift) & 255u) : 256u;
    }
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const uint32_t d = dig[it];
        const uint32_t live = __ballot_sync(0xffffffffu, d < 256u);
        const uint32_t peers = same_digit(d) & (d < 256u ? live : ~live);
        const int leader = 31 - __clz(peers);
        uint32_t before = 0;
        if (lane == leader && d < 256u) {
            before = s_whist[warp][d];
            s_whist[warp][d] = before + __popc(peers);
        }
        before = __shfl_sync(0xffffffffu, before, leader);
        rank[it] = before + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();

    // Exclusive prefix of the pass's digit counts, and per digit the exclusive prefix over the warps
    // and the tile's count.
    const int d = tid;
    uint32_t prefix = digit_count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, prefix, o);
        if (lane >= o) prefix += t;
    }
    if (lane == 31) s_digit_tot[warp] = prefix;
    uint32_t count = 0;
    if (d < 256) {
        uint32_t c[kWarps];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) c[w] = s_whist[w][d];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            s_whist[w][d] = count;
            count += c[w];
        }
    }
    __syncthreads();
    uint32_t global_off = prefix - digit_count;
    for (int w = 0; w < warp; ++w) global_off += s_digit_tot[w];
    uint32_t *my_lb = lookback + ((int64_t) pass * num_tiles + tile) * 256;
    if (d < 256) store_volatile(&my_lb[d], tile == 0 ? kFlagInc | (global_off + count) : kFlagAgg | count);

    // Exclusive scan of the tile's digit counts -> where each digit starts within the tile.
    uint32_t incl = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp_tot[warp] = incl;
    __syncthreads();
    uint32_t wbefore = 0;
    for (int w = 0; w < warp; ++w) wbefore += s_warp_tot[w];
    const uint32_t start = wbefore + incl - count;

    if (d < 256) {
        s_start[d] = start;
        // Decoupled look-back for this digit.
        uint32_t excl;
        if (tile == 0) {
            excl = global_off;
        } else {
            // the words of kLook tiles are loaded at once and used in order: with tiles publishing their
            // counts at about the same time, a tile waits for some sqrt(2 tile / kLook) round trips to L2
            excl = 0;
            int64_t t = tile - 1;
            const uint32_t *lb = lookback + (int64_t) pass * num_tiles * 256 + d;
            const unsigned long long t0 = global_timer_ns();
            bool done = false;
            while (!done) {
                uint32_t w[kLook];
#pragma unroll
                for (int i = 0; i < kLook; ++i) w[i] = t >= i ? load_volatile(lb + (t - i) * 256) : 0u;
                bool open = true;
#pragma unroll
                for (int i = 0; i < kLook; ++i) {
                    const uint32_t f = w[i] & kFlagMask;
                    open = open && f != 0u;  // a tile that has not published yet: the rest is loaded again
                    if (open && !done) {
                        excl += w[i] & kValueMask;
                        done = f == kFlagInc;
                        --t;
                    }
                }
                if (!open && !done && global_timer_ns() - t0 > wait_limit_ns) {
                    atomicOr(err, (uint32_t) kErrLookbackTimeout);
                    break;
                }
            }
            store_volatile(&my_lb[d], kFlagInc | ((excl + count) & kValueMask));
        }
        s_base[d] = (int32_t) excl - (int32_t) start;
    }
    __syncthreads();

    // Stage the tile in digit order.
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const uint32_t dd = dig[it];
        if (dd < 256u) {
            const uint32_t pos = s_start[dd] + s_whist[warp][dd] + rank[it];
            s_keys[pos] = k[it];
            s_vals[pos] = v[it];
        }
    }
    __syncthreads();

    const int tile_n = (int) ((n - base) < kTile ? (n - base) : kTile);
    for (int i = tid; i < tile_n; i += kThreads) {
        const uint64_t key = s_keys[i];
        const uint32_t dd = (uint32_t) ((key >> shift) & 255u);
        const int64_t o = (int64_t) s_base[dd] + i;
        keys_out[o] = key;
        vals_out[o] = s_vals[i];
    }
}

}  // namespace

// The one-sweep kernel's dynamic shared memory, enabled on first use per device.
static size_t tile_smem() {
    static bool ready[64] = {false};
    int device = 0;
    cudaGetDevice(&device);
    if (device < 0 || device >= 64) device = 0;
    if (!ready[device]) {
        cudaFuncSetAttribute(onesweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(TileSmem));
        ready[device] = true;
    }
    return sizeof(TileSmem);
}

int64_t sort_tiles(int64_t n) { return (n + kTile - 1) / kTile; }

cudaError_t clear_sort(int64_t n, SortWorkspace &ws, cudaStream_t s) {
    if (n <= kSmallSort) return cudaSuccess;
    return cudaMemsetAsync(ws.hist, 0, sort_words(n) * sizeof(uint32_t), s);
}

size_t sort_lookback_words(int64_t n) { return (size_t) kPasses * (size_t) (sort_tiles(n) > 0 ? sort_tiles(n) : 1) * 256; }

void launch_radix_pass(const uint64_t *keys_in, const uint32_t *vals_in, uint64_t *keys_out, uint32_t *vals_out,
                       int64_t n, int pass, const uint32_t *hist, uint32_t *lookback, uint32_t *tile_counter,
                       uint32_t *err, cudaStream_t s) {
    if (n <= 0) return;
    onesweep_kernel<<<(unsigned) sort_tiles(n), kThreads, tile_smem(), s>>>(keys_in, vals_in, keys_out, vals_out, n, pass,
                                                                   hist, lookback, tile_counter, err, kWaitLimitNs);
}

cudaError_t launch_radix_sort(const uint64_t *src, uint64_t *keys, uint32_t *vals, int64_t n, SortWorkspace &ws,
                              uint32_t *err, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (n <= kCluster * kClusterThreads) return launch_cluster_sort<1>(src, keys, vals, (int) n, s);
    if (n <= kSmallSort) return launch_cluster_sort<4>(src, keys, vals, (int) n, s);
    const int64_t tiles = sort_tiles(n);
    const size_t smem = tile_smem();
    cudaError_t e = cudaSuccess;
    const uint64_t *kin = src;
    uint64_t *kout = ws.keys_alt, *kother = keys;
    uint32_t *vin = vals, *vout = ws.vals_alt;
    for (int p = 0; p < kPasses; ++p) {
        onesweep_kernel<<<(unsigned) tiles, kThreads, smem, s>>>(kin, vin, kout, vout, n, p, ws.hist, ws.lookback,
                                                               ws.tile_counter, err, kWaitLimitNs);
        if ((e = cudaPeekAtLastError()) != cudaSuccess) return e;
        kin = kout;
        std::swap(kout, kother);
        std::swap(vin, vout);
    }
    // An even number of passes leaves the result in (keys, vals).
    static_assert(kPasses % 2 == 0, "the sorted data must end in the caller's buffers");
    return cudaSuccess;
}

}  // namespace nbg

namespace nbg {

// One pass whose look-back can never complete, to check that the bounded wait ends: a single block
// is launched with its tile ticket preset to 1, so it takes tile 1 of a two-tile input and waits on
// tile 0's flags, which nothing ever publishes. Every index stays in bounds: keys and values hold
// two tiles, the look-back buffer two tiles of 256 flags (the kernel indexes it with gridDim = 1),
// and the tile's scatter writes within the first tile's positions. Returns the error word.
cudaError_t lookback_timeout_selftest(unsigned long long wait_limit_ns, uint32_t *err_word) {
    const int64_t n = 2 * kTile;
    uint64_t *keys = nullptr, *keys_out = nullptr;
    uint32_t *vals = nullptr, *vals_out = nullptr, *hist = nullptr, *lookback = nullptr, *ticket = nullptr,
             *err = nullptr;
    cudaError_t e = cudaSuccess;
    auto alloc = [&](void **p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
        if (e == cudaSuccess) e = cudaMemset(*p, 0, bytes);
    };
    alloc((void **) &keys, n * sizeof(uint64_t));
    alloc((void **) &keys_out, n * sizeof(uint64_t));
    alloc((void **) &vals, n * sizeof(uint32_t));
    alloc((void **) &vals_out, n * sizeof(uint32_t));
    alloc((void **) &hist, kPasses * 256 * sizeof(uint32_t));  // no pass is trivial
    alloc((void **) &lookback, 2 * 256 * sizeof(uint32_t));
    alloc((void **) &ticket, kPasses * sizeof(uint32_t));
    alloc((void **) &err, sizeof(uint32_t));
    if (e == cudaSuccess) {
        const uint32_t one = 1;
        e = cudaMemcpy(ticket, &one, sizeof(one), cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) {
        onesweep_kernel<<<1, kThreads, tile_smem()>>>(keys, vals, keys_out, vals_out, n, 0, hist, lookback, ticket, err,
                                         wait_limit_ns);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(err_word, err, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    for (void *p: {(void *) keys, (void *) keys_out, (void *) vals, (void *) vals_out, (void *) hist,
                   (void *) lookback, (void *) ticket, (void *) err})
        if (p) cudaFree(p);
    return e;
}

}  // namespace nbg
