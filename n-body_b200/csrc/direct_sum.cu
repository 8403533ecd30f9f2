// Shared-memory-tiled direct sum: the NaiveSolver path (src/NBody/Simulation/Solvers/NaiveSolver.h:22-52)
// in FP32, and an FP64 variant that serves as the accuracy reference for the tree solvers.
//
// A block of eight warps stages 256 source bodies at a time in shared memory (coalesced float4 loads,
// double buffered, one barrier per tile) and sweeps the tile with broadcast reads. Its targets:
//   Z = 8: 32 targets (FP32: 64 where there are enough), every warp taking an eighth of each tile;
//   Z = 1: 256 targets (FP32: 512), for target counts that fill the GPU that way already or few sources.
// Up to eight blocks of a cluster share the sources of the same targets. Partial sums meet in shared
// memory, warps first, then the cluster's blocks (distributed shared memory), in a fixed order.
// One thread per target over all sources, 256 targets per block, left 30,011 targets on 118 of 148
// SMs with 8 warps each, and 4,096 targets on 16.
// Pair term as Gravity::particleParticle (Gravity.h:199-209): a += -R m / (|R|^2 + eps)^{3/2},
// R = target - source, identical positions skipped.
#include <algorithm>
#include <type_traits>

#include <cooperative_groups.h>

#include "nb_internal.cuh"

namespace cg = cooperative_groups;

namespace nbg {

namespace {

constexpr int kThreads = 256;
constexpr int kTile = 256;
constexpr int kMaxCluster = 8;

// Padding source: no mass, so far away that its factor is exactly zero (pair2_term).
__device__ __forceinline__ float4 load_source(const float4 *__restrict__ bodies, int64_t j, int64_t end) {
    return j < end ? __ldg(bodies + j) : make_float4(1e30f, 1e30f, 1e30f, 0.f);
}

// The sources of block `rank` of a cluster of `size`.
__device__ __forceinline__ void source_range(int64_t n, unsigned rank, unsigned size, int64_t &begin, int64_t &end) {
    begin = n * rank / size;
    end = n * (rank + 1) / size;
}

// Adds the partial sums of a target (Z per block, one block per cluster rank) in warp order, then
// rank order, and returns them on the cluster's first block, in the threads below 256 / Z. Every
// thread of the cluster must call it.
template<int Z, typename T>
__device__ __forceinline__ bool reduce_target(T (*part)[3], T &ax, T &ay, T &az) {
    cg::cluster_group cluster = cg::this_cluster();
    const int t = threadIdx.x;
    part[t][0] = ax;
    part[t][1] = ay;
    part[t][2] = az;
    __syncthreads();
    constexpr int kTargets = kThreads / Z;
    if (t < kTargets) {
#pragma unroll
        for (int z = 1; z < Z; ++z) {
            ax += part[t + z * kTargets][0];
            ay += part[t + z * kTargets][1];
            az += part[t + z * kTargets][2];
        }
        part[t][0] = ax;
        part[t][1] = ay;
        part[t][2] = az;
    }
    if (cluster.num_blocks() == 1) return t < kTargets;
    cluster.sync();
    if (cluster.block_rank() == 0 && t < kTargets) {
        for (unsigned r = 1; r < cluster.num_blocks(); ++r) {
            const T *other = cluster.map_shared_rank(&part[t][0], r);
            ax += other[0];
            ay += other[1];
            az += other[2];
        }
    }
    cluster.sync();  // the other blocks' sums stay readable until they are read
    return cluster.block_rank() == 0 && t < kTargets;
}

// Bound by the FP32 pipe: 12 lane operations per pair (six paired instructions for two) against a
// quarter of a lane's reciprocal roots per clock (300 us for 30,011 bodies). A broadcast 16-byte read
// still delivers 512 bytes to the warp's registers, four cycles of the SM's shared-memory pipe: with
// one target per lane the two reads of a source pair outweigh its arithmetic, so a lane takes T = 2 targets
// where there are enough of them.
// 30,011 bodies: 692 us before, 456 us with T = 1, 426 us now.
template<bool EPS0, int Z, int T>
__global__ void __launch_bounds__(kThreads) direct_f32_kernel(const float4 *__restrict__ bodies, int64_t n,
                                                              const float4 *__restrict__ targets, int64_t nt,
                                                              float G, float eps, float4 *__restrict__ acc) {
    // sources 2j and 2j + 1 of a tile as (x, x', y, y') and (z, z', m, m')
    __shared__ float4 tile[2][kTile];
    __shared__ float part[kThreads][3];
    constexpr int kTargets = kThreads / Z;
    cg::cluster_group cluster = cg::this_cluster();
    const int t = threadIdx.x, z = t / kTargets;
    const int64_t i0 = (int64_t) (blockIdx.x / cluster.num_blocks()) * (kTargets * T) + t % kTargets;
    float2 npx[T], npy[T], npz[T], ax[T], ay[T], az[T];
#pragma unroll
    for (int q = 0; q < T; ++q) {
        const int64_t i = i0 + q * kTargets;
        const float4 p = i < nt ? targets[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        npx[q] = make_float2(-p.x, -p.x);
        npy[q] = make_float2(-p.y, -p.y);
        npz[q] = make_float2(-p.z, -p.z);
        ax[q] = ay[q] = az[q] = make_float2(0.f, 0.f);
    }
    const float2 eps2 = make_float2(eps, eps);
    int64_t begin, end;
    source_range(n, cluster.block_rank(), cluster.num_blocks(), begin, end);
    float4 next = load_source(bodies, begin + t, end);
    int buf = 0;
    for (int64_t base = begin; base < end; base += kTile, buf ^= 1) {
        float *f = reinterpret_cast<float *>(tile[buf]) + (t >> 1) * 8 + (t & 1);
        f[0] = next.x;
        f[2] = next.y;
        f[4] = next.z;
        f[6] = next.w;
        __syncthreads();  // also: every warp is done with the other buffer
        next = load_source(bodies, base + kTile + t, end);
        const int pairs = (int) ((end - base < kTile ? end - base : kTile) + 1) >> 1;
        const float4 *src = tile[buf];
        auto terms = [&](int k) {
            const float4 u = src[2 * k], v = src[2 * k + 1];
#pragma unroll
            for (int q = 0; q < T; ++q) pair2_term<EPS0>(npx[q], npy[q], npz[q], eps2, u, v, ax[q], ay[q], az[q]);
        };
        if (pairs == kTile / 2) {
#pragma unroll 4
            for (int k = z; k < kTile / 2; k += Z) terms(k);
        } else {
            for (int k = z; k < pairs; k += Z) terms(k);
        }
    }
#pragma unroll
    for (int q = 0; q < T; ++q) {
        const int64_t i = i0 + q * kTargets;
        float sx = ax[q].x + ax[q].y, sy = ay[q].x + ay[q].y, sz = az[q].x + az[q].y;
        if (q > 0) __syncthreads();  // the target before has been added up
        if (reduce_target<Z>(part, sx, sy, sz) && i < nt) acc[i] = make_float4(G * sx, G * sy, G * sz, 0.f);
    }
}

// 1 / sqrt(x) of a normal x > 0 in FP64: the hardware's seed y and one step of Householder's third-order
// iteration, y (1 + h / 2 + 3 h^2 / 8) with h = 1 - x y^2: 5 FP64 operations, against a square root and a
// divide of some 20 each. The first term left out is 5/16 h^3. |h| is below 2^-19 (2^-19.04 at most over every
// high word of [1, 4), on which alone the seed depends), so that the term is below 2^-58; y^2 is exact (20
// mantissa bits), and the last operation's rounding is all that counts.
// FAR: x may be infinite, where the root is 0 and h a NaN. The three instructions that tell cost 6 % (1.34 -> 1.42 ms
// for 4,096 targets x 2^18 bodies), so only tiles that can need them take them.
template<bool FAR>
__device__ __forceinline__ double rsqrt_f64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double h = fma(-x, y * y, 1.0);
    const double root = fma(fma(h, 0.375, 0.5) * h, y, y);
    return FAR && __double2hiint(x) == 0x7ff00000 ? y : root;
}

__device__ __forceinline__ bool far_away(float4 p) { return isinf(p.x) || isinf(p.y) || isinf(p.z); }

// Bound by the FP64 pipe (64 lanes per SM and clock): 17 operations per pair. Sources are converted
// once per block and tile. 4,096 targets x 2^18 bodies: 52.8 ms before (16 blocks), 1.3 ms now; the
// error against extended precision fell from 1.6e-14 to 2.6e-16 (shorter chains of sums).
template<int Z>
__global__ void __launch_bounds__(kThreads) direct_f64_kernel(const float4 *__restrict__ bodies, int64_t n,
                                                              const float4 *__restrict__ targets, int64_t nt,
                                                              double G, double eps, double *__restrict__ acc3) {
    __shared__ double2 tile[2][kTile][2];  // (x, y), (z, m)
    __shared__ double part[kThreads][3];
    constexpr int kTargets = kThreads / Z;
    cg::cluster_group cluster = cg::this_cluster();
    const int t = threadIdx.x, z = t / kTargets;
    const int64_t i = (int64_t) (blockIdx.x / cluster.num_blocks()) * kTargets + t % kTargets;
    const float4 p = i < nt ? targets[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const double px = p.x, py = p.y, pz = p.z;
    const bool far_target = far_away(p) || isinf(eps);
    double ax = 0.0, ay = 0.0, az = 0.0;
    int64_t begin, end;
    source_range(n, cluster.block_rank(), cluster.num_blocks(), begin, end);
    float4 next = load_source(bodies, begin + t, end);
    int buf = 0;
    for (int64_t base = begin; base < end; base += kTile, buf ^= 1) {
        tile[buf][t][0] = make_double2(next.x, next.y);
        tile[buf][t][1] = make_double2(next.z, next.w);
        const bool far = __syncthreads_or(far_target || far_away(next));
        next = load_source(bodies, base + kTile + t, end);
        const int cnt = (int) (end - base < kTile ? end - base : kTile);
        const double2(*src)[2] = tile[buf];
        auto term = [&](int k, auto may_be_far) {
            const double2 u = src[k][0], v = src[k][1];
            const double dx = u.x - px, dy = u.y - py, dz = v.x - pz;
            const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
            const double inv = rsqrt_f64<decltype(may_be_far)::value>(d2 + eps);
            const double s = v.y * inv * (inv * inv);
            // positions of floats: d2 is zero or at least 2^-298, so its high word tells
            const double w = __double2hiint(d2) == 0 ? 0.0 : s;
            ax = fma(dx, w, ax);
            ay = fma(dy, w, ay);
            az = fma(dz, w, az);
        };
        if (cnt == kTile && !far) {
#pragma unroll 4
            for (int k = z; k < kTile; k += Z) term(k, std::false_type());
        } else {
            for (int k = z; k < cnt; k += Z) term(k, std::true_type());
        }
    }
    if (reduce_target<Z>(part, ax, ay, az) && i < nt) {
        acc3[3 * i + 0] = G * ax;
        acc3[3 * i + 1] = G * ay;
        acc3[3 * i + 2] = G * az;
    }
}

// Energy diagnostics in FP64: the kinetic energy 1/2 m v^2 and the sum over pairs of m_i m_j / sqrt(|r_ij|^2 + eps)
// (pairs at equal positions skipped, as the force skips them). Bodies are cut into tiles of 256; a
// pair of tiles is evaluated once: tile I takes the tiles I + 0 .. I + tiles / 2 around the ring of
// tiles (the farthest only from the lower half when the tile count is even), block y of its row an
// equal share of them. parts[2 block + {0, 1}] = (kinetic, sum over ordered pairs), in a fixed order.
// Bound by the FP64 pipe: 13 operations per unordered pair. 40,009 bodies: 8.93 ms before, 0.74 ms now.
__global__ void __launch_bounds__(kThreads) energy_f64_kernel(const float4 *__restrict__ bodies,
                                                              const float4 *__restrict__ vel, int64_t n, double eps,
                                                              int tiles, double *__restrict__ parts) {
    __shared__ double2 tile[2][kTile][2];
    __shared__ double red[2][kThreads];
    const int t = threadIdx.x, I = blockIdx.x;
    const int64_t i = (int64_t) I * kTile + t;
    const float4 p = i < n ? bodies[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const double px = p.x, py = p.y, pz = p.z;
    const int ring = tiles / 2 + 1 - ((tiles & 1) == 0 && I >= tiles / 2 ? 1 : 0);
    const int first = (int) ((int64_t) ring * blockIdx.y / gridDim.y), last = (int) ((int64_t) ring * (blockIdx.y + 1) / gridDim.y);
    auto fetch = [&](int o) {
        const int J = I + o < tiles ? I + o : I + o - tiles;
        return o < last ? load_source(bodies, (int64_t) J * kTile + t, n) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    double phi = 0.0;
    float4 next = fetch(first);
    int buf = 0;
    for (int o = first; o < last; ++o, buf ^= 1) {
        // a padding body has no mass: its term is zero
        tile[buf][t][0] = make_double2(next.x, next.y);
        tile[buf][t][1] = make_double2(next.z, next.w);
        __syncthreads();
        next = fetch(o + 1);
        const double2(*src)[2] = tile[buf];
        double sum = 0.0;
        auto term = [&](int k, auto may_be_far) {
            const double2 u = src[k][0], v = src[k][1];
            const double dx = u.x - px, dy = u.y - py, dz = v.x - pz;
            const double d2 = fma(dx, dx, fma(dy, dy, dz * dz));
            const double inv = rsqrt_f64<decltype(may_be_far)::value>(d2 + eps);
            sum = fma(v.y, __double2hiint(d2) == 0 ? 0.0 : inv, sum);
        };
        // a body at infinity makes the sum a NaN by the distance to itself, so only the softening matters here
        if (!isinf(eps)) {
#pragma unroll 8
            for (int k = 0; k < kTile; ++k) term(k, std::false_type());
        } else {
            for (int k = 0; k < kTile; ++k) term(k, std::true_type());
        }
        phi += o == 0 ? sum : 2.0 * sum;
    }
    const double m = p.w;
    double kinetic = 0.0;
    if (blockIdx.y == 0 && i < n) {
        const float4 v = vel[i];
        kinetic = 0.5 * m * ((double) v.x * v.x + (double) v.y * v.y + (double) v.z * v.z);
    }
    red[0][t] = kinetic;
    red[1][t] = i < n ? m * phi : 0.0;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (t < o) {
            red[0][t] += red[0][t + o];
            red[1][t] += red[1][t + o];
        }
        __syncthreads();
    }
    if (t == 0) {
        const int64_t b = (int64_t) blockIdx.y * gridDim.x + blockIdx.x;
        parts[2 * b] = red[0][0];
        parts[2 * b + 1] = red[1][0];
    }
}

// Sums the per-block parts in a fixed order: out = (kinetic, -G/2 * sum m_i phi_i).
__global__ void __launch_bounds__(kThreads) energy_sum_kernel(const double *__restrict__ parts, int64_t blocks, double G,
                                                              double *__restrict__ out) {
    __shared__ double red[2][kThreads];
    const int t = threadIdx.x;
    double k = 0.0, u = 0.0;
    for (int64_t b = t; b < blocks; b += kThreads) {
        k += parts[2 * b];
        u += parts[2 * b + 1];
    }
    red[0][t] = k;
    red[1][t] = u;
    __syncthreads();
    for (int o = kThreads / 2; o > 0; o >>= 1) {
        if (t < o) {
            red[0][t] += red[0][t + o];
            red[1][t] += red[1][t + o];
        }
        __syncthreads();
    }
    if (t == 0) {
        out[0] = red[0][0];
        out[1] = -0.5 * G * red[1][0];
    }
}

// Tiles of 256 bodies, and blocks per row of the energy kernel: enough for about 16 blocks per SM
// of a 148-SM part (a fixed number, so that the order of the sums does not depend on the device).
int energy_tiles(int64_t n) { return (int) ((n + kTile - 1) / kTile); }
int energy_rows(int64_t n) {
    const int64_t tiles = std::max(energy_tiles(n), 1);
    return (int) std::max<int64_t>(1, std::min<int64_t>(tiles / 2 + 1, (148 * 16 + tiles - 1) / tiles));
}

// Blocks that share the sources of 32 targets: enough for about twelve waves of four blocks per SM of
// a 148-SM part (one and a half waves take two waves' time), while each of a block's eight warps
// keeps 64 sources or more. Fixed numbers: the order of the sums does not depend on the device.
int cluster_for(int64_t target_blocks, int64_t n) {
    int c = 1;
    while (c < kMaxCluster && target_blocks * c < 12 * 148 * 4 && n / (2 * c * 8) >= 64) c *= 2;
    return c;
}

template<typename... Params, typename... Args>
void launch_clusters(void (*kernel)(Params...), int64_t target_blocks, int cluster, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (target_blocks * cluster));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned) cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// The wide form (Z = 1) reads sources once per 256 or 512 targets instead of once per 32 or 64, but its blocks are
// few and long: a wave that is begun costs a whole one. Where there are this many targets it pays, and, with few
// sources, where the warps' partial sums would cost as much as the sum. Measured, us, Z = 8 / Z = 1:
//   FP32, 32,768 sources: 150,000 targets 2144 / 2132, 304,000 4143 / 5023, 380,000 5159 / 5975, 450,000 6110 / 5969,
//     800,000 10799 / 10732
//   FP64, 4,096 sources: 310,000 1557 / 1690, 500,000 2490 / 2578, 700,000 3472 / 3467, 2 10^6 9884 / 9515
//   100 sources, FP32: 100,000 11.7 / 11.8, 200,000 18.8 / 16.0, 10^6 71 / 50, FP64: 100,000 23.8 / 22.5, 200,000 40.6 / 37.0;
//   300 sources, FP32: 100,000 20.1 / 25.9, 200,000 35.0 / 34.5
constexpr int64_t kWideTargets32 = 440000, kWideTargets64 = 700000;
bool wide_targets(int64_t targets, int64_t n, int64_t wide) { return targets >= (n <= 128 ? 100000 : wide); }
// From this many targets on, two per lane leave enough blocks. FP32, us, T = 1 / T = 2: 4,096 sources: 4,096 targets 16.9 /
// 17.3, 8,192 26.2 / 26.2, 20,000 53.1 / 48.7; 32,768 sources: 6,000 111 / 107, 8,192 147 / 139, 65,536 1039 / 942.
constexpr int64_t kPairTargets = 8192;

}  // namespace

int64_t energy_parts(int64_t n) { return 2 * (int64_t) std::max(energy_tiles(n), 1) * energy_rows(n) + 2; }

void launch_energy_f64(const float4 *bodies, const float4 *vel, int64_t n, double G, double eps, double *parts,
                       double *out, cudaStream_t s) {
    const int tiles = energy_tiles(n);
    const int rows = energy_rows(n);
    if (tiles > 0) energy_f64_kernel<<<dim3((unsigned) tiles, (unsigned) rows), kThreads, 0, s>>>(bodies, vel, n, eps, tiles, parts);
    energy_sum_kernel<<<1, kThreads, 0, s>>>(parts, (int64_t) tiles * rows, G, out);
}

void launch_direct_f32(const float4 *bodies, int64_t n, const float4 *targets, int64_t nt, int64_t shape_targets,
                       float G, float eps, float4 *acc, cudaStream_t s) {
    if (nt <= 0) return;
    auto launch = [&](auto narrow, auto soft, int per_block, int cluster) {
        launch_clusters(eps == 0.f ? narrow : soft, (nt + per_block - 1) / per_block, cluster, s, bodies, n, targets, nt, G,
                        eps, acc);
    };
    if (wide_targets(shape_targets, n, kWideTargets32))
        launch(direct_f32_kernel<true, 1, 2>, direct_f32_kernel<false, 1, 2>, 2 * kThreads, 1);
    else if (shape_targets >= kPairTargets)
        launch(direct_f32_kernel<true, 8, 2>, direct_f32_kernel<false, 8, 2>, 64, cluster_for((shape_targets + 63) / 64, n));
    else
        launch(direct_f32_kernel<true, 8, 1>, direct_f32_kernel<false, 8, 1>, 32, cluster_for((shape_targets + 31) / 32, n));
}

void launch_direct_f64(const float4 *bodies, int64_t n, const float4 *targets, int64_t nt, double G, double eps,
                       double *acc3, cudaStream_t s) {
    if (nt <= 0) return;
    if (wide_targets(nt, n, kWideTargets64)) {
        launch_clusters(direct_f64_kernel<1>, (nt + kThreads - 1) / kThreads, 1, s, bodies, n, targets, nt, G, eps, acc3);
    } else {
        const int64_t blocks = (nt + 31) / 32;
        launch_clusters(direct_f64_kernel<8>, blocks, cluster_for(blocks, n), s, bodies, n, targets, nt, G, eps, acc3);
    }
}

}  // namespace nbg
