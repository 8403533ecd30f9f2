// Barnes-Hut traversal of the preorder linear BVH for groups of 32 Morton-adjacent targets, one
// warp per group, in a persistent grid.
//
// Semantics are those of Descent::activeTree (src/NBody/Simulation/Solvers/Descent/activeTree.h:24-79)
// under DiagonalOverCenterDistance (DiagonalOverCenterDistance.h:18-22) with the Gravity rule
// (src/NBody/Physics/Rules/Gravity.h:199-259), decided per target: a node is approximated for a
// target iff diag^2 / |centre - p|^2 < theta^2 (the node carries the exact threshold on
// |centre - p|^2, and squared distances are formed in the reference's IEEE operation order), an
// opened leaf interacts pairwise with all its bodies, otherwise the children are visited. Every
// target therefore takes exactly the reference's decisions, and the interaction counts equal the
// reference's SimpleTrackingRule counts.
//
// Work organisation (per warp, 32 targets, 32-bit target masks):
//   1. Chunked traversal: up to 32 (node, mask) entries are popped from the warp's stack, one per
//      lane. Each lane classifies its node against the bounding box of the group's targets:
//        accept-all  if even the box point nearest the centre passes the MAC,
//        open-all    if even the farthest box corner fails it,
//        mixed       otherwise.
//      Rounding is monotone, so the rounded squared distance of every target lies between the
//      nearest and farthest values computed with the same operation sequence: the group decision
//      is exact for every target, not a heuristic.
//   2. Mixed nodes are batched and resolved lane-parallel: each lane takes one node and tests the
//      32 targets (broadcast from shared memory), producing accept and open masks.
//   3. Accepted nodes are staged in per-warp shared-memory slabs: the lane that accepted a node
//      copies its payload there asynchronously (cp.async), so the payload crosses L2 once per
//      group instead of once per target. Nodes accepted by every target go to the full slab, are
//      rewritten there as pair records and evaluated by all lanes with broadcast reads, two nodes per
//      paired FP32 instruction; nodes accepted by some targets go to the partial slab with their
//      target masks, and at evaluation a warp bit-matrix transpose of the masks gives every lane the
//      set of slab entries it owns, which it walks on its own. Opened leaves go to a (leaf, mask)
//      list, whose bodies are packed into shared-memory tiles of 32 and evaluated two per instruction;
//      opened internal nodes push both children.
//   4. Launches of few groups run the same walk with a team of eight warps per group
//      (bh_team_kernel): the walker hands its slabs and lists to the other warps.
//
// Arithmetic: FP32, one MUFU rsqrt per interaction, G applied once per target. Pair term:
// 20 flops by the usual direct-sum convention (12 FP32 instructions + rsqrt). Quadrupole node
// term (non-traceless moments about the centre of mass, Gravity.h:239-259, with D<3> contracted
// analytically: (D3:Q)_i = g3 R_i (R.Q.R) + g2 (2 (Q R)_i + R_i tr Q)): 56 flops.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <memory>
#include <new>

#include "nb_internal.cuh"

namespace nbg {

namespace {

// Launch shapes (autotuned per workload, see nb_set_traversal_shape): THREADS threads per block
// (128 or 256) and PART entries in the partial-accept slab (32 or 64). The launch bounds keep
// 1024 threads per SM resident (64 registers per thread).
constexpr int kResidentThreads = 1024;
constexpr int kList = 64;      // leaf and mixed lists: each round appends at most 32, evaluated above 32
constexpr int kFullSlab = 32;  // staged nodes accepted by the whole group
// Stack: kTraverseStack entries per warp. No bound below that size is proven for every tree, so a
// round whose pushes would not fit abandons its group and sets kErrStackOverflow (the host turns it
// into an error); every entry on the stack has been written, so no stale entry is ever popped.
constexpr unsigned kFull = 0xffffffffu;

enum : int { kNone = 0, kAcceptAll = 1, kOpenAll = 2, kMixed = 3 };

template<int PAY, int PART>
struct WarpSmem {
    float4 tpos[32];
    float4 full_pay[kFullSlab * PAY];  // payloads of group-wide accepted nodes
    float4 part_pay[(PART + 1) * PAY]; // payloads of partially accepted nodes, then the null payload
    uint32_t part_mask[PART];          // their target masks
    unsigned node_count[32], pair_count[32];  // the group's interactions per target
    int turn;                          // leaf set of the next list
    int pad[3];
    int pp_begin[kList], pp_end[kList];
    uint32_t pp_mask[kList];
    int mixed_node[kList];
    uint32_t mixed_mask[kList];
};

template<int ORDER, int THREADS, int PART>
constexpr size_t block_smem_bytes() {
    return sizeof(WarpSmem<NodeLayout<ORDER>::PAY, PART>) * (THREADS / 32);
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// 16-byte asynchronous global -> shared copy (completes at cp_async_wait_all).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const uint32_t s = (uint32_t) __cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Transpose of the 32 x 32 bit matrix whose row r is lane r's word: afterwards bit r of lane c's
// word is bit c of row r (five butterfly stages exchanging off-diagonal blocks).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const uint32_t hi = s == 16 ? 0xFFFF0000u : s == 8 ? 0xFF00FF00u : s == 4 ? 0xF0F0F0F0u
                          : s == 2 ? 0xCCCCCCCCu : 0xAAAAAAAAu;
        const uint32_t y = __shfl_xor_sync(kFull, x, s);
        x = (lane & s) ? ((x & hi) | ((y & hi) >> s)) : ((x & ~hi) | ((y & ~hi) << s));
    }
    return x;
}

// Squared distance in the reference's IEEE order: (dx*dx + dy*dy) + dz*dz, d = p - c.
__device__ __forceinline__ float ref_dist2(float px, float py, float pz, float4 c) {
    const float dx = fsub(px, c.x), dy = fsub(py, c.y), dz = fsub(pz, c.z);
    return fadd(fadd(fmul(dx, dx), fmul(dy, dy)), fmul(dz, dz));
}

template<bool EPS0>
__device__ __forceinline__ void pair_term(float4 p, float4 b, float eps, float &ax, float &ay, float &az) {
    const float rx = p.x - b.x, ry = p.y - b.y, rz = p.z - b.z;
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, fmaf(rz, rz, eps)));
    if (EPS0 && r2 == 0.f) return;  // equal positions contribute nothing (Gravity.h:203)
    const float inv = rsqrt_hw(r2);
    const float s = b.w * (inv * inv * inv);
    ax = fmaf(-rx, s, ax);
    ay = fmaf(-ry, s, ay);
    az = fmaf(-rz, s, az);
}

template<bool EPS0>
__device__ __forceinline__ void quad_term(float4 p, float4 com, float4 q0, float4 q1, float eps, float &ax,
                                          float &ay, float &az) {
    const float rx = p.x - com.x, ry = p.y - com.y, rz = p.z - com.z;
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, fmaf(rz, rz, eps)));
    if (EPS0 && r2 == 0.f) return;
    const float inv = rsqrt_hw(r2);
    const float inv2 = inv * inv;
    const float inv3 = inv2 * inv;
    const float inv5 = inv3 * inv2;
    const float inv7 = inv5 * inv2;
    const float qx = fmaf(q0.x, rx, fmaf(q0.y, ry, q0.z * rz));
    const float qy = fmaf(q0.y, rx, fmaf(q0.w, ry, q1.x * rz));
    const float qz = fmaf(q0.z, rx, fmaf(q1.x, ry, q1.y * rz));
    const float rqr = fmaf(rx, qx, fmaf(ry, qy, rz * qz));
    // q1.z holds 1.5 * (Qxx + Qyy + Qzz), precomputed per node
    const float sr = fmaf(-7.5f * inv7, rqr, fmaf(inv5, q1.z, -com.w * inv3));
    const float sq = 3.0f * inv5;
    ax = fmaf(rx, sr, fmaf(qx, sq, ax));
    ay = fmaf(ry, sr, fmaf(qy, sq, ay));
    az = fmaf(rz, sr, fmaf(qz, sq, az));
}

// Node term from a staged payload (PAY float4 in shared memory).
template<int ORDER, bool EPS0>
__device__ __forceinline__ void staged_term(const float4 *pc, float4 p, float eps, float &ax, float &ay, float &az) {
    if constexpr (ORDER == 1) {
        pair_term<EPS0>(p, pc[0], eps, ax, ay, az);
    } else {
        quad_term<EPS0>(p, pc[0], pc[1], pc[2], eps, ax, ay, az);
    }
}

template<int PAY>
__device__ __forceinline__ void stage_node(float4 *dst, const float4 *__restrict__ pay, int c) {
    const float4 *src = pay + (int64_t) c * PAY;
#pragma unroll
    for (int k = 0; k < PAY; ++k) cp_async16(dst + k, src + k);
}

// A target's sums are kept apart as one set for the approximated nodes and kLeafSets sets for the
// pairs of opened leaves (the q-th flushed list goes to set q % kLeafSets), each in the order of the
// flushed slabs and lists, and added at the end in set order. A set's terms and their order depend
// on the walk alone, so one warp (bh_kernel) and a team of warps that share the sets
// (bh_team_kernel) give the same bits.
constexpr int kLeafSets = 6;
constexpr int kLeafFlush = 32;  // a list of more leaves than this is flushed at the end of the round
static_assert(kLeafFlush + 32 <= kList, "a round appends at most 32 leaves");

// pair2_term with each body's factor set to zero where `on` is false.
template<bool EPS0>
__device__ __forceinline__ void masked_pair2(float2 npx, float2 npy, float2 npz, float2 eps2, float4 u, float4 v,
                                             bool on_a, bool on_b, float2 &ax, float2 &ay, float2 &az) {
    const float2 dx = __fadd2_rn(make_float2(u.x, u.y), npx);
    const float2 dy = __fadd2_rn(make_float2(u.z, u.w), npy);
    const float2 dz = __fadd2_rn(make_float2(v.x, v.y), npz);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
    float2 inv;
    inv.x = rsqrt_hw(r2.x);
    inv.y = rsqrt_hw(r2.y);
    float2 s = __fmul2_rn(make_float2(v.z, v.w), __fmul2_rn(__fmul2_rn(inv, inv), inv));
    s.x = on_a && !(EPS0 && r2.x == 0.f) ? s.x : 0.f;
    s.y = on_b && !(EPS0 && r2.y == 0.f) ? s.y : 0.f;
    ax = __ffma2_rn(dx, s, ax);
    ay = __ffma2_rn(dy, s, ay);
    az = __ffma2_rn(dz, s, az);
}

// Two quadrupole node terms at once in paired FP32 arithmetic, operand pairs as in pair2_term:
// u = (x_a, x_b, y_a, y_b), v = (z_a, z_b, M_a, M_b), then the moments Qxx, Qxy | Qxz, Qyy | Qyz, Qzz | 1.5 tr Q
// of both nodes. With d = com - p the terms of quad_term change sign in both factors.
template<bool EPS0>
__device__ __forceinline__ void quad2_term(float2 npx, float2 npy, float2 npz, float2 eps2, const float4 *rec,
                                           float2 &ax, float2 &ay, float2 &az) {
    const float4 u = rec[0], v = rec[1], q0 = rec[2], q1 = rec[3], q2 = rec[4];
    const float2 tr = *reinterpret_cast<const float2 *>(rec + 5);
    const float2 dx = __fadd2_rn(make_float2(u.x, u.y), npx);
    const float2 dy = __fadd2_rn(make_float2(u.z, u.w), npy);
    const float2 dz = __fadd2_rn(make_float2(v.x, v.y), npz);
    const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
    float2 inv;
    inv.x = rsqrt_hw(r2.x);
    inv.y = rsqrt_hw(r2.y);
    if (EPS0) {
        if (r2.x == 0.f) inv.x = 0.f;
        if (r2.y == 0.f) inv.y = 0.f;
    }
    const float2 inv2 = __fmul2_rn(inv, inv), inv3 = __fmul2_rn(inv2, inv);
    const float2 inv5 = __fmul2_rn(inv3, inv2), inv7 = __fmul2_rn(inv5, inv2);
    const float2 xx = make_float2(q0.x, q0.y), xy = make_float2(q0.z, q0.w), xz = make_float2(q1.x, q1.y);
    const float2 yy = make_float2(q1.z, q1.w), yz = make_float2(q2.x, q2.y), zz = make_float2(q2.z, q2.w);
    const float2 qx = __ffma2_rn(xx, dx, __ffma2_rn(xy, dy, __fmul2_rn(xz, dz)));
    const float2 qy = __ffma2_rn(xy, dx, __ffma2_rn(yy, dy, __fmul2_rn(yz, dz)));
    const float2 qz = __ffma2_rn(xz, dx, __ffma2_rn(yz, dy, __fmul2_rn(zz, dz)));
    const float2 dqd = __ffma2_rn(dx, qx, __ffma2_rn(dy, qy, __fmul2_rn(dz, qz)));
    const float2 mono = __fmul2_rn(make_float2(v.z, v.w), inv3);
    const float2 sr = __ffma2_rn(__fmul2_rn(make_float2(7.5f, 7.5f), inv7), dqd,
                                 __ffma2_rn(make_float2(-tr.x, -tr.y), inv5, mono));
    const float2 sq = __fmul2_rn(make_float2(-3.0f, -3.0f), inv5);
    ax = __ffma2_rn(dx, sr, __ffma2_rn(qx, sq, ax));
    ay = __ffma2_rn(dy, sr, __ffma2_rn(qy, sq, ay));
    az = __ffma2_rn(dz, sr, __ffma2_rn(qz, sq, az));
}

// Staged nodes accepted by the whole group (n <= 32, one payload per slot): the slots are rewritten
// as pair records in place, a null payload filling an odd last one, and every lane evaluates every
// pair (broadcast reads).
template<int ORDER, bool EPS0>
__device__ __forceinline__ void full_terms(float4 *pay, int n, float4 p, float eps, int lane, float &ax, float &ay,
                                           float &az) {
    constexpr int PAY = NodeLayout<ORDER>::PAY;
    float4 c[PAY];
#pragma unroll
    for (int k = 0; k < PAY; ++k) c[k] = k == 0 ? make_float4(1e30f, 1e30f, 1e30f, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane < n) {
#pragma unroll
        for (int k = 0; k < PAY; ++k) c[k] = pay[lane * PAY + k];
    }
    __syncwarp();
    if (lane <= n && lane < 32) {
        float *rec = reinterpret_cast<float *>(pay + (lane & ~1) * PAY) + (lane & 1);
#pragma unroll
        for (int k = 0; k < PAY; ++k) {
            rec[8 * k] = c[k].x;
            rec[8 * k + 2] = c[k].y;
            rec[8 * k + 4] = c[k].z;
            rec[8 * k + 6] = c[k].w;
        }
    }
    __syncwarp();
    const float2 npx = make_float2(-p.x, -p.x), npy = make_float2(-p.y, -p.y), npz = make_float2(-p.z, -p.z);
    const float2 eps2 = make_float2(eps, eps);
    float2 sx = make_float2(ax, 0.f), sy = make_float2(ay, 0.f), sz = make_float2(az, 0.f);
    for (int j = 0; j < n; j += 2) {
        const float4 *rec = pay + j * PAY;
        if constexpr (ORDER == 1) pair2_term<EPS0>(npx, npy, npz, eps2, rec[0], rec[1], sx, sy, sz);
        else quad2_term<EPS0>(npx, npy, npz, eps2, rec, sx, sy, sz);
    }
    ax = sx.x + sx.y;
    ay = sy.x + sy.y;
    az = sz.x + sz.y;
}

// The bodies of a list of opened leaves (n ranges [begin, end) with target masks) for every target.
// They are packed back to back into tiles of 32, stored as 16 interleaved pairs (two bodies per paired
// FP32 instruction) in shared memory (512 bytes); the transposed masks tell each lane which bodies of
// the tile its target takes, and the others' factors are set to zero. A tile's bodies are loaded,
// one per lane, while the tile before it is evaluated: the way through the tile's leaves only settles each
// lane's index, and one load follows it. A predicated load per leaf took longer where leaves are small
// (traversal of 2^20 bodies 15.43 -> 15.16 ms at leaf 16, 14.9 -> 14.7 at leaf 8; a step of 256 instances
// 76.1 -> 74.8 ms at leaf 8, 78.5 -> 77.2 at leaf 16); a prefix sum over the list instead of the way through
// it spills registers in bh_kernel (18.8 ms). Returns the lane's number of pairs.
template<bool EPS0>
__device__ __forceinline__ unsigned leaf_terms(const int *begin, const int *end, const uint32_t *mask, int n,
                                               const float4 *__restrict__ bodies, float4 *tile, float4 p, float eps,
                                               int lane, float &ax, float &ay, float &az) {
    unsigned pairs = 0;
    int j = 0, o = n > 0 ? begin[0] : 0, e = n > 0 ? end[0] : 0, fill = 0;
    float4 body;
    uint32_t who;
    auto fetch = [&]() {
        int from = 0, leaf = 0;
        fill = 0;
        while (j < n) {
            if (lane >= fill) {  // a later leaf of the tile takes over its lanes
                from = o + (lane - fill);
                leaf = j;
            }
            const int take = min(e - o, 32 - fill);
            fill += take;
            o += take;
            if (o < e) break;
            if (++j < n) {
                o = begin[j];
                e = end[j];
            }
            if (fill == 32) break;
        }
        body = make_float4(0.f, 0.f, 0.f, 0.f);
        who = 0u;
        if (lane < fill) {
            body = __ldg(bodies + from);
            who = mask[leaf];
        }
    };
    fetch();
    const float2 npx = make_float2(-p.x, -p.x), npy = make_float2(-p.y, -p.y), npz = make_float2(-p.z, -p.z);
    const float2 eps2 = make_float2(eps, eps);
    float2 sx = make_float2(ax, 0.f), sy = make_float2(ay, 0.f), sz = make_float2(az, 0.f);
    while (fill > 0) {
        const int m = fill;
        uint32_t bits = transpose32(who, lane);
        pairs += __popc(bits);
        float *f = reinterpret_cast<float *>(tile) + (lane >> 1) * 8 + (lane & 1);
        f[0] = body.x;
        f[2] = body.y;
        f[4] = body.z;
        f[6] = body.w;
        __syncwarp();
        fetch();
        for (int b = 0; b < m; b += 4, bits >>= 4) {
            const float4 u0 = tile[b], v0 = tile[b + 1], u1 = tile[b + 2], v1 = tile[b + 3];
            masked_pair2<EPS0>(npx, npy, npz, eps2, u0, v0, bits & 1u, bits & 2u, sx, sy, sz);
            masked_pair2<EPS0>(npx, npy, npz, eps2, u1, v1, bits & 4u, bits & 8u, sx, sy, sz);
        }
        __syncwarp();
    }
    ax = sx.x + sx.y;
    ay = sy.x + sy.y;
    az = sz.x + sz.y;
    return pairs;
}

// Staged nodes accepted by some targets only: the masks are transposed so that each lane holds the
// set of entries it evaluates, then every lane walks its own set. null is the slot of the null payload.
// Returns the lane's number of entries.
template<int ORDER, bool EPS0, int PART>
__device__ __forceinline__ unsigned part_terms(const float4 *pay, const uint32_t *mask, int n, float4 p, float eps,
                                               int lane, float &ax, float &ay, float &az) {
    constexpr int PAY = NodeLayout<ORDER>::PAY;
    uint32_t b0 = transpose32(lane < n ? mask[lane] : 0u, lane);
    uint32_t b1 = 0u;
    if constexpr (PART > 32) b1 = n > 32 ? transpose32(lane + 32 < n ? mask[lane + 32] : 0u, lane) : 0u;
    const unsigned taken = (unsigned) (__popc(b0) + __popc(b1));
    // a lane whose set is used up evaluates the null payload instead of branching around the term
    while (__any_sync(kFull, (b0 | b1) != 0u)) {
        int j = PART;
        if (b0) {
            j = __ffs(b0) - 1;
            b0 &= b0 - 1;
        } else if (b1) {
            j = 31 + __ffs(b1);
            b1 &= b1 - 1;
        }
        staged_term<ORDER, EPS0>(pay + j * PAY, p, eps, ax, ay, az);
    }
    return taken;
}

// The null payload: no mass and no moments at 1e30 on every axis, where the squared distance from
// any target with coordinates below 1e29 in magnitude overflows to infinity, so that every factor of
// the term is exactly zero and it adds nothing.
template<int PAY>
__device__ __forceinline__ void write_null_payload(float4 *slot, int lane) {
    if (lane < PAY) slot[lane] = lane == 0 ? make_float4(1e30f, 1e30f, 1e30f, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// Where a walk's findings go in bh_kernel: staged in the warp's slabs and evaluated by the warp
// itself when a slab or list could overflow. The node set is kept in registers; the leaf sets stay
// in global scratch (L2) and the interaction counts in shared memory between flushes.
template<int ORDER, bool EPS0, int PART>
struct WarpSink {
    static constexpr int PAY = NodeLayout<ORDER>::PAY;
    WarpSmem<PAY, PART> &S;
    const float4 *__restrict__ pay;
    const float4 *__restrict__ bodies;
    float4 p;
    float eps;
    int lane, n_bodies;
    int nfull = 0, npart = 0, npp = 0;
    float ax = 0.f, ay = 0.f, az = 0.f;  // the node set
    float *sets;  // kLeafSets x 3 x 32 floats of the warp's global scratch

    __device__ __forceinline__ void clear() {
        for (int k = 0; k < 3 * kLeafSets; ++k) sets[k * 32 + lane] = 0.f;
        S.node_count[lane] = S.pair_count[lane] = 0u;
        if (lane == 0) S.turn = 0;
    }
    __device__ __forceinline__ void flush_full() {
        cp_async_wait_all();
        __syncwarp();
        full_terms<ORDER, EPS0>(S.full_pay, nfull, p, eps, lane, ax, ay, az);
        S.node_count[lane] += (unsigned) nfull;
        nfull = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void flush_part() {
        cp_async_wait_all();
        __syncwarp();
        S.node_count[lane] += part_terms<ORDER, EPS0, PART>(S.part_pay, S.part_mask, npart, p, eps, lane, ax, ay, az);
        npart = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void flush_leaves() {
        if (nfull > 0) flush_full();  // the full slab's memory holds the tiles
        float *mine = sets + S.turn * 96 + lane;
        float sx = mine[0], sy = mine[32], sz = mine[64];
        const unsigned pairs = leaf_terms<EPS0>(S.pp_begin, S.pp_end, S.pp_mask, npp, bodies, S.full_pay, p, eps, lane,
                                                sx, sy, sz);
        mine[0] = sx;
        mine[32] = sy;
        mine[64] = sz;
        S.pair_count[lane] += pairs;
        npp = 0;
        __syncwarp();
        if (lane == 0) S.turn = S.turn + 1 < kLeafSets ? S.turn + 1 : 0;
        __syncwarp();
    }
    // accepted by every target / by the targets in mk (b: the ballot of on)
    __device__ __forceinline__ void add_full(bool on, uint32_t b, uint32_t lt, int c) {
        if (nfull + __popc(b) > kFullSlab) flush_full();
        if (on) stage_node<PAY>(S.full_pay + (nfull + __popc(b & lt)) * PAY, pay, c);
        nfull += __popc(b);
    }
    __device__ __forceinline__ void add_part(bool on, uint32_t b, uint32_t lt, int c, uint32_t mk) {
        if (npart + __popc(b) > PART) flush_part();
        if (on) {
            const int slot = npart + __popc(b & lt);
            stage_node<PAY>(S.part_pay + slot * PAY, pay, c);
            S.part_mask[slot] = mk;
        }
        npart += __popc(b);
    }
    __device__ __forceinline__ void add_leaf(bool on, uint32_t b, uint32_t lt, int l0, int l1, uint32_t mk) {
        if (on) {
            const int pos = npp + __popc(b & lt);
            S.pp_begin[pos] = min(max(l0, 0), n_bodies);
            S.pp_end[pos] = max(S.pp_begin[pos], min(l1, n_bodies));
            S.pp_mask[pos] = mk;
        }
        npp += __popc(b);
    }
    // each round appends at most 32 leaves: evaluated before the next one could overflow the list
    __device__ __forceinline__ void end_round() {
        if (npp > kLeafFlush) flush_leaves();
    }
    __device__ __forceinline__ void finish() {
        flush_full();
        flush_part();
        if (npp > 0) flush_leaves();
        for (int k = 0; k < kLeafSets; ++k) {
            const float *mine = sets + k * 96 + lane;
            ax += mine[0];
            ay += mine[32];
            az += mine[64];
        }
    }
};

// Where they go in bh_team_kernel: the same lists, handed to the team's other warps at the same
// points at which bh_kernel evaluates them.
struct NodeList {
    int count, all;  // all: accepted by every target; count < 0: the walk is done
    int node[64];
    uint32_t mask[64];
};
struct LeafList {
    int count, pad;
    int begin[kList], end[kList];
    uint32_t mask[kList];
};
constexpr int kRing = 4;                     // node lists in flight; leaf lists: kLeafRing
constexpr int kLeafRing = 8;
constexpr int kTeamWarps = 2 + kLeafSets;    // walker, node evaluator, one warp per leaf set
constexpr int kTeamThreads = 32 * kTeamWarps;
constexpr int kTeamBlocks = 4;               // resident per SM, by shared memory
// Limit of one wait. The longest that a sound pass can need is one warp's evaluation of a list that holds every
// body (coincident bodies make one leaf): about 4 s at 3e8 bodies.
constexpr unsigned long long kTeamWaitNs = 10000000000ull;

template<int PAY, int PART>
struct TeamSmem {
    int2 stack[kTraverseStack];
    float4 tpos[32];
    float4 pay[(PART + 1) * PAY];            // (at least 32) the node evaluator's staged payloads, then the null payload
    float4 tile[kLeafSets][32];              // the leaf warps' source bodies
    NodeList nodes[kRing];
    LeafList leaf[kLeafRing];
    int full_node[kFullSlab];                // the walker's open lists
    int part_node[PART];
    uint32_t part_mask[PART];
    int pp_begin[kList], pp_end[kList];
    uint32_t pp_mask[kList];
    int mixed_node[kList];
    uint32_t mixed_mask[kList];
    unsigned long long node_ready[kRing], node_free[kRing], leaf_ready[kLeafRing], leaf_free[kLeafRing];  // mbarriers
    int abandon;                             // a wait ran out: every warp leaves
};

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t) __cvta_generic_to_shared(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"((uint32_t) __cvta_generic_to_shared(bar)) : "memory");
}
// One try suspends the warp for at most kTryNs (a hint: without it the time is the system's choice).
constexpr unsigned kTryNs = 20000;
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2, %3;\n selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(ok) : "r"((uint32_t) __cvta_generic_to_shared(bar)), "r"(parity), "r"(kTryNs) : "memory");
    return ok != 0;
}
// Waits until the barrier's phase `parity` is over, at most limit_ns and not once the team is abandoned. A
// wait that runs out abandons the team with kErrTeamTimeout. Uniform over the warp.
__device__ __forceinline__ bool team_wait(unsigned long long *bar, unsigned parity, int *abandon, uint32_t *err,
                                          unsigned long long limit_ns) {
    if (__all_sync(kFull, mbar_try_wait(bar, parity))) return true;
    const unsigned long long t0 = global_timer_ns();
    for (;;) {
        if (__any_sync(kFull, *(volatile int *) abandon != 0)) return false;
        if (__any_sync(kFull, global_timer_ns() - t0 > limit_ns)) break;
        if (__all_sync(kFull, mbar_try_wait(bar, parity))) return true;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicOr(err, (uint32_t) kErrTeamTimeout);
        *(volatile int *) abandon = 1;
    }
    __syncwarp();
    return false;
}

template<int ORDER, int PART>
struct TeamSink {
    static constexpr int PAY = NodeLayout<ORDER>::PAY;
    TeamSmem<PAY, PART> &S;
    uint32_t *err;
    unsigned long long limit_ns;  // of each wait
    int lane, n_bodies;
    int nfull = 0, npart = 0, npp = 0;
    int node_lists = 0, leaf_lists = 0;  // lists handed over
    bool lost = false;                   // the team was abandoned: nothing is handed over any more

    __device__ __forceinline__ NodeList *open_nodes() {
        const int slot = node_lists % kRing, turn = node_lists / kRing;
        if (lost || (turn > 0 && !team_wait(&S.node_free[slot], (turn - 1) & 1, &S.abandon, err, limit_ns))) {
            lost = true;
            return nullptr;
        }
        return &S.nodes[slot];
    }
    __device__ __forceinline__ void hand_nodes() {
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.node_ready[node_lists % kRing]);
        ++node_lists;
    }
    __device__ __forceinline__ void flush_full() {
        if (nfull > 0)
            if (NodeList *l = open_nodes()) {
                if (lane == 0) {
                    l->count = nfull;
                    l->all = 1;
                }
                if (lane < nfull) l->node[lane] = S.full_node[lane];
                hand_nodes();
            }
        nfull = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void flush_part() {
        if (npart > 0)
            if (NodeList *l = open_nodes()) {
                if (lane == 0) {
                    l->count = npart;
                    l->all = 0;
                }
                for (int k = lane; k < npart; k += 32) {
                    l->node[k] = S.part_node[k];
                    l->mask[k] = S.part_mask[k];
                }
                hand_nodes();
            }
        npart = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void hand_leaves(int count) {
        const int slot = leaf_lists % kLeafRing, turn = leaf_lists / kLeafRing;
        if (lost || (turn > 0 && !team_wait(&S.leaf_free[slot], (turn - 1) & 1, &S.abandon, err, limit_ns))) {
            lost = true;
            return;
        }
        LeafList &l = S.leaf[slot];
        if (lane == 0) l.count = count;
        for (int k = lane; k < count; k += 32) {
            l.begin[k] = S.pp_begin[k];
            l.end[k] = S.pp_end[k];
            l.mask[k] = S.pp_mask[k];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.leaf_ready[slot]);
        ++leaf_lists;
    }
    __device__ __forceinline__ void flush_leaves() {
        flush_full();  // as the one-warp form does
        if (npp > 0) hand_leaves(npp);
        npp = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void add_full(bool on, uint32_t b, uint32_t lt, int c) {
        if (nfull + __popc(b) > kFullSlab) flush_full();
        if (on) S.full_node[nfull + __popc(b & lt)] = c;
        nfull += __popc(b);
    }
    __device__ __forceinline__ void add_part(bool on, uint32_t b, uint32_t lt, int c, uint32_t mk) {
        if (npart + __popc(b) > PART) flush_part();
        if (on) {
            const int slot = npart + __popc(b & lt);
            S.part_node[slot] = c;
            S.part_mask[slot] = mk;
        }
        npart += __popc(b);
    }
    __device__ __forceinline__ void add_leaf(bool on, uint32_t b, uint32_t lt, int l0, int l1, uint32_t mk) {
        if (on) {
            const int pos = npp + __popc(b & lt);
            S.pp_begin[pos] = min(max(l0, 0), n_bodies);
            S.pp_end[pos] = max(S.pp_begin[pos], min(l1, n_bodies));
            S.pp_mask[pos] = mk;
        }
        npp += __popc(b);
    }
    __device__ __forceinline__ void end_round() {
        if (npp > kLeafFlush) flush_leaves();
    }
    // the last lists, then one for each other warp that ends its work
    __device__ __forceinline__ void finish() {
        flush_full();
        flush_part();
        flush_leaves();
        if (NodeList *l = open_nodes()) {
            if (lane == 0) l->count = -1;
            hand_nodes();
        }
        for (int set = 0; set < kLeafSets; ++set) hand_leaves(-1);
    }
};

// Classified entries of one round, appended to the sink's lists (warp-uniform control flow):
// acc / part are accepted nodes (target mask mk for part), leaf is an opened leaf (body range
// l0..l1, mask mk), open an opened internal node (children c + 1 and l0, mask mk), mixed a node
// still to be resolved per target.
template<class Sink>
__device__ __forceinline__ bool dispatch(Sink &sink, int2 *stack, int *mixed_node, uint32_t *mixed_mask, bool acc,
                                         bool part, bool leaf, bool open, bool mixed, int c, uint32_t mk, int l0,
                                         int l1, uint32_t lt, int lane, int &nmixed, int &top, uint32_t *err) {
    uint32_t b = __ballot_sync(kFull, acc);
    if (b) sink.add_full(acc, b, lt, c);
    b = __ballot_sync(kFull, part);
    if (b) sink.add_part(part, b, lt, c, mk);
    b = __ballot_sync(kFull, leaf);
    sink.add_leaf(leaf, b, lt, l0, l1, mk);
    b = __ballot_sync(kFull, mixed);
    if (mixed) {
        const int pos = nmixed + __popc(b & lt);
        mixed_node[pos] = c;
        mixed_mask[pos] = mk;
    }
    nmixed += __popc(b);
    b = __ballot_sync(kFull, open);
    bool abandoned = false;
    if (top + 2 * __popc(b) > kTraverseStack) {
        // a push would not fit: the group is abandoned with an error (warp-uniform)
        if (lane == 0) atomicOr(err, (uint32_t) kErrStackOverflow);
        abandoned = true;
    } else {
        if (open) {
            const int sp = top + 2 * __popc(b & lt);
            stack[sp] = make_int2(l0, (int) mk);         // right child
            stack[sp + 1] = make_int2(c + 1, (int) mk);  // left child, popped first
        }
        top += 2 * __popc(b);
    }
    __syncwarp();
    sink.end_round();
    return abandoned;
}

// The walk of one group from `root` by one warp: `full` masks its valid targets, lo / hi is their
// box, tpos their positions.
template<class Sink>
__device__ __forceinline__ void walk(Sink &sink, const NodeArrays &nodes, int num_nodes, int root, uint32_t full,
                                     const float lo[3], const float hi[3], const float4 *tpos, int2 *stack,
                                     int *mixed_node, uint32_t *mixed_mask, int64_t round_limit, uint32_t lt, int lane,
                                     uint32_t *err) {
    const float4 *__restrict__ mac = nodes.mac;
    const int2 *__restrict__ link = nodes.link;
    int top = 0, nmixed = 0;
    if (num_nodes > 0 && root >= 0 && root < num_nodes) {
        if (lane == 0) stack[0] = make_int2(root, (int) full);
        top = 1;
    } else if (num_nodes > 0 && lane == 0) {
        atomicOr(err, (uint32_t) kErrTraverseLimit);  // a group without a valid tree root
    }
    __syncwarp();
    int64_t rounds = 0;
    while (top > 0 || nmixed > 0) {
        if (++rounds > round_limit) {
            if (lane == 0) atomicOr(err, (uint32_t) kErrTraverseLimit);
            break;
        }
        if (top > 0) {
            // ---- 1. pop up to 32 entries and classify them lane-parallel ----
            const int k = min(32, top);
            const int base = top - k;
            top = base;
            int c = 0, l0 = 0, l1 = -1, cls = kNone;
            uint32_t m = 0;
            if (lane < k) {
                const int2 e = stack[base + lane];
                c = e.x;
                m = (uint32_t) e.y;
                const float4 mc = __ldg(mac + c);
                const int2 lk = __ldg(link + c);
                l0 = lk.x;
                l1 = lk.y;
                // nearest box point and farthest box corner, per axis, with the reference's rounding
                const float nx = fsub(fminf(fmaxf(mc.x, lo[0]), hi[0]), mc.x);
                const float ny = fsub(fminf(fmaxf(mc.y, lo[1]), hi[1]), mc.y);
                const float nz = fsub(fminf(fmaxf(mc.z, lo[2]), hi[2]), mc.z);
                const float fx = fmaxf(fabsf(fsub(lo[0], mc.x)), fabsf(fsub(hi[0], mc.x)));
                const float fy = fmaxf(fabsf(fsub(lo[1], mc.y)), fabsf(fsub(hi[1], mc.y)));
                const float fz = fmaxf(fabsf(fsub(lo[2], mc.z)), fabsf(fsub(hi[2], mc.z)));
                const float dmin2 = fadd(fadd(fmul(nx, nx), fmul(ny, ny)), fmul(nz, nz));
                const float dmax2 = fadd(fadd(fmul(fx, fx), fmul(fy, fy)), fmul(fz, fz));
                if (!(mc.w == mc.w)) cls = kOpenAll;  // NaN threshold: never approximated
                else if (dmin2 >= mc.w) cls = kAcceptAll;
                else if (dmax2 < mc.w) cls = kOpenAll;
                else cls = kMixed;
            }
            __syncwarp();  // popped entries are read before children overwrite them
            const bool is_leaf_open = cls == kOpenAll && l1 >= 0;
            const bool is_int_open = cls == kOpenAll && l1 < 0 && l0 > c + 1 && l0 < num_nodes;
            if (cls == kOpenAll && l1 < 0 && !is_int_open) atomicOr(err, (uint32_t) kErrTraverseLimit);
            if (dispatch(sink, stack, mixed_node, mixed_mask, cls == kAcceptAll && m == full,
                         cls == kAcceptAll && m != full, is_leaf_open, is_int_open, cls == kMixed, c, m, l0, l1, lt,
                         lane, nmixed, top, err)) {
                top = 0;
                nmixed = 0;
            }
        }
        if (nmixed >= 32 || (top == 0 && nmixed > 0)) {
            // ---- 2. resolve up to 32 mixed nodes: per-target MAC, lane-parallel over nodes ----
            const int k = min(32, nmixed);
            const int base = nmixed - k;
            nmixed = base;
            int c = 0, l0 = 0, l1 = -1;
            uint32_t A = 0, O = 0;
            if (lane < k) {
                c = mixed_node[base + lane];
                const uint32_t m = mixed_mask[base + lane];
                const float4 mc = __ldg(mac + c);
                const int2 lk = __ldg(link + c);
                l0 = lk.x;
                l1 = lk.y;
                uint32_t bits = 0;
#pragma unroll 8
                for (int t = 0; t < 32; ++t) {
                    const float4 tp = tpos[t];
                    bits |= (ref_dist2(tp.x, tp.y, tp.z, mc) >= mc.w) ? (1u << t) : 0u;
                }
                A = bits & m;
                O = m & ~A;
            }
            __syncwarp();
            const bool is_int_open = O != 0 && l1 < 0 && l0 > c + 1 && l0 < num_nodes;
            if (O != 0 && l1 < 0 && !is_int_open) atomicOr(err, (uint32_t) kErrTraverseLimit);
            const bool is_acc = A != 0 && A == full;
            const bool is_part = A != 0 && A != full;
            // an entry can be accepted by some targets and opened by others: append both parts
            if (dispatch(sink, stack, mixed_node, mixed_mask, is_acc, is_part, false, false, false, c, A, l0, l1, lt,
                         lane, nmixed, top, err) ||
                dispatch(sink, stack, mixed_node, mixed_mask, false, false, O != 0 && l1 >= 0, is_int_open, false, c,
                         O, l0, l1, lt, lane, nmixed, top, err)) {
                top = 0;
                nmixed = 0;
            }
        }
    }
}

// Per axis, the box of the warp's valid targets (every lane gets it).
__device__ __forceinline__ void target_box(float4 p, bool valid, float lo[3], float hi[3]) {
    lo[0] = valid ? p.x : FLT_MAX; lo[1] = valid ? p.y : FLT_MAX; lo[2] = valid ? p.z : FLT_MAX;
    hi[0] = valid ? p.x : -FLT_MAX; hi[1] = valid ? p.y : -FLT_MAX; hi[2] = valid ? p.z : -FLT_MAX;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(kFull, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(kFull, hi[k], o));
        }
    }
}

// Adds a group's (particle-particle, node-particle) interactions to the pass's and its instance's.
__device__ __forceinline__ void add_counts(unsigned long long *counts, unsigned long long *inst_counts, int inst,
                                           unsigned pp, unsigned np) {
    if (counts) {
        atomicAdd(counts + 0, (unsigned long long) pp);
        atomicAdd(counts + 1, (unsigned long long) np);
    }
    if (inst_counts && inst >= 0) {
        atomicAdd(inst_counts + 2 * (int64_t) inst, (unsigned long long) pp);
        atomicAdd(inst_counts + 2 * (int64_t) inst + 1, (unsigned long long) np);
    }
}

// A valid tree needs fewer chunk rounds than it has nodes for one group; the cap only bounds the
// work on a corrupted tree.
__device__ __forceinline__ int64_t walk_rounds(int num_nodes) { return 4 * (int64_t) num_nodes + 64; }

template<int ORDER, bool EPS0, int THREADS, int PART>
__global__ void __launch_bounds__(THREADS, kResidentThreads / THREADS) bh_kernel(NodeArrays nodes, const int *__restrict__ num_nodes_p,
                                                         const float4 *__restrict__ bodies, int n_bodies,
                                                         const float4 *__restrict__ targets, int n_targets, float G,
                                                         float eps, float4 *__restrict__ acc,
                                                         unsigned long long *__restrict__ counts,
                                                         int2 *__restrict__ stack_base,
                                                         unsigned *__restrict__ group_counter,
                                                         uint32_t *__restrict__ err, const int4 *__restrict__ groups,
                                                         int num_group_tasks, const int *__restrict__ inst_root,
                                                         unsigned long long *__restrict__ inst_counts) {
    constexpr int PAY = NodeLayout<ORDER>::PAY;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WarpSmem<PAY, PART> &S = reinterpret_cast<WarpSmem<PAY, PART> *>(smem_raw)[warp];
    int2 *stack = stack_base + ((int64_t) blockIdx.x * (THREADS / 32) + warp) * kWarpScratch;
    const int num_nodes = *num_nodes_p;
    const int num_groups = groups ? num_group_tasks : (n_targets + 31) / 32;
    const uint32_t lt = lanemask_lt();
    const int64_t round_limit = walk_rounds(num_nodes);

    while (true) {
        int g = 0;
        if (lane == 0) g = (int) atomicAdd(group_counter, 1u);
        g = __shfl_sync(kFull, g, 0);
        if (g >= num_groups) break;
        int first = g * 32, count = min(32, n_targets - g * 32), root = 0, inst = -1;
        if (groups) {
            const int4 ge = groups[g];
            first = ge.x;
            count = ge.y;
            inst = ge.z;
            root = inst_root[inst];
        }
        const int i = first + lane;
        const bool valid = lane < count && i < n_targets;
        const float4 p = valid ? targets[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const uint32_t full = __ballot_sync(kFull, valid);
        float lo[3], hi[3];
        target_box(p, valid, lo, hi);
        S.tpos[lane] = p;
        write_null_payload<PAY>(S.part_pay + PART * PAY, lane);
        WarpSink<ORDER, EPS0, PART> sink{S, nodes.pay, bodies, p, eps, lane, n_bodies};
        sink.sets = reinterpret_cast<float *>(stack + kTraverseStack);
        sink.clear();
        walk(sink, nodes, num_nodes, root, full, lo, hi, S.tpos, stack, S.mixed_node, S.mixed_mask, round_limit, lt,
             lane, err);
        sink.finish();
        if (valid) acc[i] = make_float4(G * sink.ax, G * sink.ay, G * sink.az, 0.f);
        // interaction counts of the valid targets
        const unsigned spp = __reduce_add_sync(kFull, valid ? S.pair_count[lane] : 0u);
        const unsigned snp = __reduce_add_sync(kFull, valid ? S.node_count[lane] : 0u);
        if (lane == 0) add_counts(counts, inst_counts, inst, spp, snp);
        __syncwarp();
    }
}

// One block per group, for launches whose groups alone do not fill the GPU (team_groups): warp 0 walks, warp 1
// evaluates the approximated nodes, warp 2 + k the leaf lists of set k. Bound by the walk's chain of
// rounds (two dependent loads and several hundred instructions each); with one warp per group the
// leaf pairs came on top of it at 6 to 11 cycles per instruction, one warp per scheduler. Traversal
// time, one warp / team: 1,023-body Plummer 92 / 40 us, 10,000-body ball 427 / 115 us, 10,000-body
// Plummer 607 / 135 us, 100,003 bodies at leaf 64 and theta 0.3 6.7 / 3.9 ms.
template<int ORDER, bool EPS0, int PART>
__global__ void __launch_bounds__(kTeamThreads, kTeamBlocks)
    bh_team_kernel(NodeArrays nodes, const int *__restrict__ num_nodes_p, const float4 *__restrict__ bodies, int n_bodies,
                   const float4 *__restrict__ targets, int n_targets, float G, float eps, float4 *__restrict__ acc,
                   unsigned long long *__restrict__ counts, uint32_t *__restrict__ err, const int4 *__restrict__ groups,
                   const int *__restrict__ inst_root, unsigned long long *__restrict__ inst_counts,
                   unsigned long long wait_limit_ns) {
    constexpr int PAY = NodeLayout<ORDER>::PAY;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TeamSmem<PAY, PART> &S = *reinterpret_cast<TeamSmem<PAY, PART> *>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.x;
    int first = g * 32, count = min(32, n_targets - g * 32), root = 0, inst = -1;
    if (groups) {
        const int4 ge = groups[g];
        first = ge.x;
        count = ge.y;
        inst = ge.z;
        root = inst_root[inst];
    }
    const int i = first + lane;
    const bool valid = lane < count && i < n_targets;
    const float4 p = valid ? targets[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x == 0) {
        for (int k = 0; k < kRing; ++k) {
            mbar_init(&S.node_ready[k], 1);
            mbar_init(&S.node_free[k], 1);
        }
        for (int k = 0; k < kLeafRing; ++k) {
            mbar_init(&S.leaf_ready[k], 1);
            mbar_init(&S.leaf_free[k], 1);
        }
        S.abandon = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) S.tpos[lane] = p;
    if (warp == 1) write_null_payload<PAY>(S.pay + PART * PAY, lane);
    __syncthreads();

    float ax = 0.f, ay = 0.f, az = 0.f;
    unsigned taken = 0;
    if (warp == 0) {
        const int num_nodes = *num_nodes_p;
        const uint32_t full = __ballot_sync(kFull, valid);
        float lo[3], hi[3];
        target_box(p, valid, lo, hi);
        TeamSink<ORDER, PART> sink{S, err, wait_limit_ns, lane, n_bodies};
        walk(sink, nodes, num_nodes, root, full, lo, hi, S.tpos, S.stack, S.mixed_node, S.mixed_mask,
             walk_rounds(num_nodes), lanemask_lt(), lane, err);
        sink.finish();
    } else if (warp == 1) {
        for (int q = 0;; ++q) {
            const int slot = q % kRing;
            if (!team_wait(&S.node_ready[slot], (q / kRing) & 1, &S.abandon, err, wait_limit_ns)) break;
            const NodeList &l = S.nodes[slot];
            const int n = l.count;
            if (n < 0) break;
            for (int k = lane; k < n; k += 32) stage_node<PAY>(S.pay + k * PAY, nodes.pay, l.node[k]);
            cp_async_wait_all();
            __syncwarp();
            if (l.all) {
                full_terms<ORDER, EPS0>(S.pay, n, p, eps, lane, ax, ay, az);
                taken += (unsigned) n;
            } else {
                taken += part_terms<ORDER, EPS0, PART>(S.pay, l.mask, n, p, eps, lane, ax, ay, az);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.node_free[slot]);
        }
    } else {
        for (int q = warp - 2;; q += kLeafSets) {
            const int slot = q % kLeafRing;
            if (!team_wait(&S.leaf_ready[slot], (q / kLeafRing) & 1, &S.abandon, err, wait_limit_ns)) break;
            const LeafList &l = S.leaf[slot];
            const int n = l.count;
            if (n < 0) break;
            taken += leaf_terms<EPS0>(l.begin, l.end, l.mask, n, bodies, S.tile[warp - 2], p, eps, lane, ax, ay, az);
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.leaf_free[slot]);
        }
    }
    // the sets meet in the buffers that each warp staged its sources in (32 float4 or more each)
    __syncwarp();
    if (warp > 0) {
        float4 *mine = warp == 1 ? S.pay : S.tile[warp - 2];
        mine[lane] = make_float4(ax, ay, az, __uint_as_float(taken));
    }
    __syncthreads();
    if (warp == 0) {
        const float4 nodes_sum = S.pay[lane];
        ax = nodes_sum.x;
        ay = nodes_sum.y;
        az = nodes_sum.z;
        unsigned pairs = 0;
        for (int k = 0; k < kLeafSets; ++k) {
            const float4 v = S.tile[k][lane];
            ax += v.x;
            ay += v.y;
            az += v.z;
            pairs += __float_as_uint(v.w);
        }
        if (valid) acc[i] = make_float4(G * ax, G * ay, G * az, 0.f);
        const unsigned spp = __reduce_add_sync(kFull, valid ? pairs : 0u);
        const unsigned snp = __reduce_add_sync(kFull, valid ? __float_as_uint(nodes_sum.w) : 0u);
        if (lane == 0) add_counts(counts, inst_counts, inst, spp, snp);
    }
}

// Occupancy and SM count are fixed per device and kernel: queried once (B200 parts are identical).
// The kernel's dynamic shared memory (the warps' slabs and lists) is enabled on first use.
template<int ORDER, bool EPS0, int THREADS, int PART>
int blocks_per_sm(int device) {
    static int cached[64] = {0};
    if (device < 0 || device >= 64) device = 0;
    if (cached[device] == 0) {
        const size_t smem = block_smem_bytes<ORDER, THREADS, PART>();
        auto kernel = bh_kernel<ORDER, EPS0, THREADS, PART>;
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, THREADS, smem);
        cached[device] = b > 0 ? b : 1;
    }
    return cached[device];
}

template<int ORDER, bool EPS0, int THREADS, int PART>
int resident_warps(int device) {
    return sm_count(device) * blocks_per_sm<ORDER, EPS0, THREADS, PART>(device) * (THREADS / 32);
}

// Launches of at most this many groups run one team of warps per group, larger ones one warp per
// group. The team form has one walking warp in eight and four blocks per SM, so it loses where the groups alone
// fill the GPU. The line, in groups per SM:
//   - one wave of teams (four) always gains;
//   - above, larger leaves shift work from the walk to the leaf warps, and the line with it; a larger theta opens
//     fewer leaves, from 0.5 on at small ones, from 0.6 on at leaves of 64 (a straight line down to a fifth at theta 1);
//   - a slice of a larger set (a shard) has no sparse outskirts, whose few long groups hold one warp up
//     longest, and a deeper tree to walk;
//   - trees of few leaves give a group hardly more to do than a team's start and end cost.
// Measured, time with one warp over time with teams (g: groups per SM; Plummer spheres keep teams worth while to larger
// sets than balls, the line lies between):
//   whole sets at theta 0.5, Plummer and ball: leaf 1 1.07-1.09 at g 6, 0.96-1.07 at 8; leaf 8 1.02-1.15 at 10,
//     0.83-0.87 at 14; leaf 16 1.03-1.10 at 14, 0.96-0.99 at 18; leaf 32 0.98-1.10 at 30; leaf 64 0.99-1.07 at 54;
//   theta 0.7: leaf 8 1.00-1.08 at 10, 0.90-0.96 at 12; leaf 16 1.07-1.14 at 12, 0.95 at 14; leaf 32 1.04-1.18
//     at 18, 0.86-0.89 at 24; theta 1: leaf 8 0.99-1.12 at 8; leaf 16 0.97-1.07 at 10;
//   slices of 300,000 to 2^22 bodies: leaf 8 0.94-1.02 at 9; leaf 16 1.01-1.26 at 10.6, 0.83-1.05 at 13; leaf 32
//     0.93-1.19 at 17; leaf 64 0.93-1.17 at 32;
//   batches at leaf 16: instances of 33 to 200 bodies 1.05-1.15 at 3, 0.80-0.86 at 6, 0.5 at 18; of 500 1.5 at 3,
//     0.93 at 6; of 1000 1.09 at 6, 0.85 at 12; of 2500 1.14 at 12, 0.98 at 18; at leaf 64 1000 0.83 at 6, 2500
//     1.03 at 6, 0.81 at 12, 8000 1.04 at 29.
// Leaves above 64 bodies run one warp per group, although teams gain there too (1.15-3.2 for leaves of 65 to 256
// at theta 0.5 and up to 50 groups per SM, 1.04-1.7 for leaves of 1000).
int64_t team_groups(int device, int leaf, float theta, int64_t tree_bodies, bool slice) {
    if (leaf > 64) return 0;
    const double opened = std::min(1.0, std::max(0.2, 1.0 - 2.5 * (theta - (0.5 + leaf / 640.0))));
    const double most = 6.0 + 0.75 * (leaf * opened * (slice ? 0.45 : 1.0) + 1.5 * (1.0 - opened));
    const double few = std::min(1.0, (double) tree_bodies / (128.0 * leaf));
    return (int64_t) (sm_count(device) * (4.0 + (most - 4.0) * few * few));
}

struct LaunchArgs {
    const NodeArrays *nodes;
    const int *num_nodes;
    const float4 *bodies;
    int n_bodies;
    const float4 *targets;
    int nt;
    TreeShape shape;
    float G, eps;
    float4 *acc;
    unsigned long long *counts;
    TraverseWorkspace *ws;
    uint32_t *err;
    cudaStream_t s;
    const int4 *gtab;
    int64_t ngroups;
    const int *inst_root;
    unsigned long long *inst_counts;
    unsigned long long wait_limit_ns = kTeamWaitNs;
};

// The team kernel's dynamic shared memory is enabled on first use per device.
template<int ORDER, bool EPS0, int PART>
void launch_team(const LaunchArgs &a, int device) {
    static bool ready[64] = {false};
    constexpr size_t smem = sizeof(TeamSmem<NodeLayout<ORDER>::PAY, PART>);
    auto kernel = bh_team_kernel<ORDER, EPS0, PART>;
    if (device < 0 || device >= 64) device = 0;
    if (!ready[device]) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        ready[device] = true;
    }
    kernel<<<(unsigned) a.ngroups, kTeamThreads, smem, a.s>>>(*a.nodes, a.num_nodes, a.bodies, a.n_bodies, a.targets,
                                                              a.nt, a.G, a.eps, a.acc, a.counts, a.err, a.gtab,
                                                              a.inst_root, a.inst_counts, a.wait_limit_ns);
}

template<int ORDER, bool EPS0, int THREADS, int PART>
void launch_variant(const LaunchArgs &a) {
    constexpr int kWarps = THREADS / 32;
    int device = 0;
    cudaGetDevice(&device);
    // a slice holds at most a quarter of its set
    const bool slice = a.n_bodies / 4 >= a.nt;
    if (a.ngroups <= team_groups(device, a.shape.leaf, a.shape.theta, a.n_bodies / std::max(a.shape.trees, 1), slice)) {
        launch_team<ORDER, EPS0, PART>(a, device);
        return;
    }
    int64_t blocks = (int64_t) sm_count(device) * blocks_per_sm<ORDER, EPS0, THREADS, PART>(device);
    blocks = std::min<int64_t>(blocks, a.ws->warps / kWarps);
    blocks = std::min<int64_t>(blocks, (a.ngroups + kWarps - 1) / kWarps);
    if (blocks < 1) blocks = 1;
    bh_kernel<ORDER, EPS0, THREADS, PART><<<(unsigned) blocks, THREADS, block_smem_bytes<ORDER, THREADS, PART>(), a.s>>>(
        *a.nodes, a.num_nodes, a.bodies, a.n_bodies, a.targets, a.nt, a.G, a.eps, a.acc, a.counts, a.ws->stack,
        a.ws->group_counter, a.err, a.gtab, (int) a.ngroups, a.inst_root, a.inst_counts);
}

template<int ORDER, bool EPS0>
void launch_shape(const LaunchArgs &a, int threads, int part) {
    if (threads == 128) {
        if (part == 32) launch_variant<ORDER, EPS0, 128, 32>(a);
        else launch_variant<ORDER, EPS0, 128, 64>(a);
    } else {
        if (part == 32) launch_variant<ORDER, EPS0, 256, 32>(a);
        else launch_variant<ORDER, EPS0, 256, 64>(a);
    }
}

template<int ORDER, bool EPS0>
int max_resident_warps(int device) {
    return std::max(std::max(resident_warps<ORDER, EPS0, 128, 32>(device), resident_warps<ORDER, EPS0, 128, 64>(device)),
                    std::max(resident_warps<ORDER, EPS0, 256, 32>(device), resident_warps<ORDER, EPS0, 256, 64>(device)));
}

}  // namespace

int sm_count(int device) {
    static int cached[64] = {0};
    if (device < 0 || device >= 64) device = 0;
    if (cached[device] == 0) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cached[device] = sms > 0 ? sms : 1;
    }
    return cached[device];
}

int current_sm_count() {
    int device = 0;
    cudaGetDevice(&device);
    return sm_count(device);
}

int64_t traverse_resident_warps(int device) {
    return std::max(std::max(max_resident_warps<1, false>(device), max_resident_warps<1, true>(device)),
                    std::max(max_resident_warps<2, false>(device), max_resident_warps<2, true>(device)));
}

// The tree is a chain of `rounds` internal nodes, opened by every target, whose left children are accepted by every
// target: the walk takes one round per link (400 ns or more: two dependent loads and the classification) and
// opens no leaf, so the six leaf warps wait for its whole length. The node warp and the walker see the team
// abandoned at their next wait; the walk itself runs on to its end.
cudaError_t team_timeout_selftest(unsigned long long wait_limit_ns, uint32_t *err_word) {
    wait_limit_ns = std::min<unsigned long long>(wait_limit_ns, 100000000ull);
    const int rounds = (int) (wait_limit_ns / 100), num_nodes = 2 * rounds + 1;
    const std::unique_ptr<float4[]> mac(new (std::nothrow) float4[num_nodes]);
    const std::unique_ptr<int2[]> link(new (std::nothrow) int2[num_nodes]);
    if (!mac || !link) return cudaErrorMemoryAllocation;
    for (int c = 0; c < num_nodes; ++c) {
        const bool open = c % 2 == 0 && c + 2 < num_nodes;
        mac[c] = make_float4(0.f, 0.f, 0.f, open ? FLT_MAX : 0.f);
        link[c] = open ? make_int2(c + 2, -1) : make_int2(0, 1);
    }
    NodeArrays nodes;
    float4 *bodies = nullptr, *acc = nullptr;
    int *count = nullptr;
    uint32_t *err = nullptr;
    cudaError_t e = cudaSuccess;
    auto alloc = [&](void **p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
        if (e == cudaSuccess) e = cudaMemset(*p, 0, bytes);
    };
    alloc((void **) &nodes.mac, num_nodes * sizeof(float4));
    alloc((void **) &nodes.link, num_nodes * sizeof(int2));
    alloc((void **) &nodes.pay, num_nodes * sizeof(float4));
    alloc((void **) &bodies, 32 * sizeof(float4));
    alloc((void **) &acc, 32 * sizeof(float4));
    alloc((void **) &count, sizeof(int));
    alloc((void **) &err, sizeof(uint32_t));
    auto copy = [&](void *dst, const void *src, size_t bytes) {
        if (e == cudaSuccess) e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    };
    copy(nodes.mac, mac.get(), num_nodes * sizeof(float4));
    copy(nodes.link, link.get(), num_nodes * sizeof(int2));
    copy(count, &num_nodes, sizeof(int));
    if (e == cudaSuccess) {
        int device = 0;
        cudaGetDevice(&device);
        LaunchArgs a{&nodes, count, bodies, 32, bodies, 32, TreeShape(), 1.f, 1.f, acc, nullptr, nullptr, err, nullptr,
                     nullptr, 1, nullptr, nullptr};
        a.wait_limit_ns = wait_limit_ns;
        launch_team<1, false, 64>(a, device);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(err_word, err, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    for (void *p: {(void *) nodes.mac, (void *) nodes.link, (void *) nodes.pay, (void *) bodies, (void *) acc,
                   (void *) count, (void *) err})
        if (p) cudaFree(p);
    return e;
}

bool traversal_shape_valid(int threads, int slab) { return (threads == 128 || threads == 256) && (slab == 32 || slab == 64); }

void launch_bh_traverse(int order, const NodeArrays &nodes, const int *num_nodes, const float4 *bodies, int64_t n_bodies,
                        const float4 *targets, int64_t n_targets, TreeShape shape, float G, float eps, float4 *acc,
                        unsigned long long *counts, TraverseWorkspace &ws, uint32_t *err, cudaStream_t s,
                        const int4 *gtab, int64_t ngroups, const int *inst_root, unsigned long long *inst_counts) {
    if (n_targets <= 0) return;
    if (!gtab) ngroups = (n_targets + 31) / 32;
    const LaunchArgs a{&nodes, num_nodes, bodies, (int) n_bodies, targets, (int) n_targets, shape, G, eps, acc, counts, &ws,
                       err, s, gtab, ngroups, inst_root, inst_counts};
    const bool ok = traversal_shape_valid(ws.threads, ws.slab);
    const int threads = ok ? ws.threads : 256, part = ok ? ws.slab : 64;
    if (order == 1) {
        if (eps == 0.f) launch_shape<1, true>(a, threads, part);
        else launch_shape<1, false>(a, threads, part);
    } else {
        if (eps == 0.f) launch_shape<2, true>(a, threads, part);
        else launch_shape<2, false>(a, threads, part);
    }
}

}  // namespace nbg
