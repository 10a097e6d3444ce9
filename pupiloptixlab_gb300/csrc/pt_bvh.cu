// pt_bvh.cu -- GPU acceleration-structure build and refit.
//
// Replaces the closed OptiX builds GAS::Create / IAS::Create / IAS::Update
// (framework/world/gas_manager.cpp:69-245, framework/world/ias_manager.cpp:
// 29-151).  Pipeline (all on the device, one GPU):
//   1. primitive boxes and centroid bounds (block reduction + ordered atomics)
//   2. 63-bit Morton codes (21 bits per axis)
//   3. stable LSD radix sort of (code, primitive) pairs, 8 passes of 8 bits:
//      tile histogram -> exclusive scan per digit over the tiles -> scatter
//      (warp-private digit counters, __match_any_sync ranks)
//   4. binary tree: PLOC clustering (default) or the Karras (HPG 2012)
//      binary radix tree, equal codes split by index
//   5. with each binary node, when it forms: box, primitive count and the
//      SAH-optimal assignment of its subtree to the slots of 2/4/8-wide nodes
//      (dynamic programming, leaves of at most max_leaf_size primitives)
//   6. top-down, level-synchronous collapse that follows those choices; nodes
//      come out in breadth-first order
//   7. primitive records gathered into leaf order (depth first)
// The level and cluster counts stay on the device; the host reads them back a
// few times a build.
// Child boxes are padded outward (relative to the box and scene magnitude) so
// that the conservative slab test never rejects a primitive the exact test
// would hit.

#include "pt_nvtx.h"
#include "pt_internal.h"
#include "pt_traverse.cuh"

#include <algorithm>
#include <cfloat>
#include <cstddef>
#include <type_traits>

namespace {

using ptd::f3;

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr float kCostNode = 1.2f;
constexpr float kCostPrim = 1.0f;
constexpr float kCostCurvePiece = 3.0f;  // a round-cone test costs about three triangle tests

// SAH intersection cost of one primitive record (triangle and sphere 1).
__device__ __forceinline__ float prim_cost(const float4 *prims, uint32_t p) {
    const float4 a = prims[3 * (size_t)p], b = prims[3 * (size_t)p + 1];
    return (__float_as_int(a.w) < 0 && __float_as_int(b.w) != 0) ? kCostCurvePiece : kCostPrim;
}

__device__ __forceinline__ uint32_t f2ord(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ void prim_box(const float4 *prims, uint32_t p, float3 &lo, float3 &hi) {
    const float4 a = prims[3 * (size_t)p], b = prims[3 * (size_t)p + 1], c = prims[3 * (size_t)p + 2];
    if (__float_as_int(a.w) >= 0) {
        lo = f3(fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)));
        hi = f3(fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)));
    } else if (__float_as_int(b.w) == 0) {  // sphere
        float r = b.x;
        lo = f3(a.x - r, a.y - r, a.z - r);
        hi = f3(a.x + r, a.y + r, a.z + r);
    } else {  // round-cone curve piece: the boxes of its two end spheres
        float r0 = b.x, r1 = b.y;
        lo = f3(fminf(a.x - r0, c.x - r1), fminf(a.y - r0, c.y - r1), fminf(a.z - r0, c.z - r1));
        hi = f3(fmaxf(a.x + r0, c.x + r1), fmaxf(a.y + r0, c.y + r1), fmaxf(a.z + r0, c.z + r1));
    }
}

// 1. per-primitive box records + centroid bounds into 6 ordered uints.  A grid
// of a few blocks per SM: one atomic per block and bound (16,033 blocks spent
// most of their 174 us on six addresses).
__global__ void k_prim_bounds(const float4 *prims, uint32_t n, float4 *pbox, uint32_t *cb) {
    __shared__ float red[6][32];
    float v[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float3 lo, hi;
        prim_box(prims, i, lo, hi);
        // box record: (low, cost weight) (high, primitive count)
        ptd::st8(pbox + 2 * (size_t)i, make_float4(lo.x, lo.y, lo.z, prim_cost(prims, i)),
                 make_float4(hi.x, hi.y, hi.z, __int_as_float(1)));
        const float cx = 0.5f * (lo.x + hi.x), cy = 0.5f * (lo.y + hi.y), cz = 0.5f * (lo.z + hi.z);
        v[0] = fminf(v[0], cx);
        v[1] = fminf(v[1], cy);
        v[2] = fminf(v[2], cz);
        v[3] = fmaxf(v[3], cx);
        v[4] = fmaxf(v[4], cy);
        v[5] = fmaxf(v[5], cz);
    }
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        float x = v[k];
        for (int o = 16; o > 0; o >>= 1) {
            float y = __shfl_xor_sync(0xffffffffu, x, o);
            x = k < 3 ? fminf(x, y) : fmaxf(x, y);
        }
        if (lane == 0) red[k][warp] = x;
    }
    __syncthreads();
    if (warp == 0) {
        int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            float x = lane < nw ? red[k][lane] : (k < 3 ? FLT_MAX : -FLT_MAX);
            for (int o = 16; o > 0; o >>= 1) {
                float y = __shfl_xor_sync(0xffffffffu, x, o);
                x = k < 3 ? fminf(x, y) : fmaxf(x, y);
            }
            if (lane == 0) {
                if (k < 3) atomicMin(&cb[k], f2ord(x));
                else atomicMax(&cb[k], f2ord(x));
            }
        }
    }
}

__device__ __forceinline__ uint64_t split3(uint32_t a) {
    uint64_t x = a & 0x1fffffu;
    x = (x | x << 32) & 0x1f00000000ffffULL;
    x = (x | x << 16) & 0x1f0000ff0000ffULL;
    x = (x | x << 8) & 0x100f00f00f00f00fULL;
    x = (x | x << 4) & 0x10c30c30c30c30c3ULL;
    x = (x | x << 2) & 0x1249249249249249ULL;
    return x;
}

// 2. Morton codes of the box centroids.
__global__ void k_morton(const float4 *pbox, uint32_t n, const uint32_t *cb, uint64_t *keys, uint32_t *vals) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float mn[3] = {ord2f(cb[0]), ord2f(cb[1]), ord2f(cb[2])};
    float mx[3] = {ord2f(cb[3]), ord2f(cb[4]), ord2f(cb[5])};
    float4 lo, hi;
    ptd::ld8(pbox + 2 * (size_t)i, lo, hi);
    float c[3] = {0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z)};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float ext = mx[k] - mn[k];
        float t = ext > 0.f ? (c[k] - mn[k]) / ext : 0.f;
        float s = t * 2097152.0f;
        q[k] = (uint32_t)fminf(fmaxf(s, 0.f), 2097151.f);
    }
    keys[i] = (split3(q[0]) << 2) | (split3(q[1]) << 1) | split3(q[2]);
    vals[i] = i;
}

// 3a. per-tile digit histogram, stored digit-major: hist[d * tiles + tile].
__global__ void k_radix_hist(const uint64_t *keys, uint32_t n, int shift, uint32_t *hist, uint32_t tiles) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    size_t base = (size_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int k = 0; k < kSortItems; k++) {
        size_t idx = base + (size_t)k * kSortThreads + threadIdx.x;
        if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// 3b. one block per digit: exclusive scan of its tile counts, in place, and
// their total.  (One block over all 256 * tiles counts took about 100 us a pass
// at 4 million primitives.)
__global__ void __launch_bounds__(256) k_radix_scan(uint32_t *hist, uint32_t tiles, uint32_t *total) {
    __shared__ uint32_t wsum[8];
    uint32_t *row = hist + (size_t)blockIdx.x * tiles;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < tiles; b += 256) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < tiles ? row[i] : 0u;
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (uint32_t w = 0; w < 8; w++) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (i < tiles) row[i] = carry + before + x - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) total[blockIdx.x] = carry;
}

// 3c. stable scatter.  Each warp owns a contiguous eighth of the tile and
// counts its digits in order (the rank of an entry = its warp's count so far +
// its rank among the equal digits of its 32).  The tile is put in digit order
// in shared memory first, so that runs of equal digits are written together
// (written straight from the registers: 98 us a pass at 4.1 million pairs).
constexpr int kScatterSmem = kSortTile * 12;
__global__ void __launch_bounds__(kSortThreads, 3) k_radix_scatter(const uint64_t *kin, const uint32_t *vin, uint64_t *kout,
                                                                uint32_t *vout, uint32_t n, int shift,
                                                                const uint32_t *hist, uint32_t tiles,
                                                                const uint32_t *total) {
    constexpr int kWarps = kSortThreads / 32;
    extern __shared__ uint64_t sort_smem[];
    uint64_t *skey = sort_smem;
    uint32_t *sval = reinterpret_cast<uint32_t *>(skey + kSortTile);
    __shared__ uint32_t wcnt[kWarps][256];
    __shared__ uint32_t gbase[256];  // output position of a digit's first entry, minus its place in the tile
    __shared__ uint32_t wsum[2][kWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t lt = (1u << lane) - 1u;
    for (int d = lane; d < 256; d += 32) wcnt[warp][d] = 0;
    __syncwarp();
    const uint32_t t0 = blockIdx.x * kSortTile;
    const uint32_t base = warp * (32 * kSortItems) + lane;
    uint64_t key[kSortItems];
    uint32_t rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t i = base + k * 32;
        key[k] = t0 + i < n ? kin[t0 + i] : ~0ull;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const bool valid = t0 + base + k * 32 < n;
        const uint32_t digit = (uint32_t)(key[k] >> shift) & 255u;
        const uint32_t peers = __match_any_sync(0xffffffffu, valid ? digit : 256u);
        uint32_t old = 0;
        if (valid) old = wcnt[warp][digit];
        __syncwarp();
        if (valid && (peers & lt) == 0) wcnt[warp][digit] = old + __popc(peers);
        __syncwarp();
        rank[k] = old + __popc(peers & lt);
    }
    __syncthreads();
    {  // thread = digit: starts of the digits in the output (over the totals) and in the tile
        uint32_t mine = 0;
        for (int w = 0; w < kWarps; w++) mine += wcnt[w][tid];
        const uint32_t tot = total[tid];
        uint32_t a = tot, b = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t ya = __shfl_up_sync(0xffffffffu, a, o), yb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) {
                a += ya;
                b += yb;
            }
        }
        if (lane == 31) {
            wsum[0][warp] = a;
            wsum[1][warp] = b;
        }
        __syncthreads();
        a -= tot;
        b -= mine;
        for (int w = 0; w < warp; w++) {
            a += wsum[0][w];
            b += wsum[1][w];
        }
        gbase[tid] = a + hist[(size_t)tid * tiles + blockIdx.x] - b;
        uint32_t run = b;
        for (int w = 0; w < kWarps; w++) {
            const uint32_t c = wcnt[w][tid];
            wcnt[w][tid] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const uint32_t i = t0 + base + k * 32;
        if (i >= n) continue;
        const uint32_t at = wcnt[warp][(uint32_t)(key[k] >> shift) & 255u] + rank[k];
        skey[at] = key[k];
        sval[at] = vin[i];
    }
    __syncthreads();
    const uint32_t count = min((uint32_t)kSortTile, n - t0);
    for (uint32_t i = tid; i < count; i += kSortThreads) {
        const uint64_t key_i = skey[i];
        const uint32_t pos = gbase[(uint32_t)(key_i >> shift) & 255u] + i;
        kout[pos] = key_i;
        vout[pos] = sval[i];
    }
}

__device__ __forceinline__ int delta(const uint64_t *keys, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    uint64_t a = keys[i], b = keys[j];
    if (a == b) return 64 + __clz((uint32_t)(i ^ j));
    return __clzll(a ^ b);
}

// 4. Karras binary radix tree.  Internal nodes 0..n-2, leaf k is node n-1+k.
__global__ void k_karras(const uint64_t *keys, int n, int4 *links, int *parent) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s = 0;
    int div = 2, t;
    do {
        t = (l + div - 1) / div;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
        div <<= 1;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int first = min(i, j), last = max(i, j);
    int lc = (first == gamma) ? (n - 1 + gamma) : gamma;
    int rc = (last == gamma + 1) ? (n - 1 + gamma + 1) : gamma + 1;
    links[i] = make_int4(lc, rc, 0, 0);
    parent[lc] = i;
    parent[rc] = i;
}

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
    float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
    return ex * ey + ey * ez + ez * ex;
}

// A binary node's box record: (low, summed cost weight) (high, primitive count).
struct NodeBox {
    float4 lo, hi;
    __device__ __forceinline__ float area() const { return half_area(lo, hi); }
    __device__ __forceinline__ float weight() const { return lo.w; }
    __device__ __forceinline__ int count() const { return __float_as_int(hi.w); }
};
__device__ __forceinline__ NodeBox load_box(const float4 *nb, int x) {
    NodeBox b;
    ptd::ld8(nb + 2 * (size_t)x, b.lo, b.hi);
    return b;
}
__device__ __forceinline__ NodeBox merged(const NodeBox &a, const NodeBox &b) {
    NodeBox u;
    u.lo = make_float4(fminf(a.lo.x, b.lo.x), fminf(a.lo.y, b.lo.y), fminf(a.lo.z, b.lo.z), a.lo.w + b.lo.w);
    u.hi = make_float4(fmaxf(a.hi.x, b.hi.x), fmaxf(a.hi.y, b.hi.y), fmaxf(a.hi.z, b.hi.z),
                       __int_as_float(a.count() + b.count()));
    return u;
}

// The binary tree: internal nodes 0..n-2, leaf k (sorted primitive k) is node
// n-1+k.
struct Tree {
    int n, max_leaf;
    int4 *links;   // per internal node: left, right, the choices (below), the left child's primitive count
    float4 *nb;    // 2 per node
    float *dval;   // K per internal node: S(x, 1..K) below
};

// 5. SAH-optimal wide collapse (Ylitie, Karras and Laine, HPG 2017): for
// every binary node x and i = 1..K, S(x, i) is the cheapest way to represent
// its subtree with at most i slots of a wide parent:
//   S(x, 1) = min(leaf: area * primitive weight (if count <= max_leaf),
//                 wide node: 1.2 * area + min_j S(l, j) + S(r, K - j))
//   S(x, i) = min(S(x, i - 1), min_j S(l, j) + S(r, i - j))
// Formed with the node itself, when its children are complete.  The choices, 3
// bits each: 0 the wide node's split j, i - 1 the split for i = 2..K slots (0:
// use i - 1 slots); bit 31: leaf.
constexpr uint32_t kSelLeaf = 1u << 31;
__device__ __forceinline__ int sel_of(int sel, int i) { return (sel >> (3 * i)) & 7; }

template <int K>
__device__ __forceinline__ void load_costs(const Tree &t, int x, const NodeBox &b, float *c) {
    if (x >= t.n - 1) {
        const float v = b.area() * b.weight();
#pragma unroll
        for (int i = 0; i < K; i++) c[i] = v;
    } else {
#pragma unroll
        for (int i = 0; i < K; i++) c[i] = __ldcg(t.dval + (size_t)x * K + i);
    }
}

// Node `id` over children l and r (boxes bl, br): links, box, costs, choices.
template <int K>
__device__ __forceinline__ NodeBox form_node(const Tree &t, int id, int l, int r, const NodeBox &bl, const NodeBox &br) {
    const NodeBox u = merged(bl, br);
    float sl[K], sr[K], sx[K];
    load_costs<K>(t, l, bl, sl);
    load_costs<K>(t, r, br, sr);
    const float area = u.area();
    float best = FLT_MAX;
    int jw = 1;
#pragma unroll
    for (int j = 1; j < K; j++) {
        const float c = sl[j - 1] + sr[K - j - 1];
        if (c < best) {
            best = c;
            jw = j;
        }
    }
    const float c_wide = kCostNode * area + best;
    // the limit is a condition, not a cost: an area may overflow to infinity (the
    // split then stays j = 1, and the node is wide)
    const float c_leaf = area * u.weight();
    const bool mk_leaf = u.count() <= t.max_leaf && c_leaf <= c_wide;
    sx[0] = mk_leaf ? c_leaf : c_wide;
    uint32_t sel = (uint32_t)jw | (mk_leaf ? kSelLeaf : 0);
#pragma unroll
    for (int i = 2; i <= K; i++) {
        float v = sx[i - 2];
        int pick = 0;
#pragma unroll
        for (int j = 1; j < i; j++) {
            const float c = sl[j - 1] + sr[i - j - 1];
            if (c < v) {
                v = c;
                pick = j;
            }
        }
        sx[i - 1] = v;
        sel |= (uint32_t)pick << (3 * (i - 1));
    }
#pragma unroll
    for (int i = 0; i < K; i++) t.dval[(size_t)id * K + i] = sx[i];
    t.links[id] = make_int4(l, r, (int)sel, bl.count());
    ptd::st8(t.nb + 2 * (size_t)id, u.lo, u.hi);
    return u;
}

// The sorted primitives as leaves.
__global__ void k_leaf_boxes(int n, const uint32_t *order, const float4 *pbox, float4 *nb, int *cl) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const NodeBox b = load_box(pbox, (int)order[k]);
    ptd::st8(nb + 2 * (size_t)(n - 1 + k), b.lo, b.hi);
    cl[k] = n - 1 + k;
}

// Radix tree, bottom up (second arrival forms a node).
template <int K>
__global__ void k_bottom_up(const Tree t, const int *parent, int *flags) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= t.n) return;
    int cur = parent[t.n - 1 + k];
    while (cur >= 0) {
        __threadfence();
        if (atomicAdd(&flags[cur], 1) == 0) return;
        __threadfence();
        const int l = t.links[cur].x, r = t.links[cur].y;
        NodeBox bl, br;
        bl.lo = __ldcg(t.nb + 2 * (size_t)l);
        bl.hi = __ldcg(t.nb + 2 * (size_t)l + 1);
        br.lo = __ldcg(t.nb + 2 * (size_t)r);
        br.hi = __ldcg(t.nb + 2 * (size_t)r + 1);
        form_node<K>(t, cur, l, r, bl, br);
        cur = parent[cur];
    }
}

// 4'. PLOC: parallel locally-ordered clustering (Meister and Bittner,
// IEEE TVCG 2018), the default build.  The Morton-sorted primitives start as
// clusters; each pass every cluster finds the cluster within kPlocRadius
// positions whose union has the smallest surface area (ties to the lower
// position, so the closest pair is always mutual), mutual nearest neighbours
// merge into a new internal node (id from a counter, 0..n-2) that takes the
// lower position, and the array is compacted.  A pass is two launches: neighbours
// and merging share a tile with a halo of two radii, and each compaction tile
// sums the survivor counts of the tiles before it.  The counts stay on the
// device: the host bounds the grids by the count it last read.  The last
// kPlocTail clusters are merged by one block in shared memory.
// The neighbour search is bound by shared-memory reads (64 128-bit loads a
// position, 181 us for 4.1 million), so a thread searches for PER = 4
// consecutive positions, whose windows share 28 of 36 boxes; where few tiles
// are left the time is one thread's chain (20 us at PER = 4), so PER = 1.
constexpr int kPlocRadius = 16;
constexpr int kPlocThreads = 288;
__host__ __device__ constexpr int ploc_tile(int per) { return kPlocThreads * per - 2 * kPlocRadius; }  // every thread searches once
constexpr int kPlocTail = 2048;
constexpr int kPlocMaxPasses = 64 + 8 * 28;
constexpr int kPlocPassesPerRead = 8;  // clusters shrink by about a quarter a pass
constexpr uint32_t kPlocWide = 300000;  // clusters from which PER = 4 is used (about two tiles an SM)

// Device-side counts of a build.
constexpr int kMaxLevels = 128;
struct BuildCounts {
    uint32_t centroid[6];   // ordered-float bounds
    uint32_t nodes;         // PLOC internal nodes formed
    uint32_t fail;
    double sah, root_area;
    uint32_t level[kMaxLevels + 1];            // wide nodes per level
    uint32_t clusters[kPlocMaxPasses + 2];     // PLOC clusters before pass p
};

// Nearest neighbours of the positions i..i+PER-1 among the boxes lo/hi in shared
// memory (box of position i + o at place(o); out of range: an unbounded box).
template <int PER, class Place>
__device__ __forceinline__ void nearest(const float4 *lo, const float4 *hi, const Place &place, int i, int *bj) {
    float4 al[PER], ah[PER];
    float best[PER];
#pragma unroll
    for (int q = 0; q < PER; q++) {
        al[q] = lo[place(q)];
        ah[q] = hi[place(q)];
        best[q] = FLT_MAX;
        bj[q] = -1;
    }
#pragma unroll
    for (int o = -kPlocRadius; o < PER + kPlocRadius; o++) {
        const float4 bl = lo[place(o)], bh = hi[place(o)];
#pragma unroll
        for (int q = 0; q < PER; q++) {
            if (o == q || o - q > kPlocRadius || q - o > kPlocRadius) continue;
            const float4 ul = make_float4(fminf(al[q].x, bl.x), fminf(al[q].y, bl.y), fminf(al[q].z, bl.z), 0.f);
            const float4 uh = make_float4(fmaxf(ah[q].x, bh.x), fmaxf(ah[q].y, bh.y), fmaxf(ah[q].z, bh.z), 0.f);
            const float a = half_area(ul, uh);
            if (a < best[q]) {  // positions are visited in increasing order: ties keep the lower one
                best[q] = a;
                bj[q] = i + o;
            }
        }
    }
}
__device__ __forceinline__ void unbounded(float4 &lo, float4 &hi) {
    lo = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f);
    hi = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.f);
}

template <int K, int PER>
__global__ void __launch_bounds__(kPlocThreads) k_ploc_merge(const Tree t, BuildCounts *bc, int pass, const int *cl,
                                                             int *out_id, uint32_t *tile_count) {
    constexpr int R = kPlocRadius, kTile = ploc_tile(PER);
    // boxes of the positions [t0 - 2R, t0 + kTile + 2R), PER rows: the boxes a
    // warp reads together are neighbours in a row (no bank conflicts)
    constexpr int kCols = kPlocThreads + 2 * R / PER + (PER > 1 ? 1 : 0);
    __shared__ float4 slo[PER * kCols], shi[PER * kCols];
    constexpr int kWarps = kPlocThreads / 32, kRounds = (kTile + kPlocThreads - 1) / kPlocThreads;
    __shared__ int snn[kTile + 2 * R];
    __shared__ uint32_t merges[kRounds * kWarps], kept, first_node;
    const auto at = [](int k) { return PER == 1 ? k : (k % PER) * kCols + k / PER; };  // place of position t0 - 2R + k
    const int m = (int)bc->clusters[pass];
    const int t0 = blockIdx.x * kTile;
    if (t0 >= m) return;  // uniform
    if (threadIdx.x == 0) kept = 0;
    for (int k = threadIdx.x; k < kTile + 4 * R; k += kPlocThreads) {
        const int g = t0 - 2 * R + k;
        if (g >= 0 && g < m) {
            const NodeBox b = load_box(t.nb, cl[g]);
            slo[at(k)] = b.lo;
            shi[at(k)] = b.hi;
        } else {
            unbounded(slo[at(k)], shi[at(k)]);
        }
    }
    __syncthreads();
    {
        const int c = threadIdx.x * PER;  // positions t0 - R + c ...
        int bj[PER];
        // place of position t0 - R + c + o (c a multiple of PER)
        const auto place = [](int o) { return (R + o) % PER * kCols + (int)threadIdx.x + (R + o) / PER; };
        nearest<PER>(slo, shi, place, t0 - R + c, bj);
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int g = t0 - R + c + q;
            snn[c + q] = g >= 0 && g < m ? bj[q] : -1;
        }
    }
    __syncthreads();
    // new nodes are numbered by one atomic per tile (a warp's atomic at a time, all on one
    // address: the 16 wide passes of 4.1M triangles 0.89 ms, so 0.72)
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t mine = 0, rank[kRounds];
    int partner[kRounds];  // position merged with; -1 not merged; kNone: merged by the partner, or no position
    constexpr int kNone = -2;
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const int k = r * kPlocThreads + threadIdx.x, i = t0 + k;
        const bool valid = k < kTile && i < m;
        const int j = valid ? snn[k + R] : -1;
        const bool mutual = j >= 0 && snn[j - t0 + R] == i, merge = mutual && i < j;
        partner[r] = merge ? j : valid && !mutual ? -1 : kNone;
        const unsigned b = __ballot_sync(FULL, merge);
        rank[r] = __popc(b & ((1u << lane) - 1u));
        if (lane == 0) merges[r * kWarps + warp] = __popc(b);
        mine += partner[r] != kNone ? 1u : 0u;
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t sum = 0;
        for (int e0 = 0; e0 < kRounds * kWarps; e0 += 32) {
            const int e = e0 + lane;
            const uint32_t v = e < kRounds * kWarps ? merges[e] : 0u;
            uint32_t x = v;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += y;
            }
            if (e < kRounds * kWarps) merges[e] = sum + x - v;
            sum += __shfl_sync(FULL, x, 31);
        }
        if (lane == 0) first_node = atomicAdd(&bc->nodes, sum);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const int k = r * kPlocThreads + threadIdx.x, i = t0 + k;
        if (k >= kTile || i >= m) continue;
        int out = -1;
        if (partner[r] == -1) {
            out = cl[i];
        } else if (partner[r] >= 0) {
            const int j = partner[r];
            NodeBox a, b;
            a.lo = slo[at(k + 2 * R)];
            a.hi = shi[at(k + 2 * R)];
            b.lo = slo[at(j - t0 + 2 * R)];
            b.hi = shi[at(j - t0 + 2 * R)];
            out = (int)(first_node + merges[r * kWarps + warp] + rank[r]);
            form_node<K>(t, out, cl[i], cl[j], a, b);
        }
        out_id[i] = out;
    }
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&kept, mine);
    __syncthreads();
    if (threadIdx.x == 0) tile_count[blockIdx.x] = kept;
}

// Order-preserving compaction of a tile's survivors behind those of the tiles
// before it; the last tile records the next pass's counts.
template <int PER>
__global__ void __launch_bounds__(kPlocThreads) k_ploc_compact(BuildCounts *bc, int pass, const int *out_id,
                                                               const uint32_t *tile_count, int *cl_next) {
    constexpr int kWarps = kPlocThreads / 32, kTile = ploc_tile(PER);
    constexpr int kRounds = (kTile + kPlocThreads - 1) / kPlocThreads;
    __shared__ uint32_t before[kWarps];
    __shared__ uint32_t wc[kRounds * kWarps];
    const int m = (int)bc->clusters[pass];
    const int t0 = blockIdx.x * kTile;
    if (t0 >= m) return;  // uniform
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t sum = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kPlocThreads) sum += tile_count[b];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) before[warp] = sum;
    int id[kRounds];
    unsigned bal[kRounds];
#pragma unroll
    for (int k = 0; k < kRounds; k++) {
        const int at = k * kPlocThreads + (int)threadIdx.x;
        id[k] = at < kTile && t0 + at < m ? out_id[t0 + at] : -1;
        bal[k] = __ballot_sync(0xffffffffu, id[k] >= 0);
        if (lane == 0) wc[k * kWarps + warp] = __popc(bal[k]);
    }
    __syncthreads();
    uint32_t start = 0;
    for (int w = 0; w < kWarps; w++) start += before[w];
#pragma unroll
    for (int k = 0; k < kRounds; k++) {
        uint32_t at = start;
        for (uint32_t w = 0; w < kWarps; w++) {
            if (w < warp) at += wc[k * kWarps + w];
            start += wc[k * kWarps + w];
        }
        if (id[k] >= 0) cl_next[at + __popc(bal[k] & ((1u << lane) - 1u))] = id[k];
    }
    if (t0 + kTile >= m && threadIdx.x == 0) bc->clusters[pass + 1] = start;
}

// The passes from `pass` on, at most kPlocTail clusters, in one block.
template <int K>
__global__ void __launch_bounds__(1024) k_ploc_tail(const Tree t, BuildCounts *bc, int pass, const int *cl) {
    constexpr int R = kPlocRadius, kPer = kPlocTail / 1024;
    extern __shared__ float4 tail_smem[];
    float4 *slo = tail_smem, *shi = slo + kPlocTail + 2 * R;
    int *sid = reinterpret_cast<int *>(shi + kPlocTail + 2 * R), *snn = sid + kPlocTail;
    __shared__ uint32_t wc[kPer * 32];
    __shared__ uint32_t ctr, survivors;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int m = (int)bc->clusters[pass];
    if (m > kPlocTail || m < 1) {  // uniform: the host starts this kernel only below the limit
        if (tid == 0) bc->fail = 1;
        return;
    }
    if (tid == 0) ctr = bc->nodes;
    for (int i = tid; i < kPlocTail + 2 * R; i += 1024) unbounded(slo[i], shi[i]);
    __syncthreads();
    for (int i = tid; i < m; i += 1024) {
        const int id = cl[i];
        const NodeBox b = load_box(t.nb, id);
        sid[i] = id;
        slo[i + R] = b.lo;
        shi[i + R] = b.hi;
    }
    __syncthreads();
    while (m > 1 && pass < kPlocMaxPasses) {
        for (int i = tid; i < m; i += 1024) nearest<1>(slo, shi, [&](int o) { return i + R + o; }, i, snn + i);
        __syncthreads();
        int id[kPer];
        NodeBox box[kPer];
        unsigned bal[kPer];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const int i = k * 1024 + tid;
            id[k] = -1;
            if (i < m) {
                const int j = snn[i];
                const bool mutual = j >= 0 && snn[j] == i;
                box[k].lo = slo[i + R];
                box[k].hi = shi[i + R];
                if (!mutual) {
                    id[k] = sid[i];
                } else if (i < j) {
                    NodeBox b;
                    b.lo = slo[j + R];
                    b.hi = shi[j + R];
                    id[k] = (int)atomicAdd(&ctr, 1u);
                    box[k] = form_node<K>(t, id[k], sid[i], sid[j], box[k], b);
                }
            }
            bal[k] = __ballot_sync(0xffffffffu, id[k] >= 0);
            if (lane == 0) wc[k * 32 + warp] = __popc(bal[k]);
        }
        __syncthreads();  // boxes and ids are read, nodes are formed
        if (warp == 0) {
            uint32_t carry = 0;
            for (int k = 0; k < kPer; k++) {
                const uint32_t v = wc[k * 32 + lane];
                uint32_t x = v;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                wc[k * 32 + lane] = carry + x - v;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) survivors = carry;
        }
        __syncthreads();
        const int next = (int)survivors;
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            if (id[k] < 0) continue;
            const int at = (int)(wc[k * 32 + warp] + __popc(bal[k] & ((1u << lane) - 1u)));
            sid[at] = id[k];
            slo[at + R] = box[k].lo;
            shi[at + R] = box[k].hi;
        }
        __syncthreads();
        for (int i = next + tid; i < m; i += 1024) unbounded(slo[i + R], shi[i + R]);
        __syncthreads();
        pass++;
        if (next >= m) break;  // uniform: no pair merged (boxes without a finite area)
        m = next;
    }
    if (tid == 0) {
        bc->nodes = ctr;
        if (m != 1 || ctr != (uint32_t)(t.n - 1)) bc->fail = 1;
    }
}

__device__ __forceinline__ void padded(float4 lo, float4 hi, float scene_mag, float3 &plo, float3 &phi) {
    float mag = fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(lo.z), fabsf(hi.x))), fmaxf(fabsf(hi.y), fabsf(hi.z)));
    float ext = fmaxf(fmaxf(hi.x - lo.x, hi.y - lo.y), hi.z - lo.z);
    float pad = 4e-7f * (mag + scene_mag) + 1e-6f * ext;
    plo = f3(lo.x - pad, lo.y - pad, lo.z - pad);
    phi = f3(hi.x + pad, hi.y + pad, hi.z + pad);
}

__device__ __forceinline__ int item_count(int item) { return ptd::is_leaf(item) ? ptd::leaf_count(item) : 0; }
// The primitives of leaf x (at most 15), depth first, from position `first` on.
__device__ __forceinline__ void leaf_positions(const Tree &t, int x, int first, const uint32_t *order,
                                               uint32_t *leaf_order) {
    int st[16];
    int sp = 0;
    for (;;) {
        if (x >= t.n - 1) {
            leaf_order[first++] = order[x - (t.n - 1)];
            if (sp == 0) return;
            x = st[--sp];
        } else {
            const int4 l = t.links[x];
            if (sp < 16) st[sp++] = l.y;  // (15 primitives: at most 14 pending)
            x = l.x;
        }
    }
}

// 6. one level of the collapse, following the choices of form_node: the wide
// node of binary node b gets the slots of left(b) (choice 0 of them) and
// right(b) (the rest), each expanded while its choice splits it further.  The
// wide nodes of level L are [start, start + level[L]); their inner children,
// appended by one atomic per block, follow them.  wide[w]: binary node of wide
// node w and the position of its first primitive in leaf order (depth first:
// a right subtree follows its left one), which the leaves found here get.
// Also sums the SAH cost of what it writes.  A small level's time is the chain
// of one thread's dependent loads, hence one 16-byte record per binary node.
template <int K>
__global__ void __launch_bounds__(128) k_collapse(const Tree t, BuildCounts *bc, int level, int root, int2 *wide,
                                                  float *nodes, float scene_mag, const uint32_t *order,
                                                  uint32_t *leaf_order) {
    __shared__ uint32_t s_start, s_child, s_inner[4];
    __shared__ double s_sah;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (bc->fail) return;  // uniform
    const uint32_t count = bc->level[level];
    if (blockIdx.x * blockDim.x >= count) return;  // uniform
    if (threadIdx.x == 0) s_sah = 0.0;
    if (threadIdx.x < 32) {
        uint32_t v = 0;
        for (int l = lane; l < level; l += 32) v += bc->level[l];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if (lane == 0) s_start = v;
    }
    __syncthreads();
    const uint32_t start = s_start;
    const int n = t.n;
    double sah = 0.0;
    for (uint32_t k0 = blockIdx.x * blockDim.x; k0 < count; k0 += gridDim.x * blockDim.x) {  // uniform per block
        const uint32_t k = k0 + threadIdx.x;
        const bool valid = k < count;
        int slot[K], first[K];  // binary node and first position of each slot
        int ns = 0;
        uint32_t inner = 0;  // bit c: slot c is an inner node
        if (valid) {
            const int2 w = level == 0 ? make_int2(root, 0) : wide[start + k];
            const int4 lb = w.x < n - 1 ? t.links[w.x] : make_int4(0, 0, (int)kSelLeaf, 0);
            if (level == 0 && (lb.z & (int)kSelLeaf)) {  // the whole scene is one leaf
                slot[0] = w.x;
                first[0] = 0;
                ns = 1;
            } else {
                int stn[K], sti[K], stf[K];  // pending (node, slots, first position); their slots sum to at most K
                int sp = 0;
                const int jw = sel_of(lb.z, 0);
                stn[sp] = lb.y;
                stf[sp] = w.y + lb.w;
                sti[sp++] = K - jw;
                stn[sp] = lb.x;
                stf[sp] = w.y;
                sti[sp++] = jw;
                while (sp > 0) {
                    --sp;
                    const int x = stn[sp], f0 = stf[sp];
                    int si = sti[sp];
                    const int4 lx = x < n - 1 ? t.links[x] : make_int4(0, 0, (int)kSelLeaf, 0);
                    while (si > 1 && sel_of(lx.z, si - 1) == 0) si--;
                    if (si <= 1 || sp + 2 > K) {  // (the stack cannot overflow: its slots sum to at most K)
                        if (ns < K) {
                            if (!(lx.z & (int)kSelLeaf)) inner |= 1u << ns;
                            first[ns] = f0;
                            slot[ns++] = x;
                        }
                        continue;
                    }
                    const int pick = sel_of(lx.z, si - 1);
                    stn[sp] = lx.y;
                    stf[sp] = f0 + lx.w;
                    sti[sp++] = si - pick;
                    stn[sp] = lx.x;
                    stf[sp] = f0;
                    sti[sp++] = pick;
                }
            }
        }
        // ids of the inner children
        const uint32_t mine = __popc(inner);
        uint32_t x = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        const int warp = threadIdx.x >> 5;
        if (lane == 31) s_inner[warp] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (int w = 0; w < 4; w++) {
            const uint32_t c = s_inner[w];
            if (w < warp) before += c;
            all += c;
        }
        if (threadIdx.x == 0) s_child = all ? atomicAdd(&bc->level[level + 1], all) : 0;
        __syncthreads();
        uint32_t child = start + count + s_child + before + x - mine;
        __syncthreads();
        if (!valid) continue;
        float f[8 * K];
        float3 rlo = f3(FLT_MAX, FLT_MAX, FLT_MAX), rhi = f3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
#pragma unroll
        for (int c = 0; c < K; c++) {
            float3 lo = f3(1e30f, 1e30f, 1e30f), hi = lo;  // empty slot: a point box far away
            int item = ptd::kNoItem;
            if (c < ns) {
                const int y = slot[c];
                const NodeBox b = load_box(t.nb, y);
                padded(b.lo, b.hi, scene_mag, lo, hi);
                const float ex = hi.x - lo.x, ey = hi.y - lo.y, ez = hi.z - lo.z;
                const float a = ex * ey + ey * ez + ez * ex;
                if ((inner >> c) & 1u) {
                    item = (int)child;
                    wide[child++] = make_int2(y, first[c]);
                    sah += (double)a * (double)kCostNode;
                } else {
                    item = ptd::make_leaf(first[c], b.count());
                    leaf_positions(t, y, first[c], order, leaf_order);
                    sah += (double)a * (double)kCostPrim * b.count();
                }
                rlo = f3(fminf(rlo.x, lo.x), fminf(rlo.y, lo.y), fminf(rlo.z, lo.z));
                rhi = f3(fmaxf(rhi.x, hi.x), fmaxf(rhi.y, hi.y), fmaxf(rhi.z, hi.z));
            }
            f[c] = lo.x;
            f[K + c] = hi.x;
            f[2 * K + c] = lo.y;
            f[3 * K + c] = hi.y;
            f[4 * K + c] = lo.z;
            f[5 * K + c] = hi.z;
            f[6 * K + c] = __int_as_float(item);
            f[7 * K + c] = 0.f;
        }
        float4 *node = reinterpret_cast<float4 *>(nodes) + (size_t)(start + k) * 2 * K;
        const uint32_t x4 = ptd::node_swizzle<K>(start + k) / 4;
#pragma unroll
        for (int i = 0; i < K; i++) {
            const float4 a = make_float4(f[8 * i], f[8 * i + 1], f[8 * i + 2], f[8 * i + 3]);
            const float4 b = make_float4(f[8 * i + 4], f[8 * i + 5], f[8 * i + 6], f[8 * i + 7]);
            ptd::st8(node + ((2 * i) ^ (x4 & ~1u)), x4 & 1 ? b : a, x4 & 1 ? a : b);
        }
        if (level == 0) {
            const double ex = rhi.x - rlo.x, ey = rhi.y - rlo.y, ez = rhi.z - rlo.z;
            bc->root_area = ex * ey + ey * ez + ez * ex;
        }
    }
    for (int o = 16; o > 0; o >>= 1) sah += __shfl_xor_sync(FULL, sah, o);
    if (lane == 0) atomicAdd(&s_sah, sah);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&bc->sah, s_sah);
}

// A scene without primitives: one node of empty slots.
template <int K>
__global__ void k_empty_root(float *nodes) {
    if (threadIdx.x < 8 * K)
        nodes[threadIdx.x] = threadIdx.x < 6 * K ? 1e30f : threadIdx.x < 7 * K ? __int_as_float(ptd::kNoItem) : 0.f;
}

// 7. primitive records into leaf order, one float4 a thread.
__global__ void k_gather_prims(const float4 *src, const uint32_t *order, uint32_t n, float4 *dst) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t k = i / 3, j = i - 3 * k;
    if (k >= n) return;
    dst[3 * (size_t)k + j] = src[3 * (size_t)order[k] + j];
}

// Refit of the nodes [first, last), K lanes a node, one a slot: leaf slots from
// the primitives, inner slots from the union of the child node's slots (deeper
// levels are refit first).  Returns the slots' SAH cost; plo, phi: this lane's box.
template <int K>
__device__ __forceinline__ double refit_node(float *nodes, uint32_t i, uint32_t c, const float4 *prims_bvh,
                                             float scene_mag, float3 &plo, float3 &phi) {
    float *node = nodes + (size_t)i * 8 * K;
    const uint32_t swz = ptd::node_swizzle<K>(i);
    const int item = __float_as_int(node[(6 * K + c) ^ swz]);
    plo = f3(FLT_MAX, FLT_MAX, FLT_MAX);
    phi = f3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    if (item == ptd::kNoItem) return 0.0;
    const int cnt = item_count(item);
    float4 lo = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.f), hi = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, 0.f);
    if (cnt > 0) {
        const int at = ptd::leaf_first(item);
        for (int j = 0; j < cnt; j += 2) {  // two at a time (the last alone: twice)
            float3 a, b, a2, b2;
            prim_box(prims_bvh, (uint32_t)(at + j), a, b);
            prim_box(prims_bvh, (uint32_t)(at + min(j + 1, cnt - 1)), a2, b2);
            lo = make_float4(fminf(lo.x, fminf(a.x, a2.x)), fminf(lo.y, fminf(a.y, a2.y)),
                             fminf(lo.z, fminf(a.z, a2.z)), 0.f);
            hi = make_float4(fmaxf(hi.x, fmaxf(b.x, b2.x)), fmaxf(hi.y, fmaxf(b.y, b2.y)),
                             fmaxf(hi.z, fmaxf(b.z, b2.z)), 0.f);
        }
    } else {
        const float4 *rec = reinterpret_cast<const float4 *>(nodes) + (size_t)item * 2 * K;
        float f[8 * K];
#pragma unroll
        for (int q = 0; q < (7 * K + 3) / 4; q++) {
            const float4 v = rec[q ^ (ptd::node_swizzle<K>(item) / 4)];
            f[4 * q] = v.x;
            f[4 * q + 1] = v.y;
            f[4 * q + 2] = v.z;
            f[4 * q + 3] = v.w;
        }
#pragma unroll
        for (int g = 0; g < K; g++) {
            if (__float_as_int(f[6 * K + g]) == ptd::kNoItem) continue;
            lo = make_float4(fminf(lo.x, f[g]), fminf(lo.y, f[2 * K + g]), fminf(lo.z, f[4 * K + g]), 0.f);
            hi = make_float4(fmaxf(hi.x, f[K + g]), fmaxf(hi.y, f[3 * K + g]), fmaxf(hi.z, f[5 * K + g]), 0.f);
        }
    }
    padded(lo, hi, scene_mag, plo, phi);
    node[c ^ swz] = plo.x;
    node[(K + c) ^ swz] = phi.x;
    node[(2 * K + c) ^ swz] = plo.y;
    node[(3 * K + c) ^ swz] = phi.y;
    node[(4 * K + c) ^ swz] = plo.z;
    node[(5 * K + c) ^ swz] = phi.z;
    const float ex = phi.x - plo.x, ey = phi.y - plo.y, ez = phi.z - plo.z;
    const float area = ex * ey + ey * ez + ez * ex;
    return (double)area * (cnt > 0 ? (double)kCostPrim * cnt : (double)kCostNode);
}
// The SAH sum's partial sums, 32 bytes apart: with one of them, a warp's atomic add
// at a time, the sum alone took 2 ns a warp, 100 us for the widest level.
constexpr uint32_t kSahSums = 64, kSahStride = 4;
constexpr size_t kSahDoubles = 1 + kSahSums * kSahStride;  // the root's area, then the sums
__device__ __forceinline__ void add_sah(double sah, double *acc) {
    for (int o = 16; o > 0; o >>= 1) sah += __shfl_xor_sync(0xffffffffu, sah, o);
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if ((threadIdx.x & 31) == 0 && sah != 0.0) atomicAdd(acc + 1 + warp % kSahSums * kSahStride, sah);
}

// One level, also summing the SAH cost.  Bound by the latency of its
// gathers: 4.1M triangles (1.15M nodes), all levels with the SAH sum 0.17 ms, 0.53
// with a thread a node, every level its own launch and the SAH in a pass of its
// own.  One launch in which the last child's lanes go on with the parent (a counter
// and two fences a node) took 0.26.
template <int K>
__global__ void __launch_bounds__(128) k_refit_level(float *nodes, uint32_t first, uint32_t last,
                                                     const float4 *prims_bvh, float scene_mag, double *acc) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, i = first + t / K;
    float3 plo, phi;
    add_sah(i < last ? refit_node<K>(nodes, i, t % K, prims_bvh, scene_mag, plo, phi) : 0.0, acc);
}

// The levels from `top` up to the root (short ones, at most kTopLevels of them) in
// one block, and the root's area into acc[0].
constexpr int kTopLevels = 32;
constexpr uint32_t kTopNodes = 256;  // of a level refit by one block
struct TopLevels {
    uint32_t start[kTopLevels + 1];  // first node of each level from the root down, then the end
};
template <int K>
__global__ void __launch_bounds__(1024) k_refit_top(float *nodes, TopLevels lv, int levels, const float4 *prims_bvh,
                                                    float scene_mag, double *acc) {
    double sah = 0.0;
    float3 plo = f3(0.f, 0.f, 0.f), phi = plo;
    for (int l = levels - 1; l >= 0; l--) {
        for (uint32_t t = threadIdx.x; t / K < lv.start[l + 1] - lv.start[l]; t += blockDim.x)
            sah += refit_node<K>(nodes, lv.start[l] + t / K, t % K, prims_bvh, scene_mag, plo, phi);
        __syncthreads();  // the level above reads these nodes
    }
    if (threadIdx.x < K) {  // each holds its slot of the root
        const unsigned slots = (1u << K) - 1u;
        for (int o = 1; o < K; o <<= 1) {
            plo = f3(fminf(plo.x, __shfl_xor_sync(slots, plo.x, o)), fminf(plo.y, __shfl_xor_sync(slots, plo.y, o)),
                     fminf(plo.z, __shfl_xor_sync(slots, plo.z, o)));
            phi = f3(fmaxf(phi.x, __shfl_xor_sync(slots, phi.x, o)), fmaxf(phi.y, __shfl_xor_sync(slots, phi.y, o)),
                     fmaxf(phi.z, __shfl_xor_sync(slots, phi.z, o)));
        }
        const double ex = phi.x - plo.x, ey = phi.y - plo.y, ez = phi.z - plo.z;
        if (threadIdx.x == 0) acc[0] = plo.x <= phi.x ? ex * ey + ey * ez + ez * ex : 0.0;
    }
    __syncthreads();
    add_sah(sah, acc);
}

// World-space re-transform of one mesh instance's vertices (same arithmetic
// order as the host flattening: x' = m0*x + m1*y + m2*z + m3, unfused).
__global__ void k_transform_vertices(const float *obj, uint32_t nv, float4 m0, float4 m1, float4 m2, float4 *vpos) {
    uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    float x = obj[3 * v], y = obj[3 * v + 1], z = obj[3 * v + 2];
    float wx = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m0.x, x), __fmul_rn(m0.y, y)), __fmul_rn(m0.z, z)), m0.w);
    float wy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m1.x, x), __fmul_rn(m1.y, y)), __fmul_rn(m1.z, z)), m1.w);
    float wz = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m2.x, x), __fmul_rn(m2.y, y)), __fmul_rn(m2.z, z)), m2.w);
    vpos[v] = make_float4(wx, wy, wz, 0.f);
}
// A vertex of a triangle per thread, so that a record is written in one piece (4.1M triangles
// 68 us; a triangle per thread 100).
__global__ void k_rebuild_tri_records(const uint32_t *tri_vidx, const float4 *vpos, uint32_t first, uint32_t count,
                                      float4 *prims) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t t = j / 3, v = j - 3 * t;
    if (t >= count) return;
    const size_t at = 3 * (size_t)first + j;
    const float4 a = vpos[tri_vidx[at]];
    prims[at] = make_float4(a.x, a.y, a.z, v == 0 ? __int_as_float((int)(first + t)) : 0.f);  // its id
}

// All mesh instances at once: world vertex v belongs to the instance whose
// range [vstart, vstart + count) holds it (binary search over vstart).
struct XformRec {
    uint32_t vstart, count, src;  // world vertex range, first object vertex of its mesh
    uint32_t pad;
    float4 m0, m1, m2;
};
__global__ void k_transform_all(const float *obj, const XformRec *recs, uint32_t nrec, uint32_t total, float4 *vpos) {
    uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= total) return;
    uint32_t lo = 0, hi = nrec - 1;
    while (lo < hi) {
        uint32_t mid = (lo + hi + 1) >> 1;
        if (recs[mid].vstart <= v) lo = mid;
        else hi = mid - 1;
    }
    const XformRec r = recs[lo];
    uint32_t k = r.src + (v - r.vstart);
    float x = obj[3 * (size_t)k], y = obj[3 * (size_t)k + 1], z = obj[3 * (size_t)k + 2];
    float wx = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.m0.x, x), __fmul_rn(r.m0.y, y)), __fmul_rn(r.m0.z, z)), r.m0.w);
    float wy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.m1.x, x), __fmul_rn(r.m1.y, y)), __fmul_rn(r.m1.z, z)), r.m1.w);
    float wz = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r.m2.x, x), __fmul_rn(r.m2.y, y)), __fmul_rn(r.m2.z, z)), r.m2.w);
    vpos[v] = make_float4(wx, wy, wz, 0.f);
}

inline uint32_t blocks(size_t n, int b) { return (uint32_t)((n + b - 1) / b); }

// Compressed copies of 8-wide float nodes (layout in pt_traverse.cuh, same
// node indices).  The grid origin is the low corner of the union of the
// children's boxes; each axis's cell size is the smallest power of two for
// which 255 cells span the union; each child's cells are rounded outwards and
// then checked with the same fused multiply-add the traversal evaluates, so
// the decoded box always encloses the child's padded float box.  Children go
// to slots by a greedy matching on dot(child centroid - node centroid,
// direction of the slot's octant), smallest first (Ylitie, Karras and Laine,
// HPG 2017): slot s holds the child met first by rays of octant s.
__global__ void k_compress8(const float *nodes, uint32_t n, float4 *out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float *f = nodes + (size_t)i * 64;
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        uint32_t occupied = 0;
        for (int c = 0; c < 8; c++) {
            if (__float_as_int(f[48 + c]) == ptd::kNoItem) continue;
            occupied |= 1u << c;
            for (int a = 0; a < 3; a++) {
                lo[a] = fminf(lo[a], f[16 * a + c]);
                hi[a] = fmaxf(hi[a], f[16 * a + 8 + c]);
            }
        }
        float4 *q = out + (size_t)i * ptd::kCwFloat4;
        if (!occupied) {
            q[0] = make_float4(0.f, 0.f, 0.f, __uint_as_float(127u | 127u << 8 | 127u << 16));
            q[1] = q[2] = q[3] = make_float4(0.f, 0.f, 0.f, 0.f);
            q[4] = q[5] = make_float4(__int_as_float(ptd::kNoItem), __int_as_float(ptd::kNoItem),
                                      __int_as_float(ptd::kNoItem), __int_as_float(ptd::kNoItem));
            continue;
        }
        uint32_t eb[3];
        float cell[3];
        for (int a = 0; a < 3; a++) {
            const float r = __fdiv_ru(__fsub_ru(hi[a], lo[a]), 255.f);
            uint32_t e = 1;
            if (r > 0.f) {
                const uint32_t bits = __float_as_uint(r);
                e = (bits >> 23) + ((bits & 0x7fffffu) ? 1u : 0u);
                e = e < 1u ? 1u : e;
            }
            while (e < 254u && __fmaf_rn(255.f, __uint_as_float(e << 23), lo[a]) < hi[a]) e++;
            eb[a] = e;
            cell[a] = __uint_as_float(e << 23);
        }
        // slot assignment
        float cen[8][3];
        for (int c = 0; c < 8; c++)
            for (int a = 0; a < 3; a++)
                cen[c][a] = (occupied >> c) & 1u ? 0.5f * (f[16 * a + c] + f[16 * a + 8 + c]) - 0.5f * (lo[a] + hi[a])
                                                 : 0.f;
        int slot_of[8];
        for (int c = 0; c < 8; c++) slot_of[c] = -1;
        uint32_t used = 0, todo = occupied;
        while (todo) {
            float best = FLT_MAX;
            int bc = -1, bs = -1;
            for (int c = 0; c < 8; c++) {
                if (!((todo >> c) & 1u)) continue;
                for (int sl = 0; sl < 8; sl++) {
                    if ((used >> sl) & 1u) continue;
                    const float cost = (sl & 1 ? -cen[c][0] : cen[c][0]) + (sl & 2 ? -cen[c][1] : cen[c][1]) +
                                       (sl & 4 ? -cen[c][2] : cen[c][2]);
                    if (bc < 0 || cost < best) {
                        best = cost;
                        bc = c;
                        bs = sl;
                    }
                }
            }
            slot_of[bc] = bs;
            used |= 1u << bs;
            todo &= ~(1u << bc);
        }
        uint32_t cl[3][2] = {{0, 0}, {0, 0}, {0, 0}}, ch[3][2] = {{0, 0}, {0, 0}, {0, 0}};
        int items[8];
        for (int sl = 0; sl < 8; sl++) items[sl] = ptd::kNoItem;
        for (int c = 0; c < 8; c++) {
            const int sl = slot_of[c];
            if (sl < 0) continue;
            for (int a = 0; a < 3; a++) {
                const float clo = f[16 * a + c], chi = f[16 * a + 8 + c];
                const float inv_cell = __frcp_rn(cell[a]);
                int ql = (int)floorf(__fmul_rd(__fsub_rd(clo, lo[a]), inv_cell));
                ql = min(max(ql, 0), 255);
                while (ql > 0 && __fmaf_rn((float)ql, cell[a], lo[a]) > clo) ql--;
                int qh = (int)ceilf(__fmul_ru(__fsub_ru(chi, lo[a]), inv_cell));
                qh = min(max(qh, 0), 255);
                while (qh < 255 && __fmaf_rn((float)qh, cell[a], lo[a]) < chi) qh++;
                cl[a][sl >> 2] |= (uint32_t)ql << (8 * (sl & 3));
                ch[a][sl >> 2] |= (uint32_t)qh << (8 * (sl & 3));
            }
            items[sl] = __float_as_int(f[48 + c]);
        }
        q[0] = make_float4(lo[0], lo[1], lo[2], __uint_as_float(eb[0] | eb[1] << 8 | eb[2] << 16 | used << 24));
        for (int a = 0; a < 3; a++)
            q[1 + a] = make_float4(__uint_as_float(cl[a][0]), __uint_as_float(cl[a][1]), __uint_as_float(ch[a][0]),
                                   __uint_as_float(ch[a][1]));
        q[4] = make_float4(__int_as_float(items[0]), __int_as_float(items[1]), __int_as_float(items[2]),
                           __int_as_float(items[3]));
        q[5] = make_float4(__int_as_float(items[4]), __int_as_float(items[5]), __int_as_float(items[6]),
                           __int_as_float(items[7]));
    }
}

// Scratch of a build: one allocation, carved.
struct Scratch {
    uint64_t *keys[2];
    uint32_t *vals[2];
    uint32_t *hist, *digit_total;
    float4 *pbox;
    int *parent, *flags;  // radix tree only
    int *cl[2], *out_id;  // PLOC
    uint32_t *tile_count;
    int2 *wide;           // of each wide node: its binary node, its first primitive's position
    Tree tree;
    BuildCounts *counts;
};

// Carves the scratch for n primitives from base; returns the bytes taken.
size_t carve(Scratch &sc, char *base, size_t n, uint32_t tiles, int K) {
    size_t at = 0;
    auto take = [&](auto *&p, size_t count) {
        using T = std::remove_reference_t<decltype(*p)>;
        p = reinterpret_cast<T *>(base + at);
        at += (count * sizeof(T) + 255) & ~size_t(255);
    };
    take(sc.counts, 1);
    take(sc.keys[0], n);
    take(sc.keys[1], n);
    take(sc.vals[0], n);
    take(sc.vals[1], n);
    take(sc.hist, (size_t)256 * tiles);
    take(sc.digit_total, 256);
    take(sc.pbox, 2 * n);
    take(sc.parent, 2 * n);
    take(sc.flags, n);
    take(sc.cl[0], n);
    take(sc.cl[1], n);
    take(sc.out_id, n);
    take(sc.tile_count, n / ploc_tile(1) + 1);
    take(sc.wide, n);
    take(sc.tree.links, n);
    take(sc.tree.nb, 4 * n);
    take(sc.tree.dval, (size_t)K * n);
    return at;
}

// The collapse, the records in leaf order and the counts (level_start, SAH
// cost, *sah) read back.  *ok = false: clustering failed, or the wide tree is
// deeper than max_levels.
template <int K>
int build_wide(pt_scene *s, const Scratch &sc, uint32_t n, int root, uint32_t max_levels, float *sah, bool *ok,
               cudaStream_t st) {
    *ok = true;
    s->level_start.clear();
    int e = s->nodes.ensure((size_t)std::max<uint32_t>(1, n > 1 ? n - 1 : 1) * 32 * K);
    if (e != PT_OK) return e;
    float *nodes = s->nodes.as<float>();
    if (n == 0) {
        k_empty_root<K><<<1, 64, 0, st>>>(nodes);
        PT_CUDA_TRY(cudaGetLastError());
        s->level_start = {0, 1};
        *sah = 0.f;
        return PT_OK;
    }
    BuildCounts *bc = sc.counts;
    PT_CUDA_TRY(cudaMemsetAsync(&bc->sah, 0, 2 * sizeof(double) + sizeof(bc->level), st));
    const uint32_t one = 1;
    PT_CUDA_TRY(cudaMemcpyAsync(bc->level, &one, sizeof(one), cudaMemcpyHostToDevice, st));
    // levels in batches; a launch past the last level returns at once
    constexpr int kBatch = 20;
    BuildCounts h;
    const size_t head = offsetof(BuildCounts, clusters);
    const uint32_t most = std::min<uint32_t>(blocks(n, 128), (uint32_t)s->num_sms * 16u);
    uint32_t bound = 1;  // nodes of a level: at most K times the level above, and n - 1
    int level = 0;
    for (bool more = true; more && level < kMaxLevels;) {
        const int end = std::min(level + (level ? 8 : kBatch), kMaxLevels);
        for (; level < end; level++) {
            k_collapse<K><<<std::min(most, blocks(bound, 128)), 128, 0, st>>>(sc.tree, bc, level, root, sc.wide, nodes,
                                                                             s->scene_mag, sc.vals[0],
                                                                             s->bvh_order.as<uint32_t>());
            bound = std::min<uint32_t>(n, bound * K);
        }
        PT_CUDA_TRY(cudaGetLastError());
        PT_CUDA_TRY(cudaMemcpyAsync(&h, bc, head, cudaMemcpyDeviceToHost, st));
        PT_CUDA_TRY(cudaStreamSynchronize(st));
        more = !h.fail && h.level[end] != 0;
    }
    uint32_t start = 0;
    for (int l = 0; l <= kMaxLevels && h.level[l]; l++) {
        s->level_start.push_back(start);
        start += h.level[l];
    }
    s->level_start.push_back(start);
    if (h.fail || h.level[kMaxLevels] || s->level_start.size() - 1 > max_levels) {
        *ok = false;
        return PT_OK;
    }
    k_gather_prims<<<blocks(3 * (size_t)n, 256), 256, 0, st>>>(s->prims_world.as<float4>(), s->bvh_order.as<uint32_t>(),
                                                               n, s->prims_bvh.as<float4>());
    PT_CUDA_TRY(cudaGetLastError());
    *sah = h.root_area > 0 ? (float)((kCostNode * h.root_area + h.sah) / h.root_area) : 0.f;
    return PT_OK;
}

template <int K>
void refit_tree(pt_scene *s, cudaStream_t st) {
    float *nodes = s->nodes.as<float>();
    const float4 *prims = s->prims_bvh.as<float4>();
    double *acc = s->sah_scratch.as<double>();
    const std::vector<uint32_t> &ls = s->level_start;
    const int levels = (int)ls.size() - 1;
    TopLevels tl = {};
    int top = 0;  // levels of the last launch
    while (top < std::min(levels, kTopLevels) && ls[top + 1] - ls[top] <= kTopNodes) {
        tl.start[top] = ls[top];
        tl.start[top + 1] = ls[top + 1];
        top++;
    }
    for (int l = levels - 1; l >= top; l--)
        k_refit_level<K><<<blocks((size_t)(ls[l + 1] - ls[l]) * K, 128), 128, 0, st>>>(nodes, ls[l], ls[l + 1], prims,
                                                                                      s->scene_mag, acc);
    k_refit_top<K><<<1, 1024, 0, st>>>(nodes, tl, top, prims, s->scene_mag, acc);
}

// PLOC over the sorted order in sc.vals[0] (n >= 2); the root is node n - 2.
// *stalled: clustering made no progress (boxes without a finite area); the
// caller then builds the radix tree.
template <int K>
int ploc_build(const Scratch &sc, uint32_t n, bool *stalled, cudaStream_t st) {
    *stalled = false;
    BuildCounts *bc = sc.counts;
    PT_CUDA_TRY(cudaMemcpyAsync(bc->clusters, &n, sizeof(n), cudaMemcpyHostToDevice, st));
    uint32_t bound = n;  // clusters, at most
    int cur = 0, pass = 0;
    while (bound > (uint32_t)kPlocTail) {
        if (pass + kPlocPassesPerRead > kPlocMaxPasses) {
            *stalled = true;
            return PT_OK;
        }
        const bool wide = bound >= kPlocWide;
        const uint32_t tile = (uint32_t)ploc_tile(wide ? 4 : 1), tiles = (bound + tile - 1) / tile;
        for (int k = 0; k < kPlocPassesPerRead; k++, pass++, cur ^= 1) {
            if (wide) {
                k_ploc_merge<K, 4><<<tiles, kPlocThreads, 0, st>>>(sc.tree, bc, pass, sc.cl[cur], sc.out_id,
                                                                  sc.tile_count);
                k_ploc_compact<4><<<tiles, kPlocThreads, 0, st>>>(bc, pass, sc.out_id, sc.tile_count, sc.cl[cur ^ 1]);
            } else {
                k_ploc_merge<K, 1><<<tiles, kPlocThreads, 0, st>>>(sc.tree, bc, pass, sc.cl[cur], sc.out_id,
                                                                  sc.tile_count);
                k_ploc_compact<1><<<tiles, kPlocThreads, 0, st>>>(bc, pass, sc.out_id, sc.tile_count, sc.cl[cur ^ 1]);
            }
        }
        PT_CUDA_TRY(cudaGetLastError());
        uint32_t m = 0;
        PT_CUDA_TRY(cudaMemcpyAsync(&m, bc->clusters + pass, sizeof(m), cudaMemcpyDeviceToHost, st));
        PT_CUDA_TRY(cudaStreamSynchronize(st));
        if (m == 0 || m >= bound) {
            *stalled = true;
            return PT_OK;
        }
        bound = m;
    }
    constexpr int smem = (kPlocTail + 2 * kPlocRadius) * 32 + kPlocTail * 8;
    PT_CUDA_TRY(cudaFuncSetAttribute(k_ploc_tail<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_ploc_tail<K><<<1, 1024, smem, st>>>(sc.tree, bc, pass, sc.cl[cur]);
    PT_CUDA_TRY(cudaGetLastError());
    return PT_OK;
}

template <int K>
int build_tree(pt_scene *s, const pt_bvh_opts *o, cudaStream_t st, float *sah, bool *clustered) {
    const uint32_t n = s->num_prims;
    const uint32_t tiles = std::max<uint32_t>(1, (n + kSortTile - 1) / kSortTile);
    const size_t nn = std::max<uint32_t>(n, 2);
    Scratch sc;
    int e = s->bvh_scratch.ensure(carve(sc, nullptr, nn, tiles, K));
    if (e != PT_OK) return e;
    carve(sc, static_cast<char *>(s->bvh_scratch.ptr), nn, tiles, K);
    sc.tree.n = (int)n;
    sc.tree.max_leaf = (int)o->max_leaf_size;
    if ((e = s->bvh_order.ensure(std::max<size_t>(4 * (size_t)n, 16))) != PT_OK) return e;
    if ((e = s->prims_bvh.ensure(std::max<size_t>(48 * (size_t)n, 48))) != PT_OK) return e;

    const int tb = 256;
    PT_CUDA_TRY(cudaMemsetAsync(sc.counts, 0, sizeof(BuildCounts), st));
    PT_CUDA_TRY(cudaMemsetAsync(sc.counts->centroid, 0xff, 3 * sizeof(uint32_t), st));
    if (n > 0) {
        k_prim_bounds<<<std::min<uint32_t>(blocks(n, tb), (uint32_t)s->num_sms * 8u), tb, 0, st>>>(s->prims_world.as<float4>(), n, sc.pbox, sc.counts->centroid);
        k_morton<<<blocks(n, tb), tb, 0, st>>>(sc.pbox, n, sc.counts->centroid, sc.keys[0], sc.vals[0]);
        PT_CUDA_TRY(cudaFuncSetAttribute(k_radix_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, kScatterSmem));
        for (int pass = 0, cur = 0; pass < 8; pass++, cur ^= 1) {  // back in buffer 0 after 8 passes
            const int shift = pass * 8;
            k_radix_hist<<<tiles, kSortThreads, 0, st>>>(sc.keys[cur], n, shift, sc.hist, tiles);
            k_radix_scan<<<256, 256, 0, st>>>(sc.hist, tiles, sc.digit_total);
            k_radix_scatter<<<tiles, kSortThreads, kScatterSmem, st>>>(sc.keys[cur], sc.vals[cur], sc.keys[cur ^ 1], sc.vals[cur ^ 1],
                                                             n, shift, sc.hist, tiles, sc.digit_total);
        }
        k_leaf_boxes<<<blocks(n, tb), tb, 0, st>>>((int)n, sc.vals[0], sc.pbox, sc.tree.nb, sc.cl[0]);
        PT_CUDA_TRY(cudaGetLastError());
    }
    // binary tree: PLOC by default, the radix tree for PT_BVH_FAST_BUILD, for
    // a PLOC build that did not converge, or one whose wide tree is deeper
    // than the traversal stack covers (kShortStack + kSpillStack entries)
    const auto radix_tree = [&]() -> int {
        PT_CUDA_TRY(cudaMemsetAsync(&sc.counts->fail, 0, sizeof(uint32_t), st));
        if (n == 0) return PT_OK;  // no primitives: nothing to sort or link (2n - 1 would wrap)
        PT_CUDA_TRY(cudaMemsetAsync(sc.parent, 0xff, 4 * (2 * (size_t)n - 1), st));
        PT_CUDA_TRY(cudaMemsetAsync(sc.flags, 0, 4 * (size_t)n, st));
        if (n > 1)
            k_karras<<<blocks(n - 1, tb), tb, 0, st>>>(sc.keys[0], (int)n, sc.tree.links, sc.parent);
        k_bottom_up<K><<<blocks(n, tb), tb, 0, st>>>(sc.tree, sc.parent, sc.flags);
        PT_CUDA_TRY(cudaGetLastError());
        return PT_OK;
    };
    // curve pieces (long, thin, often diagonal) trace faster under the radix
    // tree although PLOC gives them a lower SAH cost, so curve-dominated scenes
    // use it: 50,000 cubic strands at 1080p, 64 spp 646 against 622 Msamples/s, linear
    // ones at 16 spp 65.6 against 68.8 ms, 10,000 cubic 52.1 against 52.9 (641 x 361, 8
    // spp 4.34 / 4.46, but 2,000 3.54 / 3.48 and 300 1.87 / 1.76); build 1.6 / 2.4 ms
    const bool curve_heavy = 2ull * s->num_curve_pieces > n;
    *clustered = n > 1 && !(o->flags & PT_BVH_FAST_BUILD) && !curve_heavy;
    if (*clustered) {
        bool stalled = false;
        if ((e = ploc_build<K>(sc, n, &stalled, st)) != PT_OK) return e;
        bool ok = false;
        const uint32_t stack_levels = (uint32_t)ptd::kTraversalStackEntries / (uint32_t)(K - 1);
        if (!stalled && (e = build_wide<K>(s, sc, n, (int)n - 2, stack_levels, sah, &ok, st)) != PT_OK) return e;
        if (ok) return PT_OK;
        *clustered = false;
    }
    if ((e = radix_tree()) != PT_OK) return e;
    bool ok = false;
    if ((e = build_wide<K>(s, sc, n, 0, kMaxLevels, sah, &ok, st)) != PT_OK) return e;
    if (!ok) {
        pt_set_error("pt_bvh_build: the tree is deeper than %d levels", kMaxLevels);
        return PT_ERR_UNSUPPORTED;
    }
    return PT_OK;
}

}  // namespace

int pt_bvh_build_impl(pt_scene *s, const pt_bvh_opts *o, cudaStream_t st) {
    pt_nvtx::Range nv("pt_bvh_build");
    const uint32_t n = s->num_prims;
    const int K = (int)o->width;
    PT_CUDA_TRY(cudaEventRecord(s->ev0, st));
    float sah = 0.f;
    bool clustered = false;
    int e;
    switch (K) {
        case 2: e = build_tree<2>(s, o, st, &sah, &clustered); break;
        case 4: e = build_tree<4>(s, o, st, &sah, &clustered); break;
        default: e = build_tree<8>(s, o, st, &sah, &clustered); break;
    }
    if (e != PT_OK) return e;
    if (o->width == 8) {  // the traversal reads compressed copies of the 8-wide nodes
        const uint32_t nn = s->level_start.back();
        if ((e = s->cnodes.ensure((size_t)std::max<uint32_t>(nn, 1) * 16 * ptd::kCwFloat4)) != PT_OK) return e;
        if ((e = pt_compress_wide8(s->nodes.as<float>(), nn, s->cnodes.as<float4>(), st)) != PT_OK) return e;
    }
    PT_CUDA_TRY(cudaEventRecord(s->ev1, st));
    PT_CUDA_TRY(cudaEventSynchronize(s->ev1));
    float ms = 0.f;
    PT_CUDA_TRY(cudaEventElapsedTime(&ms, s->ev0, s->ev1));
    s->bvh_opts = *o;

    pt_bvh_stats &bs = s->bvh_stats;
    bs.width = o->width;
    bs.num_nodes = s->level_start.back();
    bs.num_prims = n;
    bs.max_depth = (uint32_t)s->level_start.size() - 1;
    bs.sah_cost = sah;
    bs.build_ms = ms;
    bs.node_bytes = (uint64_t)bs.num_nodes * (K == 8 ? 16 * ptd::kCwFloat4 : 32 * K);  // the bytes the traversal reads
    bs.builder = clustered ? PT_BVH_BUILDER_PLOC : PT_BVH_BUILDER_RADIX;
    bs.prim_bytes = (uint64_t)n * 48;
    bs.num_leaves = 0;

    ptd::DevScene &d = s->dev;
    d.nodes = s->nodes.as<float4>();
    d.cnodes = o->width == 8 ? s->cnodes.as<float4>() : nullptr;
    d.prims = s->prims_bvh.as<float4>();
    d.width = o->width;
    d.num_nodes = bs.num_nodes;
    uint32_t max_smem = (uint32_t)std::max(0, s->max_smem_per_block - 64 * 1024) / (32 * K);
    d.smem_nodes = o->width == 8 ? 0 : std::min<uint32_t>(std::min(o->smem_nodes, bs.num_nodes), max_smem);
    d.pad_mag = s->scene_mag;
    s->bvh_built = true;
    return PT_OK;
}

int pt_compress_wide8(const float *nodes, uint32_t n, float4 *out, cudaStream_t st) {
    if (n) k_compress8<<<blocks(n, 128), 128, 0, st>>>(nodes, n, out);
    PT_CUDA_TRY(cudaGetLastError());
    return PT_OK;
}

int pt_bvh_refit_impl(pt_scene *s, cudaStream_t st) {
    pt_nvtx::Range nv("pt_bvh_refit");
    const uint32_t n = s->num_prims;
    int e = s->sah_scratch.ensure(kSahDoubles * sizeof(double));
    if (e != PT_OK) return e;
    PT_CUDA_TRY(cudaEventRecord(s->ev0, st));
    PT_CUDA_TRY(cudaMemsetAsync(s->sah_scratch.ptr, 0, kSahDoubles * sizeof(double), st));
    if (n > 0)
        k_gather_prims<<<blocks(3 * (size_t)n, 256), 256, 0, st>>>(s->prims_world.as<float4>(), s->bvh_order.as<uint32_t>(), n,
                                                        s->prims_bvh.as<float4>());
    switch (s->bvh_opts.width) {
        case 2: refit_tree<2>(s, st); break;
        case 4: refit_tree<4>(s, st); break;
        default: refit_tree<8>(s, st); break;
    }
    PT_CUDA_TRY(cudaGetLastError());
    if (s->bvh_opts.width == 8) {
        e = pt_compress_wide8(s->nodes.as<float>(), s->bvh_stats.num_nodes, s->cnodes.as<float4>(), st);
        if (e != PT_OK) return e;
    }
    PT_CUDA_TRY(cudaEventRecord(s->ev1, st));
    double h[kSahDoubles] = {};
    PT_CUDA_TRY(cudaMemcpyAsync(h, s->sah_scratch.ptr, sizeof(h), cudaMemcpyDeviceToHost, st));
    PT_CUDA_TRY(cudaStreamSynchronize(st));
    float ms = 0.f;
    PT_CUDA_TRY(cudaEventElapsedTime(&ms, s->ev0, s->ev1));
    s->bvh_stats.build_ms = ms;
    double sah = 0.0;  // node cost 1.2, primitive cost 1, relative to the root's area
    for (uint32_t k = 0; k < kSahSums; k++) sah += h[1 + k * kSahStride];
    s->bvh_stats.sah_cost = h[0] > 0 ? (float)((kCostNode * h[0] + sah) / h[0]) : 0.f;
    return PT_OK;
}

int pt_update_all_world_vertices(pt_scene *s, const float *d_obj_pos, cudaStream_t st) {
    const uint32_t nrec = (uint32_t)s->mesh_instances.size();
    if (nrec == 0) return PT_OK;
    if (!s->xform_table.ptr) {
        std::vector<uint64_t> mesh_start(s->mesh_num_vertices.size() + 1, 0);
        for (size_t m = 0; m < s->mesh_num_vertices.size(); m++) mesh_start[m + 1] = mesh_start[m] + s->mesh_num_vertices[m];
        std::vector<XformRec> recs(nrec);
        for (uint32_t i = 0; i < nrec; i++) {
            const MeshInstanceRef &r = s->mesh_instances[i];
            const float *m = r.to_world;
            recs[i].vstart = r.vertex_offset;
            recs[i].count = s->mesh_num_vertices[r.mesh];
            recs[i].src = (uint32_t)mesh_start[r.mesh];
            recs[i].pad = 0;
            recs[i].m0 = make_float4(m[0], m[1], m[2], m[3]);
            recs[i].m1 = make_float4(m[4], m[5], m[6], m[7]);
            recs[i].m2 = make_float4(m[8], m[9], m[10], m[11]);
        }
        int e = s->xform_table.ensure(sizeof(XformRec) * nrec);
        if (e != PT_OK) return e;
        PT_CUDA_TRY(cudaMemcpy(s->xform_table.ptr, recs.data(), sizeof(XformRec) * nrec, cudaMemcpyHostToDevice));
    }
    const uint32_t total = s->num_vertices;
    if (total) k_transform_all<<<blocks(total, 256), 256, 0, st>>>(d_obj_pos, s->xform_table.as<XformRec>(), nrec, total,
                                                                   s->vpos.as<float4>());
    if (s->num_tris)
        k_rebuild_tri_records<<<blocks(3 * (size_t)s->num_tris, 256), 256, 0, st>>>(s->tri_vidx.as<uint32_t>(), s->vpos.as<float4>(), 0,
                                                                        s->num_tris, s->prims_world.as<float4>());
    PT_CUDA_TRY(cudaGetLastError());
    PT_CUDA_TRY(cudaStreamSynchronize(st));
    return PT_OK;
}

int pt_update_world_vertices(pt_scene *s, uint32_t mesh, const float *d_obj_pos, uint32_t nv, cudaStream_t st) {
    for (const MeshInstanceRef &r : s->mesh_instances) {
        if (r.mesh != mesh) continue;
        const float *m = r.to_world;
        float4 m0 = make_float4(m[0], m[1], m[2], m[3]), m1 = make_float4(m[4], m[5], m[6], m[7]),
               m2 = make_float4(m[8], m[9], m[10], m[11]);
        if (nv) k_transform_vertices<<<blocks(nv, 256), 256, 0, st>>>(d_obj_pos, nv, m0, m1, m2, s->vpos.as<float4>() + r.vertex_offset);
        uint32_t first = r.prim_offset;
        uint32_t count = 0;
        // triangles of this instance: up to the next mesh instance's first primitive
        uint32_t next = s->num_tris;
        for (const MeshInstanceRef &q : s->mesh_instances)
            if (q.prim_offset > first && q.prim_offset < next) next = q.prim_offset;
        count = next - first;
        if (count) k_rebuild_tri_records<<<blocks(3 * (size_t)count, 256), 256, 0, st>>>(s->tri_vidx.as<uint32_t>(), s->vpos.as<float4>(),
                                                                             first, count, s->prims_world.as<float4>());
    }
    PT_CUDA_TRY(cudaGetLastError());
    PT_CUDA_TRY(cudaStreamSynchronize(st));
    return PT_OK;
}
