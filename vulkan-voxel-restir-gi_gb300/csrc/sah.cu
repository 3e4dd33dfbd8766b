// Batched GPU binned-SAH BVH builder reproducing bvh/build.rs exactly.
//
// The reference builds recursively (subdivide, build.rs:130-233): a node
// with n > 2 prims is split at the best of 3 axes x 31 planes over 32
// centroid bins (find_best_plane, build.rs:45-128), its prim indices are
// partitioned in place, and the two children are appended to the node list
// together before the left subtree is built.  The index of every node is
// therefore a closed form of the split sizes: a node whose children start at
// `base` puts its left child at base, its right child at base+1, the left
// child's children at base+2 and the right child's at base + 2*n_left (a
// subtree of k leaves has 2k-1 nodes).  This builder runs the recursion
// level by level, carrying (node index, children base) so the node array comes
// out in the reference's order without a renumbering pass: trees of up to
// TREE_MAX prims by one CTA each, all levels in one launch (k_sah_tree), larger
// ones in a launch per level over all of them (k_sah_level).
//
// A node is split by a warp, the largest of a CTA's tree by the whole CTA: it
// reduces the node AABB and centroid bounds (order-independent min/max), bins
// prims per axis with shared-memory atomic counts and ordered-integer atomic
// min/max (exact), evaluates the 93 plane costs with the reference's float
// expression, takes the first minimum in (axis, plane) order, and partitions
// the node's slice in a parallel two-sided (Hoare) pass: the k-th
// predicate-false element from the left is swapped with the k-th predicate-true
// element from the right, the pairing of the serial two-pointer partition.  A
// node of up to SMALL_NODE prims takes its plane costs from the prims' boxes,
// without bins.
#include <algorithm>
#include <cfloat>

#include "vrg_internal.h"

namespace vrg {

namespace {

struct Item {
    uint32_t tree, node, base, first, count, parent;
};

constexpr int TREE_THREADS = 512, TREE_WARPS = TREE_THREADS / 32;
constexpr uint32_t TREE_BIG = 256;   // prims above which the whole CTA splits a node
constexpr uint32_t TREE_MAX = 2560;  // prims of a tree one CTA builds (its arrays fill an SM's shared memory)
constexpr int SAH_WARPS = 8;
constexpr int NB = 32;

__device__ __forceinline__ int f2o(float f) {
    int b = __float_as_int(f);
    return b ^ ((b >> 31) & 0x7FFFFFFF);
}
__device__ __forceinline__ float o2f(int o) { return __int_as_float(o ^ ((o >> 31) & 0x7FFFFFFF)); }

__device__ __forceinline__ uint32_t bin_index(float v) {  // Rust `as usize` then min(31)
    if (!(v > 0.0f)) return 0;
    if (v >= 31.0f) return 31;
    return (uint32_t)v;
}

__device__ __forceinline__ float area_of(float lx, float ly, float lz, float hx, float hy, float hz) {
    float dx = hx - lx, dy = hy - ly, dz = hz - lz;
    return 2.0f * ((dx * dy + dx * dz) + dy * dz);  // aabb.rs:44-52
}

// A tree's prims as the splitting reads them: boxes, centroids (w = power) and
// the prim order, by the prim's index in the tree.
struct Prims {
    const float4 *lo, *hi, *cen;
    const uint32_t *id;
    uint32_t *perm;
};

__device__ void write_leaf(const SahOutputs &out, const SahTree &T, const Prims &Q, uint32_t node,
                           uint32_t parent, uint32_t p) {
    const float4 lo = Q.lo[p], hi = Q.hi[p];
    vrg_bvh_node n;
    n.left_node_idx = INVALID;
    n.right_node_idx_or_prim_idx = Q.id[p];
    n.min[0] = lo.x; n.min[1] = lo.y; n.min[2] = lo.z;
    n.power = Q.cen[p].w;
    n.max[0] = hi.x; n.max[1] = hi.y; n.max[2] = hi.z;
    n.parent_idx = parent;
    out.nodes[T.node_off + node] = n;
    out.leaf_prim[T.node_off + node] = p;
}

__device__ void write_internal(const SahOutputs &out, const SahTree &T, uint32_t node, uint32_t parent,
                               uint32_t base, const float lo[3], const float hi[3]) {
    const float pad = 0.0001f;  // build.rs:300
    vrg_bvh_node n;
    n.left_node_idx = base;
    n.right_node_idx_or_prim_idx = base + 1;
    for (int k = 0; k < 3; k++) { n.min[k] = lo[k] - pad; n.max[k] = hi[k] + pad; }
    n.power = 0.0f;
    n.parent_idx = parent;
    out.nodes[T.node_off + node] = n;
    out.leaf_prim[T.node_off + node] = INVALID;
}

// node with exactly two prims: internal node + two leaves in current order
__device__ void write_pair(const SahOutputs &out, const SahTree &T, const Prims &Q, uint32_t node,
                           uint32_t parent, uint32_t base, uint32_t first) {
    const uint32_t p0 = Q.perm[first], p1 = Q.perm[first + 1];
    const float4 a0 = Q.lo[p0], b0 = Q.hi[p0], a1 = Q.lo[p1], b1 = Q.hi[p1];
    const float lo[3] = {fminf(a0.x, a1.x), fminf(a0.y, a1.y), fminf(a0.z, a1.z)};
    const float hi[3] = {fmaxf(b0.x, b1.x), fmaxf(b0.y, b1.y), fmaxf(b0.z, b1.z)};
    write_internal(out, T, node, parent, base, lo, hi);
    write_leaf(out, T, Q, base, node, p0);
    write_leaf(out, T, Q, base + 1, node, p1);
}

struct Bins {
    union {
        struct {
            int cnt[3 * NB], lo[3 * NB][3], hi[3 * NB][3];
        };
        struct {  // a node of few prims: their boxes and the three axes' bins (8 bits each)
            float4 plo[32], phi[32];
            uint32_t pbin[32];
        };
    };
    uint32_t swap[2][32];  // a partition step's values from the left and from the right
};

__device__ __forceinline__ void bins_clear(Bins &B, int i, int step) {
    for (int b = i; b < 3 * NB; b += step) {
        B.cnt[b] = 0;
        for (int k = 0; k < 3; k++) { B.lo[b][k] = f2o(INFINITY); B.hi[b][k] = f2o(-INFINITY); }
    }
}

// one prim into the bins of the three axes (build.rs:68-85)
__device__ __forceinline__ void bins_add(Bins &B, const float clo[3], const float scale[3], float4 a, float4 b,
                                         float4 m) {
    const float cc[3] = {m.x, m.y, m.z};
    const int l0 = f2o(a.x), l1 = f2o(a.y), l2 = f2o(a.z), h0 = f2o(b.x), h1 = f2o(b.y), h2 = f2o(b.z);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int bi = d * NB + (int)bin_index((cc[d] - clo[d]) * scale[d]);
        atomicAdd(&B.cnt[bi], 1);
        atomicMin(&B.lo[bi][0], l0); atomicMin(&B.lo[bi][1], l1); atomicMin(&B.lo[bi][2], l2);
        atomicMax(&B.hi[bi][0], h0); atomicMax(&B.hi[bi][1], h1); atomicMax(&B.hi[bi][2], h2);
    }
}

// a warp's best plane of axis d (build.rs:87-125): lane p holds bin p, the
// left side of plane p is the prefix up to it, the right side the suffix past
// it; cost and key of the first minimum in plane order, in every lane
__device__ __forceinline__ void best_plane(const Bins &B, int d, float &cost, int &key) {
    const int lane = threadIdx.x & 31;
    const int bi = d * NB + lane;
    uint32_t nl = (uint32_t)B.cnt[bi];
    float l[3], h[3], rl[3], rh[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        l[k] = fminf(INFINITY, o2f(B.lo[bi][k]));  // (a bin whose bound is NaN has none)
        h[k] = fmaxf(-INFINITY, o2f(B.hi[bi][k]));
        // the suffix past this lane: starts from the next lane's bin
        rl[k] = __shfl_down_sync(0xffffffffu, l[k], 1);
        rh[k] = __shfl_down_sync(0xffffffffu, h[k], 1);
        if (lane == 31) { rl[k] = INFINITY; rh[k] = -INFINITY; }
    }
    uint32_t nr = __shfl_down_sync(0xffffffffu, nl, 1);
    if (lane == 31) nr = 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t un = __shfl_up_sync(0xffffffffu, nl, o), dn = __shfl_down_sync(0xffffffffu, nr, o);
        if (lane >= o) nl += un;
        if (lane + o < 32) nr += dn;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float ul = __shfl_up_sync(0xffffffffu, l[k], o), uh = __shfl_up_sync(0xffffffffu, h[k], o);
            const float dl = __shfl_down_sync(0xffffffffu, rl[k], o), dh = __shfl_down_sync(0xffffffffu, rh[k], o);
            if (lane >= o) { l[k] = fminf(l[k], ul); h[k] = fmaxf(h[k], uh); }
            if (lane + o < 32) { rl[k] = fminf(rl[k], dl); rh[k] = fmaxf(rh[k], dh); }
        }
    }
    const float al = nl ? area_of(l[0], l[1], l[2], h[0], h[1], h[2]) : 0.0f;
    const float ar = nr ? area_of(rl[0], rl[1], rl[2], rh[0], rh[1], rh[2]) : 0.0f;
    const float c = al * (float)nl + ar * (float)nr;
    cost = FLT_MAX;
    key = 0x7FFFFFFF;
    if (lane < NB - 1 && c < FLT_MAX) {  // (a NaN cost never compares less)
        cost = c;
        key = d * (NB - 1) + lane;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float oc = __shfl_xor_sync(0xffffffffu, cost, o);
        const int ok = __shfl_xor_sync(0xffffffffu, key, o);
        if (oc < cost || (oc == cost && ok < key)) { cost = oc; key = ok; }
    }
}

__device__ __forceinline__ float axis_of(float4 m, uint32_t dim) { return dim == 0 ? m.x : (dim == 1 ? m.y : m.z); }

__device__ __forceinline__ float split_of(int key, const float clo[3], const float chi[3], uint32_t &dim) {
    dim = 0;
    if (key == 0x7FFFFFFF) return 0.0f;
    dim = (uint32_t)(key / (NB - 1));
    const int pl = key % (NB - 1);
    const float lo_d = dim == 0 ? clo[0] : (dim == 1 ? clo[1] : clo[2]);
    const float hi_d = dim == 0 ? chi[0] : (dim == 1 ? chi[1] : chi[2]);
    return lo_d + ((float)pl + 1.0f) * ((hi_d - lo_d) / (float)NB);
}

// the two-sided partition of a slice by a warp; returns the true count
__device__ uint32_t warp_partition(const float4 *cen, uint32_t *perm, uint32_t c, uint32_t dim, float split, Bins &B) {
    const int lane = threadIdx.x & 31;
    uint32_t n_true = 0;
    for (uint32_t base = 0; base < c; base += 32) {
        const uint32_t i = base + lane;
        bool pr = false;
        if (i < c) pr = axis_of(cen[perm[i]], dim) < split;
        n_true += __popc(__ballot_sync(0xffffffffu, pr));
    }
    if (n_true == 0 || n_true == c) return c / 2;  // build.rs:151-157, current order kept
    // left region [0, n_true) ascending looking for false, right region
    // [n_true, c) descending looking for true
    uint32_t L = 0;
    int32_t R = (int32_t)c - 1;
    uint32_t lmask = 0, rmask = 0, lval = 0, rval = 0;
    bool lload = true, rload = true;
    while (true) {
        if (lload) {
            if (L >= n_true) break;
            const uint32_t i = L + lane;
            bool f = false;
            if (i < n_true) {
                lval = perm[i];
                f = !(axis_of(cen[lval], dim) < split);
            }
            lmask = __ballot_sync(0xffffffffu, f);
            lload = false;
        }
        if (rload) {
            if (R < (int32_t)n_true) break;  // unreachable: both regions hold the misplaced ones
            const int32_t i = R - lane;
            bool t = false;
            if (i >= (int32_t)n_true) {
                rval = perm[i];
                t = axis_of(cen[rval], dim) < split;
            }
            rmask = __ballot_sync(0xffffffffu, t);
            rload = false;
        }
        if (lmask == 0) { L += 32; lload = true; continue; }
        if (rmask == 0) { R -= 32; rload = true; continue; }
        const uint32_t k = min(__popc(lmask), __popc(rmask));
        // lanes holding the first k set bits of each mask pair by rank
        const uint32_t lrank = __popc(lmask & ((1u << lane) - 1u)), rrank = __popc(rmask & ((1u << lane) - 1u));
        const bool lact = ((lmask >> lane) & 1u) && lrank < k, ract = ((rmask >> lane) & 1u) && rrank < k;
        if (lact) B.swap[0][lrank] = lval;
        if (ract) B.swap[1][rrank] = rval;
        __syncwarp();
        if (lact) perm[L + lane] = B.swap[1][lrank];
        if (ract) perm[R - lane] = B.swap[0][rrank];
        __syncwarp();
        for (uint32_t j = 0; j < k; j++) { lmask &= lmask - 1u; rmask &= rmask - 1u; }  // drop the paired bits
    }
    return n_true;
}

// The split of a node of 3 to SMALL_NODE prims: a lane per prim, and a lane
// per (axis, prim) for the planes.  The planes between two occupied bins share
// a cost, so the first minimum is at a prim's own bin (bin 0 always holds the
// lowest centroid); each such plane takes the minima and maxima over the prims
// on its sides straight from their boxes, without the 96 bins.  Returns 0, with
// nothing changed, for a node with a value that is not finite (raw prims may
// hold one): its bounds and bins are those of the general path.
constexpr uint32_t SMALL_NODE = 10;  // three axes' prims in a warp
__device__ uint32_t warp_split_small(const Prims &Q, uint32_t *perm, uint32_t c, Bins &B, float nlo[3], float nhi[3]) {
    const uint32_t lane = threadIdx.x & 31;
    const bool own = lane < c;
    const uint32_t p = own ? perm[lane] : 0u;
    float4 a = make_float4(INFINITY, INFINITY, INFINITY, 0.0f), b = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f);
    float4 m = a;
    if (own) { a = Q.lo[p]; b = Q.hi[p]; m = Q.cen[p]; }
    const float lo[3] = {a.x, a.y, a.z}, hi[3] = {b.x, b.y, b.z}, cc[3] = {m.x, m.y, m.z};
    float zero = 0.0f;  // NaN once a value is not finite
#pragma unroll
    for (int k = 0; k < 3; k++) zero = __fmaf_rn(lo[k], 0.0f, __fmaf_rn(hi[k], 0.0f, __fmaf_rn(cc[k], 0.0f, zero)));
    if (__any_sync(0xffffffffu, own && zero != 0.0f)) return 0;
    float clo[3], chi[3];
    uint32_t bins = 0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        nlo[k] = o2f(__reduce_min_sync(0xffffffffu, f2o(lo[k])));
        nhi[k] = o2f(__reduce_max_sync(0xffffffffu, f2o(hi[k])));
        clo[k] = o2f(__reduce_min_sync(0xffffffffu, f2o(own ? cc[k] : FLT_MAX)));
        chi[k] = o2f(__reduce_max_sync(0xffffffffu, f2o(own ? cc[k] : -FLT_MAX)));
        bins |= bin_index((cc[k] - clo[k]) * ((float)NB / (chi[k] - clo[k]))) << (8 * k);
    }
    if (own) {
        B.plo[lane] = a;
        B.phi[lane] = b;
        B.pbin[lane] = bins;
    }
    __syncwarp();
    const uint32_t d = lane / SMALL_NODE, i = lane % SMALL_NODE;
    float cost = FLT_MAX;
    int key = 0x7FFFFFFF;
    if (d < 3 && i < c) {
        const uint32_t bi = (B.pbin[i] >> (8 * d)) & 255u;
        uint32_t nl = 0;
        float l0 = INFINITY, l1 = INFINITY, l2 = INFINITY, h0 = -INFINITY, h1 = -INFINITY, h2 = -INFINITY;
        float r0 = INFINITY, r1 = INFINITY, r2 = INFINITY, g0 = -INFINITY, g1 = -INFINITY, g2 = -INFINITY;
        for (uint32_t j = 0; j < c; j++) {
            const float4 x = B.plo[j], y = B.phi[j];
            if (((B.pbin[j] >> (8 * d)) & 255u) <= bi) {
                nl++;
                l0 = fminf(l0, x.x); l1 = fminf(l1, x.y); l2 = fminf(l2, x.z);
                h0 = fmaxf(h0, y.x); h1 = fmaxf(h1, y.y); h2 = fmaxf(h2, y.z);
            } else {
                r0 = fminf(r0, x.x); r1 = fminf(r1, x.y); r2 = fminf(r2, x.z);
                g0 = fmaxf(g0, y.x); g1 = fmaxf(g1, y.y); g2 = fmaxf(g2, y.z);
            }
        }
        const uint32_t nr = c - nl;
        const float al = area_of(l0, l1, l2, h0, h1, h2);
        const float ar = nr ? area_of(r0, r1, r2, g0, g1, g2) : 0.0f;
        const float v = al * (float)nl + ar * (float)nr;
        if (bi < NB - 1 && v < FLT_MAX) {  // (a NaN cost never compares less)
            cost = v;
            key = (int)(d * (NB - 1) + bi);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float oc = __shfl_xor_sync(0xffffffffu, cost, o);
        const int ok = __shfl_xor_sync(0xffffffffu, key, o);
        if (oc < cost || (oc == cost && ok < key)) { cost = oc; key = ok; }
    }
    uint32_t dim;
    const float split = split_of(key, clo, chi, dim);
    // the partition in one step: the k-th false of the left side and the k-th
    // true from the right trade places
    const bool t = own && axis_of(m, dim) < split;
    const uint32_t tm = __ballot_sync(0xffffffffu, t), n_true = __popc(tm);
    if (n_true == 0 || n_true == c) return c / 2;  // build.rs:151-157, current order kept
    const bool lf = own && lane < n_true && !t, rt = t && lane >= n_true;
    const uint32_t lm = __ballot_sync(0xffffffffu, lf), rm = __ballot_sync(0xffffffffu, rt);
    const uint32_t lrank = __popc(lm & ((1u << lane) - 1u)), rrank = __popc(rm & ~((2u << lane) - 1u));
    if (lf) B.swap[0][lrank] = p;
    if (rt) B.swap[1][rrank] = p;
    __syncwarp();
    if (lf) perm[lane] = B.swap[1][lrank];
    if (rt) perm[lane] = B.swap[0][rrank];
    __syncwarp();
    return n_true;
}

// The split of a node of c > 2 prims by a warp: its bounds (blas_leaf_bounds,
// build.rs:36-43) and the left child's count, the slice partitioned.  Bounds
// and bins are order-independent minima and maxima.
__device__ uint32_t warp_split(const Prims &Q, uint32_t *perm, uint32_t c, Bins &B, float nlo[3], float nhi[3]) {
    if (c <= SMALL_NODE) {
        const uint32_t n_left = warp_split_small(Q, perm, c, B, nlo, nhi);
        if (n_left) return n_left;
    }
    const int lane = threadIdx.x & 31;
    float clo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, chi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (int k = 0; k < 3; k++) { nlo[k] = INFINITY; nhi[k] = -INFINITY; }
    for (uint32_t i = lane; i < c; i += 32) {
        const uint32_t g = perm[i];
        const float4 a = Q.lo[g], b = Q.hi[g], m = Q.cen[g];
        nlo[0] = fminf(nlo[0], a.x); nlo[1] = fminf(nlo[1], a.y); nlo[2] = fminf(nlo[2], a.z);
        nhi[0] = fmaxf(nhi[0], b.x); nhi[1] = fmaxf(nhi[1], b.y); nhi[2] = fmaxf(nhi[2], b.z);
        clo[0] = fminf(clo[0], m.x); clo[1] = fminf(clo[1], m.y); clo[2] = fminf(clo[2], m.z);
        chi[0] = fmaxf(chi[0], m.x); chi[1] = fmaxf(chi[1], m.y); chi[2] = fmaxf(chi[2], m.z);
    }
    bins_clear(B, lane, 32);
    float scale[3];
    for (int k = 0; k < 3; k++) {
        nlo[k] = o2f(__reduce_min_sync(0xffffffffu, f2o(nlo[k])));
        nhi[k] = o2f(__reduce_max_sync(0xffffffffu, f2o(nhi[k])));
        clo[k] = o2f(__reduce_min_sync(0xffffffffu, f2o(clo[k])));
        chi[k] = o2f(__reduce_max_sync(0xffffffffu, f2o(chi[k])));
        scale[k] = (float)NB / (chi[k] - clo[k]);
    }
    __syncwarp();
    for (uint32_t i = lane; i < c; i += 32) {
        const uint32_t g = perm[i];
        bins_add(B, clo, scale, Q.lo[g], Q.hi[g], Q.cen[g]);
    }
    __syncwarp();
    float best = FLT_MAX;
    int key = 0x7FFFFFFF;
    for (int d = 0; d < 3; d++) {  // first minimum in (axis, plane) order
        float cost;
        int k;
        best_plane(B, d, cost, k);
        if (cost < best) { best = cost; key = k; }
    }
    uint32_t dim;
    const float split = split_of(key, clo, chi, dim);
    const uint32_t n_left = warp_partition(Q.cen, perm, c, dim, split, B);
    __syncwarp();
    return n_left;
}

__global__ void k_perm_init(const SahTree *trees, uint32_t *perm) {
    SahTree T = trees[blockIdx.y];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < T.n; i += gridDim.x * blockDim.x)
        perm[T.prim_off + i] = i;
}

// One level of the trees larger than TREE_MAX, a warp per node.
__global__ void __launch_bounds__(SAH_WARPS * 32) k_sah_level(const SahTree *trees, SahInputs in, SahOutputs out,
                                                              const Item *items, const uint32_t *n_items_p,
                                                              Item *next, uint32_t *n_next) {
    __shared__ Bins s_bins[SAH_WARPS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t n_items = *n_items_p;
    for (uint32_t it = blockIdx.x * SAH_WARPS + w; it < n_items; it += gridDim.x * SAH_WARPS) {
        const Item I = items[it];
        const SahTree T = trees[I.tree];
        const Prims Q{in.lo + T.prim_off, in.hi + T.prim_off, in.cen + T.prim_off, in.id + T.prim_off,
                      out.perm + T.prim_off};
        const uint32_t c = I.count;
        if (c == 1) {
            if (lane == 0) write_leaf(out, T, Q, I.node, I.parent, Q.perm[I.first]);
            continue;
        }
        if (c == 2) {
            if (lane == 0) write_pair(out, T, Q, I.node, I.parent, I.base, I.first);
            continue;
        }
        float nlo[3], nhi[3];
        const uint32_t n_left = warp_split(Q, Q.perm + I.first, c, s_bins[w], nlo, nhi);
        if (lane == 2) write_internal(out, T, I.node, I.parent, I.base, nlo, nhi);
        if (lane < 2) {  // a lane per child
            const uint32_t s = lane, node = I.base + s;
            const uint32_t cn = s ? c - n_left : n_left, base = s ? I.base + 2 * n_left : I.base + 2;
            const uint32_t first = s ? I.first + n_left : I.first;
            if (cn == 1) write_leaf(out, T, Q, node, I.node, Q.perm[first]);
            else if (cn == 2) write_pair(out, T, Q, node, I.node, base, first);
            else next[atomicAdd(n_next, 1u)] = Item{I.tree, node, base, first, cn, I.node};
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// k_sah_tree: one CTA builds one tree of up to TREE_MAX prims, all levels in
// one launch, its prims, order and level lists in shared memory.
//
// A launch per level with the host waiting for the next level's count spent a
// chunk's build on round trips, on the top nodes that one warp each binned
// alone, and on the latency of the prims' loads through the order.  Here the
// CTA keeps two lists per level: nodes of more than TREE_BIG prims are split
// by all its threads, one after the other, the others by a warp each, and
// levels are separated by a barrier.  The steps and their results are those of
// k_sah_level; the CTA's partition pairs the k-th misplaced prim of the left
// side with the k-th from the right through two position lists.  Whole calls of
// vrg_build_tl_bvh_batched: 30 prims 580 -> 130 us, 300 704 -> 187, 1200 877 ->
// 351; past TREE_MAX, where only the node's work is cheaper (warp_split), 5000
// prims 1462 -> 1002 us, 65536 10.5 -> 8.2 ms.  (A CTA on trees past its shared
// memory, its prims in global memory: 16000 prims 5665 us, so those stay level
// by level over all SMs.)
// ---------------------------------------------------------------------------
struct ItemS {  // an Item of a tree of at most TREE_MAX prims
    uint16_t node, base, first, count, parent, pad;
};
constexpr uint16_t NO_PARENT = 0xFFFF;
static_assert(2 * TREE_MAX < NO_PARENT, "node indices in 16 bits");

// shared memory of a tree of n prims: the static part is the bins
__host__ __device__ constexpr uint32_t tree_small_cap(uint32_t n) { return n / 3 + 1; }
__host__ __device__ constexpr uint32_t tree_big_cap(uint32_t n) { return n / TREE_BIG + 1; }
__host__ __device__ constexpr size_t tree_smem(uint32_t n) {
    return (size_t)n * (3 * 16 + 3 * 4) + 2 * (size_t)(tree_small_cap(n) + tree_big_cap(n)) * sizeof(ItemS);
}

// exclusive scan of a flag over the CTA; total in every thread
__device__ __forceinline__ uint32_t cta_rank(bool f, uint32_t *sh, uint32_t &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t m = __ballot_sync(0xffffffffu, f);
    if (lane == 0) sh[w] = __popc(m);
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int k = 0; k < TREE_WARPS; k++) {
        const uint32_t n = sh[k];
        if (k < w) before += n;
        all += n;
    }
    __syncthreads();
    total = all;
    return before + __popc(m & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(TREE_THREADS) k_sah_tree(const SahTree *trees, SahInputs in, SahOutputs out,
                                                           uint32_t *arrive, uint32_t *levels) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ Bins s_bins[TREE_WARPS];
    __shared__ int s_box[12];            // a big node's bounds: node lo, hi, centroid lo, hi (ordered integers)
    __shared__ uint32_t s_scan[TREE_WARPS], s_n[2][2], s_best_key[3];
    __shared__ float s_best_cost[3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, tid = (int)threadIdx.x;
    const SahTree T = trees[blockIdx.x];
    const uint32_t n = T.n;
    if (n == 0) return;
    float4 *lo = reinterpret_cast<float4 *>(s_dyn), *hi = lo + n, *cen = hi + n;
    uint32_t *perm0 = reinterpret_cast<uint32_t *>(cen + n), *pos0 = perm0 + n, *ids = pos0 + n;
    ItemS *lists = reinterpret_cast<ItemS *>(ids + n);
    ItemS *small[2] = {lists, lists + tree_small_cap(n)};
    ItemS *big[2] = {small[1] + tree_small_cap(n), small[1] + tree_small_cap(n) + tree_big_cap(n)};
    const Prims Q{lo, hi, cen, ids, perm0};
    for (uint32_t i = tid; i < n; i += TREE_THREADS) {
        lo[i] = in.lo[T.prim_off + i];
        hi[i] = in.hi[T.prim_off + i];
        cen[i] = in.cen[T.prim_off + i];
        ids[i] = in.id[T.prim_off + i];
        perm0[i] = i;
    }
    if (T.flags & SAH_POWER)
        for (uint32_t i = tid; i < 2 * n - 1; i += TREE_THREADS) arrive[T.node_off + i] = 0;
    __syncthreads();
    if (tid == 0) {
        s_n[0][0] = s_n[0][1] = s_n[1][0] = s_n[1][1] = 0;
        const ItemS root{0, 1, 0, (uint16_t)n, NO_PARENT, 0};
        if (n == 1) write_leaf(out, T, Q, 0, INVALID, 0);
        else if (n == 2) write_pair(out, T, Q, 0, INVALID, 1, 0);
        else if (n > TREE_BIG) { big[0][0] = root; s_n[0][1] = 1; }
        else { small[0][0] = root; s_n[0][0] = 1; }
    }
    __syncthreads();
    // a warp's first three lanes: each child (a leaf, two leaves, or onto the
    // next level's lists) and the node
    auto emit = [&](const ItemS &I, uint32_t n_left, const float nlo[3], const float nhi[3], uint32_t nxt) {
        if (lane == 2) write_internal(out, T, I.node, I.parent == NO_PARENT ? INVALID : I.parent, I.base, nlo, nhi);
        if (lane >= 2) return;
        const uint32_t node = I.base + (uint32_t)lane, cn = lane ? I.count - n_left : n_left;
        const uint32_t base = lane ? I.base + 2 * n_left : I.base + 2u, first = lane ? I.first + n_left : I.first;
        const ItemS c{(uint16_t)node, (uint16_t)base, (uint16_t)first, (uint16_t)cn, I.node, 0};
        if (cn == 1) write_leaf(out, T, Q, node, I.node, perm0[first]);
        else if (cn == 2) write_pair(out, T, Q, node, I.node, base, first);
        else if (cn > TREE_BIG) big[nxt][atomicAdd(&s_n[nxt][1], 1u)] = c;
        else small[nxt][atomicAdd(&s_n[nxt][0], 1u)] = c;
    };
    uint32_t lv = 0, cur = 0;
    while (true) {
        const uint32_t n_small = s_n[cur][0], n_big = s_n[cur][1], nxt = cur ^ 1u;
        lv++;
        if (n_small + n_big == 0 || lv > TREE_MAX) break;  // (a level is shorter than the one above it)
        for (uint32_t it = 0; it < n_big; it++) {
            const ItemS I = big[cur][it];
            const uint32_t c = I.count;
            uint32_t *perm = perm0 + I.first, *pos = pos0 + I.first;
            if (tid < 12)
                s_box[tid] = f2o((tid % 6) < 3 ? (tid < 6 ? INFINITY : FLT_MAX) : (tid < 6 ? -INFINITY : -FLT_MAX));
            bins_clear(s_bins[0], tid, TREE_THREADS);
            __syncthreads();
            {
                float v[12];
                for (int k = 0; k < 3; k++) {
                    v[k] = INFINITY; v[3 + k] = -INFINITY; v[6 + k] = FLT_MAX; v[9 + k] = -FLT_MAX;
                }
                for (uint32_t i = tid; i < c; i += TREE_THREADS) {
                    const uint32_t g = perm[i];
                    const float4 a = lo[g], b = hi[g], m = cen[g];
                    v[0] = fminf(v[0], a.x); v[1] = fminf(v[1], a.y); v[2] = fminf(v[2], a.z);
                    v[3] = fmaxf(v[3], b.x); v[4] = fmaxf(v[4], b.y); v[5] = fmaxf(v[5], b.z);
                    v[6] = fminf(v[6], m.x); v[7] = fminf(v[7], m.y); v[8] = fminf(v[8], m.z);
                    v[9] = fmaxf(v[9], m.x); v[10] = fmaxf(v[10], m.y); v[11] = fmaxf(v[11], m.z);
                }
#pragma unroll
                for (int k = 0; k < 12; k++) {
                    const int o = (k % 6) < 3 ? __reduce_min_sync(0xffffffffu, f2o(v[k]))
                                              : __reduce_max_sync(0xffffffffu, f2o(v[k]));
                    if (lane == 0) {
                        if ((k % 6) < 3) atomicMin(&s_box[k], o);
                        else atomicMax(&s_box[k], o);
                    }
                }
            }
            __syncthreads();
            float nlo[3], nhi[3], clo[3], chi[3], scale[3];
            for (int k = 0; k < 3; k++) {
                nlo[k] = o2f(s_box[k]); nhi[k] = o2f(s_box[3 + k]);
                clo[k] = o2f(s_box[6 + k]); chi[k] = o2f(s_box[9 + k]);
                scale[k] = (float)NB / (chi[k] - clo[k]);
            }
            for (uint32_t i = tid; i < c; i += TREE_THREADS) {
                const uint32_t g = perm[i];
                bins_add(s_bins[0], clo, scale, lo[g], hi[g], cen[g]);
            }
            __syncthreads();
            if (w < 3) {
                float cost;
                int key;
                best_plane(s_bins[0], w, cost, key);
                if (lane == 0) {
                    s_best_cost[w] = cost;
                    s_best_key[w] = (uint32_t)key;
                }
            }
            __syncthreads();
            float best = FLT_MAX;
            int key = 0x7FFFFFFF;
            for (int d = 0; d < 3; d++)
                if (s_best_cost[d] < best) { best = s_best_cost[d]; key = (int)s_best_key[d]; }
            uint32_t dim;
            const float split = split_of(key, clo, chi, dim);
            uint32_t n_true = 0;
            for (uint32_t base = 0; base < c; base += TREE_THREADS) {
                const uint32_t i = base + tid;
                uint32_t all;
                cta_rank(i < c && axis_of(cen[perm[min(i, c - 1)]], dim) < split, s_scan, all);
                n_true += all;
            }
            uint32_t n_left = c / 2;  // build.rs:151-157, current order kept
            if (n_true != 0 && n_true != c) {
                n_left = n_true;
                // the misplaced prims' positions: falses of the left side
                // ascending, trues of the right side descending; the k-th of
                // each swap (each list holds at most c / 2)
                uint32_t nf = 0, nt = 0;
                for (uint32_t base = 0; base < n_true; base += TREE_THREADS) {
                    const uint32_t i = base + tid;
                    const bool f = i < n_true && !(axis_of(cen[perm[min(i, c - 1)]], dim) < split);
                    uint32_t all;
                    const uint32_t k = cta_rank(f, s_scan, all);
                    if (f) pos[nf + k] = i;
                    nf += all;
                }
                for (uint32_t base = 0; base < c - n_true; base += TREE_THREADS) {
                    const uint32_t j = base + tid, i = c - 1 - min(j, c - 1);
                    const bool t = j < c - n_true && axis_of(cen[perm[i]], dim) < split;
                    uint32_t all;
                    const uint32_t k = cta_rank(t, s_scan, all);
                    if (t) pos[c / 2 + nt + k] = i;
                    nt += all;
                }
                __syncthreads();
                for (uint32_t k = tid; k < nf; k += TREE_THREADS) {
                    const uint32_t a = pos[k], b = pos[c / 2 + k], va = perm[a], vb = perm[b];
                    perm[a] = vb;
                    perm[b] = va;
                }
            }
            __syncthreads();
            if (w == 0) emit(I, n_left, nlo, nhi, nxt);
        }
        for (uint32_t it = w; it < n_small; it += TREE_WARPS) {
            const ItemS I = small[cur][it];
            float nlo[3], nhi[3];
            const uint32_t n_left = warp_split(Q, perm0 + I.first, I.count, s_bins[w], nlo, nhi);
            emit(I, n_left, nlo, nhi, nxt);
            __syncwarp();
        }
        __syncthreads();
        if (tid == 0) s_n[cur][0] = s_n[cur][1] = 0;
        cur = nxt;
        __syncthreads();
    }
    for (uint32_t i = tid; i < n; i += TREE_THREADS) out.perm[T.prim_off + i] = perm0[i];
    if (tid == 0 && levels) atomicMax(levels, max(lv - 1, 1u));
    // powers bottom-up (build.rs:341-357): (0 + left) + right
    if (T.flags & SAH_POWER) {
        vrg_bvh_node *base = out.nodes + T.node_off;
        for (uint32_t i = tid; i < 2 * n - 1; i += TREE_THREADS) {
            if (base[i].left_node_idx != INVALID) continue;
            uint32_t at = i;
            for (uint32_t guard = 0; guard < 2 * n; guard++) {
                const uint32_t parent = base[at].parent_idx;
                if (parent == INVALID) break;
                __threadfence_block();
                if (atomicAdd(&arrive[T.node_off + parent], 1u) == 0) break;  // sibling not done yet
                __threadfence_block();
                volatile vrg_bvh_node *vb = base;
                const float lp = vb[vb[parent].left_node_idx].power;
                const float rp = vb[vb[parent].right_node_idx_or_prim_idx].power;
                float p = 0.0f;
                p += lp;
                p += rp;
                vb[parent].power = p;
                at = parent;
            }
        }
    }
}

// power of an internal node = (0 + left) + right, bottom-up (build.rs:341-357)
__global__ void k_power_up(const SahTree *trees, vrg_bvh_node *nodes, uint32_t *arrive) {
    SahTree T = trees[blockIdx.y];
    if (T.n == 0) return;
    uint32_t n_nodes = 2 * T.n - 1;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_nodes; i += gridDim.x * blockDim.x) {
        vrg_bvh_node *base = nodes + T.node_off;
        if (base[i].left_node_idx != INVALID) continue;
        uint32_t cur = i;
        for (uint32_t guard = 0; guard < n_nodes; guard++) {
            uint32_t parent = base[cur].parent_idx;
            if (parent == INVALID) break;
            __threadfence();
            if (atomicAdd(&arrive[T.node_off + parent], 1u) == 0) break;  // sibling not done yet
            __threadfence();
            volatile vrg_bvh_node *vb = base;
            float lp = vb[vb[parent].left_node_idx].power;
            float rp = vb[vb[parent].right_node_idx_or_prim_idx].power;
            float p = 0.0f;
            p += lp;
            p += rp;
            vb[parent].power = p;
            cur = parent;
        }
    }
}

}  // namespace

// Shared memory of k_sah_tree beyond the default 48 KB.  The attribute belongs
// to the context current at the call, so it is asked for before every build: a
// process may build on several devices, reset one, or build under contexts of
// its own (vrg_build_tl_bvh_noalloc).
static vrg_status tree_smem_init() {
    VRG_CUDA_TRY(cudaFuncSetAttribute(k_sah_tree, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)tree_smem(TREE_MAX)));
    return VRG_OK;
}

vrg_status sah_build(Context *ctx, std::vector<SahTree> &trees, uint32_t total_prims, uint32_t total_nodes,
                     const SahInputs &in, const SahOutputs &out, uint32_t *levels, uint32_t *levels_dev) {
    cudaStream_t s = ctx->stream;
    if (trees.empty() || total_prims == 0) {
        if (levels) *levels = 0;
        return VRG_OK;
    }
    const uint32_t nt = (uint32_t)trees.size();
    if (nt > 65535) {
        set_error("sah_build: %u trees exceeds one launch (65535)", nt);
        return VRG_ERR_UNSUPPORTED;
    }
    VRG_TRY(tree_smem_init());
    // largest first: the trees past TREE_MAX go level by level, the others by
    // a CTA each.  A CTA's shared memory is its launch's largest tree's, so
    // more trees than SMs go in launches by size; up to one per SM they go in
    // one, since launches of a few CTAs each would only follow one another.
    std::stable_sort(trees.begin(), trees.end(), [](const SahTree &a, const SahTree &b) { return a.n > b.n; });
    uint32_t n_large = 0;
    while (n_large < nt && trees[n_large].n > TREE_MAX) n_large++;
    // scratch: trees, counters, arrival flags; the level lists of large trees
    const size_t q_cap = n_large ? std::max<size_t>(n_large, (size_t)total_prims / 3 + 1) : 0;
    const size_t bytes = nt * sizeof(SahTree) + 2 * q_cap * sizeof(Item) + 64 + (size_t)total_nodes * 4;
    DevBufPtr scratch;
    VRG_TRY(dev_alloc(ctx, bytes, scratch));
    uint8_t *p = (uint8_t *)scratch->ptr;
    SahTree *d_trees = (SahTree *)p; p += nt * sizeof(SahTree);
    Item *q0 = (Item *)p; p += q_cap * sizeof(Item);
    Item *q1 = (Item *)p; p += q_cap * sizeof(Item);
    uint32_t *cnt = (uint32_t *)p; p += 64;
    uint32_t *arrive = (uint32_t *)p;
    VRG_CUDA_TRY(cudaMemcpyAsync(d_trees, trees.data(), nt * sizeof(SahTree), cudaMemcpyHostToDevice, s));
    if (!levels_dev) VRG_CUDA_TRY(cudaMemsetAsync(cnt, 0, 64, s));
    uint32_t *lv_dev = levels_dev ? levels_dev : cnt + 8;
    for (uint32_t a = n_large; a < nt && trees[a].n;) {
        uint32_t b = a;
        const uint32_t n = trees[a].n;
        while (b < nt && trees[b].n && (nt - n_large <= (uint32_t)ctx->num_sms || 2 * trees[b].n > n)) b++;
        k_sah_tree<<<b - a, TREE_THREADS, tree_smem(n), s>>>(d_trees + a, in, out, arrive, lv_dev);
        VRG_CUDA_TRY(cudaGetLastError());
        a = b;
    }
    uint32_t lv = 0, h_cnt = 0;
    if (n_large) {
        const uint32_t max_n = trees[0].n;
        std::vector<Item> roots;
        for (uint32_t t = 0; t < n_large; t++) roots.push_back(Item{t, 0, 1, 0, trees[t].n, INVALID});
        uint32_t n_cur = n_large;
        // (the flags of the CTAs' trees are theirs: all before them is zeroed here)
        for (uint32_t t = 0; t < n_large; t++)
            VRG_CUDA_TRY(cudaMemsetAsync(arrive + trees[t].node_off, 0, (2 * (size_t)trees[t].n - 1) * 4, s));
        VRG_CUDA_TRY(cudaMemcpyAsync(q0, roots.data(), roots.size() * sizeof(Item), cudaMemcpyHostToDevice, s));
        VRG_CUDA_TRY(cudaMemcpyAsync(cnt, &n_cur, 4, cudaMemcpyHostToDevice, s));
        k_perm_init<<<dim3(std::min(1024u, (max_n + 255) / 256), n_large), 256, 0, s>>>(d_trees, out.perm);
        VRG_CUDA_TRY(cudaGetLastError());
        Item *cur = q0, *nxt = q1;
        uint32_t cur_slot = 0;
        while (n_cur > 0) {
            uint32_t next_slot = cur_slot ^ 1u;
            VRG_CUDA_TRY(cudaMemsetAsync(cnt + next_slot, 0, 4, s));
            uint32_t blocks = std::min<uint32_t>((n_cur + SAH_WARPS - 1) / SAH_WARPS, 152u * 16u);
            k_sah_level<<<blocks, SAH_WARPS * 32, 0, s>>>(d_trees, in, out, cur, cnt + cur_slot, nxt, cnt + next_slot);
            VRG_CUDA_TRY(cudaGetLastError());
            VRG_CUDA_TRY(cudaMemcpyAsync(&h_cnt, cnt + next_slot, 4, cudaMemcpyDeviceToHost, s));
            VRG_CUDA_TRY(cudaStreamSynchronize(s));
            n_cur = h_cnt;
            std::swap(cur, nxt);
            cur_slot = next_slot;
            lv++;
            if (lv > 100000) {
                set_error("sah_build: level loop did not terminate");
                return VRG_ERR_STATE;
            }
        }
        const uint32_t max_nodes = 2 * max_n - 1;
        k_power_up<<<dim3(std::min(1024u, (max_nodes + 255) / 256), n_large), 256, 0, s>>>(d_trees, out.nodes, arrive);
        VRG_CUDA_TRY(cudaGetLastError());
    }
    if (levels && levels_dev) {
        *levels = lv;
    } else if (levels) {
        VRG_CUDA_TRY(cudaMemcpyAsync(&h_cnt, cnt + 8, 4, cudaMemcpyDeviceToHost, s));
        VRG_CUDA_TRY(cudaStreamSynchronize(s));
        *levels = std::max(lv, h_cnt);
    }
    return VRG_OK;
}

}  // namespace vrg

namespace vrg {

// ---------------------------------------------------------------------------
// Build without allocating: vrg_build_tl_bvh_noalloc
//
// For callers that must not allocate device memory while they run: a game or
// engine that owns the whole device-memory budget and hands this library
// only the buffers it has set aside, or a chunk-streaming worker that builds
// BVHs next to a frame in flight, where cudaMalloc/cudaFree may synchronize
// the device and stall the frame.  The builder's scratch (work queues,
// level counters, bottom-up arrival flags, prepared prim bounds) lives in
// the fixed device array below instead of a cudaMallocAsync allocation.
// ---------------------------------------------------------------------------

namespace {

constexpr uint32_t NOALLOC_MAX_PRIMS = 32768;  // one chunk's worth of blocks
constexpr size_t NOALLOC_QCAP = NOALLOC_MAX_PRIMS / 3 + 2;
constexpr size_t NOALLOC_OFF_LO = 0;
constexpr size_t NOALLOC_OFF_HI = NOALLOC_OFF_LO + (size_t)NOALLOC_MAX_PRIMS * 16;
constexpr size_t NOALLOC_OFF_CEN = NOALLOC_OFF_HI + (size_t)NOALLOC_MAX_PRIMS * 16;
constexpr size_t NOALLOC_OFF_Q0 = NOALLOC_OFF_CEN + (size_t)NOALLOC_MAX_PRIMS * 16;
constexpr size_t NOALLOC_OFF_Q1 = NOALLOC_OFF_Q0 + NOALLOC_QCAP * sizeof(Item);
constexpr size_t NOALLOC_OFF_CNT = (NOALLOC_OFF_Q1 + NOALLOC_QCAP * sizeof(Item) + 255) & ~(size_t)255;
constexpr size_t NOALLOC_OFF_TREE = NOALLOC_OFF_CNT + 256;
constexpr size_t NOALLOC_OFF_ARRIVE = NOALLOC_OFF_TREE + 256;
constexpr size_t NOALLOC_OFF_LEAF = NOALLOC_OFF_ARRIVE + (size_t)2 * NOALLOC_MAX_PRIMS * 4;
constexpr size_t NOALLOC_BYTES = NOALLOC_OFF_LEAF + (size_t)2 * NOALLOC_MAX_PRIMS * 4;  // about 2.4 MiB

// inputs of build_tl_bvh with identity isometries: AABB as given, centroid
// (min+max)/2 (build.rs:391-400), w = power
__global__ void k_noalloc_prep(const float *aabbs, const float *power, uint32_t n, float4 *lo, float4 *hi,
                               float4 *cen) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *a = aabbs + 6 * (size_t)i;
    float l[3], h[3];
    for (int k = 0; k < 3; k++) {
        float x0 = a[k] + 0.0f, x1 = a[3 + k] + 0.0f;  // translation by zero, as k_tl_inputs
        l[k] = fminf(x0, x1);
        h[k] = fmaxf(x0, x1);
    }
    lo[i] = make_float4(l[0], l[1], l[2], 0.0f);
    hi[i] = make_float4(h[0], h[1], h[2], 0.0f);
    cen[i] = make_float4((l[0] + h[0]) / 2.0f, (l[1] + h[1]) / 2.0f, (l[2] + h[2]) / 2.0f, power[i]);
}

}  // namespace
}  // namespace vrg

// The scratch array every call of vrg_build_tl_bvh_noalloc shares.  Each GPU
// that loads the library holds it until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[vrg::NOALLOC_BYTES];

extern "C" VRG_API vrg_status vrg_build_tl_bvh_noalloc(const float *aabbs, const float *power, const uint32_t *ids,
                                                       uint32_t n, vrg_bvh_node *nodes, uint32_t *prim_order,
                                                       void *stream) {
    using namespace vrg;
    if (!aabbs || !power || !ids || !nodes || !prim_order || n == 0) {
        set_error("vrg_build_tl_bvh_noalloc: null pointer or n == 0");
        return VRG_ERR_INVALID_ARGUMENT;
    }
    if (n > NOALLOC_MAX_PRIMS) {
        set_error("vrg_build_tl_bvh_noalloc: %u prims exceed the fixed scratch capacity of %u prims", n,
                  NOALLOC_MAX_PRIMS);
        return VRG_ERR_INVALID_ARGUMENT;
    }
    cudaStream_t s = (cudaStream_t)stream;
    // The device address of the array in the context current now (its name in
    // host code is only a host-side stand-in).  Looked up on every call, so a
    // device reset or another current context never leaves a stale address;
    // the lookup allocates nothing.
    void *base = nullptr;
    {
        cudaError_t e = cudaGetSymbolAddress(&base, g_noalloc_scratch);
        if (e != cudaSuccess || !base) {
            set_error("cudaGetSymbolAddress(g_noalloc_scratch) failed: %s", cudaGetErrorString(e));
            return VRG_ERR_CUDA;
        }
    }
    // Everything from the first enqueue on: on an error return the stream is
    // synchronized first, so no work that uses the shared array is still
    // queued when the call returns.
    auto build = [&]() -> vrg_status {
        uint8_t *B = (uint8_t *)base;
        float4 *lo = (float4 *)(B + NOALLOC_OFF_LO), *hi = (float4 *)(B + NOALLOC_OFF_HI),
               *cen = (float4 *)(B + NOALLOC_OFF_CEN);
        Item *q0 = (Item *)(B + NOALLOC_OFF_Q0), *q1 = (Item *)(B + NOALLOC_OFF_Q1);
        uint32_t *cnt = (uint32_t *)(B + NOALLOC_OFF_CNT);
        SahTree *d_tree = (SahTree *)(B + NOALLOC_OFF_TREE);
        uint32_t *arrive = (uint32_t *)(B + NOALLOC_OFF_ARRIVE);
        uint32_t *leaf = (uint32_t *)(B + NOALLOC_OFF_LEAF);
        const uint32_t n_nodes = 2 * n - 1;
        // tree descriptor and root work item: copies of host stack values
        SahTree tree{n, 0, 0, SAH_POWER};
        Item root{0, 0, 1, 0, n, INVALID};
        uint32_t one = 1;
        VRG_CUDA_TRY(cudaMemcpyAsync(d_tree, &tree, sizeof(tree), cudaMemcpyHostToDevice, s));
        k_noalloc_prep<<<(n + 255) / 256, 256, 0, s>>>(aabbs, power, n, lo, hi, cen);
        VRG_CUDA_TRY(cudaGetLastError());
        SahInputs in{lo, hi, cen, ids};
        SahOutputs out{nodes, prim_order, leaf};
        if (n <= TREE_MAX) {
            VRG_TRY(tree_smem_init());
            k_sah_tree<<<1, TREE_THREADS, tree_smem(n), s>>>(d_tree, in, out, arrive, nullptr);
            VRG_CUDA_TRY(cudaGetLastError());
            VRG_CUDA_TRY(cudaStreamSynchronize(s));
            return VRG_OK;
        }
        // the array keeps the previous call's contents: reset what must start at
        // zero (k_sah_tree resets its own)
        VRG_CUDA_TRY(cudaMemsetAsync(arrive, 0, (size_t)n_nodes * 4, s));
        VRG_CUDA_TRY(cudaMemsetAsync(cnt, 0, 256, s));
        VRG_CUDA_TRY(cudaMemcpyAsync(q0, &root, sizeof(root), cudaMemcpyHostToDevice, s));
        VRG_CUDA_TRY(cudaMemcpyAsync(cnt, &one, 4, cudaMemcpyHostToDevice, s));
        k_perm_init<<<dim3(std::max(1u, (n + 255) / 256), 1), 256, 0, s>>>(d_tree, prim_order);
        VRG_CUDA_TRY(cudaGetLastError());
        uint32_t n_cur = 1, cur_slot = 0, lv = 0;
        Item *cur = q0, *nxt = q1;
        while (n_cur > 0) {
            uint32_t next_slot = cur_slot ^ 1u;
            VRG_CUDA_TRY(cudaMemsetAsync(cnt + next_slot, 0, 4, s));
            uint32_t blocks = std::min<uint32_t>((n_cur + SAH_WARPS - 1) / SAH_WARPS, 152u * 16u);
            k_sah_level<<<blocks, SAH_WARPS * 32, 0, s>>>(d_tree, in, out, cur, cnt + cur_slot, nxt, cnt + next_slot);
            VRG_CUDA_TRY(cudaGetLastError());
            uint32_t h_next = 0;
            VRG_CUDA_TRY(cudaMemcpyAsync(&h_next, cnt + next_slot, 4, cudaMemcpyDeviceToHost, s));
            VRG_CUDA_TRY(cudaStreamSynchronize(s));
            n_cur = h_next;
            std::swap(cur, nxt);
            cur_slot = next_slot;
            if (++lv > 4 * NOALLOC_MAX_PRIMS) {
                set_error("vrg_build_tl_bvh_noalloc: level loop did not terminate");
                return VRG_ERR_STATE;
            }
        }
        k_power_up<<<dim3(std::max(1u, (n_nodes + 255) / 256), 1), 256, 0, s>>>(d_tree, nodes, arrive);
        VRG_CUDA_TRY(cudaGetLastError());
        VRG_CUDA_TRY(cudaStreamSynchronize(s));
        return VRG_OK;
    };
    const vrg_status st = build();
    if (st != VRG_OK) (void)cudaStreamSynchronize(s);
    return st;
}
