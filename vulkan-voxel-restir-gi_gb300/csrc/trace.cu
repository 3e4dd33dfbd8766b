// Wavefront bounce kernels: per bounce, the closest hit over the world-space
// voxel BVH (k_trace, with ray generation at bounce 0), the shading with its
// light-BVH next-event estimation (k_shade), and the light-sampling pdf of the
// chosen direction in three passes (k_anyhit, k_hit_eval, k_hit_sum), which
// run on their own stream beside the next bounce.
//
// Reference stages covered here (one dispatch each in the reference):
//   raygen        raygen.rs:84-111
//   raytrace      raytrace.rs:390-578 (closest hit replaces the driver ray
//                 query; traverseBvh 218-281 is the light descent)
//   nee_pdf       nee_pdf.rs:281-337 (any-hit over light triangles along the
//                 chosen direction; reverseTraverseBvh 154-228)
// Work distribution: the closest hit and the any-hit walk are persistent
// warps in which each lane takes a new ray from the bounce's queue when its
// walk ends; rays that continue, and light-pdf jobs, are compacted into the
// next queues with one warp ballot + one atomic per warp.  A path's ray and its
// per-bounce record (E, w=pdf/q) (R, q), which feeds the backward radiance
// recurrence of the resolve kernel, are 32-byte entries.
#include <cstring>
#include <mutex>

#include "vrg_frame.cuh"
#include "vrg_internal.h"

namespace vrg {

// Per (face, half), FACE_ROW float4: (normal, corner bits of the triangle's
// vertices: 3 x 3 bits), unused, tangent, bitangent.  In global memory, not constant memory: the lanes
// of a warp shade different faces, and constant loads serialize over them.
__device__ __align__(32) float4 d_faces[12 * FACE_ROW];

namespace {

// The shading point's part of nodeImportance, the same for every node of a
// walk, worked out once per walk.  Voxel-face normals are one of +-x, +-y,
// +-z: then dot(c - p, n) is exactly +-(c_a - p_a) (the other two products are
// +-0), so the 8 corners reduce to the box's min and max along the normal
// axis, 4 corners each.
struct ImpPt {
    f3 point, normal;
    int ax;         // the normal's axis when it is +-1 on one axis and 0 on the others, else -1
    float sg, sp;   // its sign there; -sg * point[ax]
};
__device__ __forceinline__ ImpPt imp_point(f3 point, f3 normal) {
    ImpPt P;
    P.point = point;
    P.normal = normal;
    P.ax = -1;
    P.sg = P.sp = 0.0f;
    const bool nx = normal.x != 0.0f, ny = normal.y != 0.0f, nz = normal.z != 0.0f;
    if ((int)nx + (int)ny + (int)nz == 1) {
        const int ax = nx ? 0 : (ny ? 1 : 2);
        const float na = cmp3(normal, ax);
        if (na == 1.0f || na == -1.0f) {
            P.ax = ax;
            P.sg = na;
            P.sp = -na * cmp3(point, ax);
        }
    }
    return P;
}

// nodeImportance (raytrace.rs:181-208: uint visibility, EPS 1e-3;
// nee_pdf.rs:125-152: float visibility, EPS 1e-4) of both children of light
// node g: power / max(|e|^2, |c|^2) * the visible share of the 8 corners of
// the axis-aligned box that v000 and v111 span (as in the reference, not the
// transformed box), c the vector from the point to the box's centre.
// Packed operations (two per instruction) are fused multiply-adds only, where
// one rounding is what the shader does: the centre's 0.5 * (v000 + v111) is
// exact, and v * sign - sign * p rounds as v - p.  (The assembler contracts a
// packed product followed by a packed sum, with .rn and without -fmad, so the
// exact |c|^2 stays scalar.)
struct LightPair {
    float2 power, ee, cx, cy, cz, vis;  // of (left, right)
    int left, right;                    // refs
    __device__ __forceinline__ float imp_l() const {
        return power.x / fmaxf(ee.x, (cx.x * cx.x + cy.x * cy.x) + cz.x * cz.x) * vis.x;
    }
    __device__ __forceinline__ float imp_r() const {
        return power.y / fmaxf(ee.y, (cx.y * cx.y + cy.y * cy.y) + cz.y * cz.y) * vis.y;
    }
    // both within 2^-20: fused sums and an approximate reciprocal
    __device__ __forceinline__ float2 imp_near() const {
        const float2 cc = __ffma2_rn(cx, cx, __ffma2_rn(cy, cy, __fmul2_rn(cz, cz)));
        float a, b;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(fmaxf(ee.x, cc.x)));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(fmaxf(ee.y, cc.y)));
        return make_float2(power.x * vis.x * a, power.y * vis.y * b);
    }
};
template <bool NEE>
__device__ __forceinline__ LightPair light_pair(const DevScene &sc, const ImpPt &P, uint32_t g) {
    const float4 *q = sc.light_pair + LIGHT_PAIR * (size_t)g;
    float4 a, b;
    ldg2(q, a, b);
    const float4 d = __ldg(q + 2);
    const float eps = NEE ? EPS_NEE : EPS_TRACE;
    const float2 half = make_float2(0.5f, 0.5f);
    const f3 point = P.point;
    LightPair R;
    R.cx = __ffma2_rn(half, make_float2(a.x, a.y), make_float2(-point.x, -point.x));
    R.cy = __ffma2_rn(half, make_float2(a.z, a.w), make_float2(-point.y, -point.y));
    R.cz = __ffma2_rn(half, make_float2(b.x, b.y), make_float2(-point.z, -point.z));
    R.ee = make_float2(b.z, b.w);
    R.power = make_float2(d.x, d.y);
    R.left = __float_as_int(d.z);
    R.right = __float_as_int(d.w);
    if (P.ax >= 0) {
        const float4 w = __ldg(q + 3 + P.ax);
        const float2 s2 = make_float2(P.sg, P.sg), p2 = make_float2(P.sp, P.sp);
        const float2 u = __ffma2_rn(make_float2(w.x, w.y), s2, p2), v = __ffma2_rn(make_float2(w.z, w.w), s2, p2);
        R.vis.x = (u.x >= eps ? 0.5f : 0.0f) + (v.x >= eps ? 0.5f : 0.0f);
        R.vis.y = (u.y >= eps ? 0.5f : 0.0f) + (v.y >= eps ? 0.5f : 0.0f);
    } else {
        const float4 x = __ldg(q + 3), y = __ldg(q + 4), z = __ldg(q + 5);
        float n[2] = {0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float2 kx = (k & 4) ? make_float2(x.z, x.w) : make_float2(x.x, x.y);
            const float2 ky = (k & 2) ? make_float2(y.z, y.w) : make_float2(y.x, y.y);
            const float2 kz = (k & 1) ? make_float2(z.z, z.w) : make_float2(z.x, z.y);
            n[0] += dot3(sub3(f3{kx.x, ky.x, kz.x}, point), P.normal) >= eps ? 0.125f : 0.0f;
            n[1] += dot3(sub3(f3{kx.y, ky.y, kz.y}, point), P.normal) >= eps ? 0.125f : 0.0f;
        }
        R.vis = make_float2(n[0], n[1]);
    }
    return R;
}

struct Descent {
    bool success;
    uint32_t inst, leaf;
    float importance;
};

// traverseBvh (raytrace.rs:218-281)
__device__ Descent light_descent(const DevScene &sc, f3 point, f3 normal, uint32_t seed) {
    Descent R;
    R.success = false;
    R.inst = 0;
    R.leaf = 0;
    R.importance = 0.0f;
    int ref = sc.light_root;
    if (ref == EMPTY_ROOT) return R;
    const ImpPt P = imp_point(point, normal);
    float importance = 0.0f;
    bool top = true;
    for (int guard = 0; guard < 256; guard++) {
        if (ref < 0) {
            if (!top) {
                R.success = true;
                R.leaf = (uint32_t)~ref;
                R.importance = importance;
                return R;
            }
            // an instance: on with its BLAS root, whose importance counts
            // when the top level's was 0
            R.inst = (uint32_t)~ref;
            top = false;
            const InstDev &I = sc.inst[R.inst];
            if (importance == 0.0f) importance = light_pair<false>(sc, P, I.light_tl).imp_l();
            ref = (int)I.light_base;
            if (I.light_leaf) {
                ref = ~0;
                continue;
            }
        }
        // left iff rnd < lI / (lI + rI), in the shader's rounded arithmetic.
        // Values within 2^-20 decide it when the sides of rnd * (lI + rI) < lI
        // are more than 2^-16 of the sum apart (and the sum far from over- and
        // underflow); else the exact ones do.  Only the sign of the chosen
        // importance is used, and a child chosen so has over 2^-16 of the sum.
        const LightPair c = light_pair<false>(sc, P, (uint32_t)ref);
        const float rnd = mm_rand(seed);
        const float2 near = c.imp_near();
        float lI = near.x, rI = near.y;
        const float tot = lI + rI, diff = __fmaf_rn(rnd, tot, -lI);
        bool left = diff < 0.0f;
        if (!(fabsf(diff) > tot * (1.0f / 65536.0f) && tot > 1e-20f && tot < 1e20f)) {
            lI = c.imp_l();
            rI = c.imp_r();
            left = rnd < lI / (lI + rI);  // the shader's right ratio is never read
        }
        ref = left ? c.left : c.right;
        importance = left ? lI : rI;
        seed = mm_combine(seed, 0);
    }
    return R;
}

// reverseTraverseBvh (nee_pdf.rs:154-228)
__device__ float reverse_walk(const DevScene &sc, f3 point, f3 normal, uint32_t ii, uint32_t leaf) {
    float probability = 1.0f;
    const ImpPt P = imp_point(point, normal);
    uint32_t up = __ldg(sc.light_par + sc.inst[ii].light_base + leaf);
    for (int guard = 0; guard < 256 && up != INVALID; guard++) {
        const uint32_t g = up >> 1, right = up & 1u;
        up = __ldg(sc.light_par + g);
        const LightPair c = light_pair<true>(sc, P, g);
        const float lI = c.imp_l(), rI = c.imp_r();
        probability *= (right ? rI : lI) / (lI + rI);
    }
    return probability;
}

// world-space vertices of the light triangle of light-BLAS leaf `leaf` of
// instance ii (the triangleTransform of raytrace.rs:155-159, nee_pdf.rs:95-101)
__device__ __forceinline__ void light_tri_world(const DevScene &sc, uint32_t ii, uint32_t leaf, f3 tv[3]) {
    const InstDev &I = sc.inst[ii];
    uint32_t t = __ldg(I.light_leaf_tri + leaf);
    if (I.flags & INST_MESH) {
        const float4 *r = sc.tri_rec + 3 * (size_t)(I.tri_base + t);
        tv[0] = ld3(__ldg(r));
        tv[1] = ld3(__ldg(r + 1));
        tv[2] = ld3(__ldg(r + 2));
        return;
    }
    int lx = (int)(t & 31u), ly = (int)((t >> 5) & 31u), lz = (int)((t >> 10) & 31u);
    int f = (int)((t >> 15) & 7u), h = (int)((t >> 18) & 1u);
#pragma unroll
    for (int j = 0; j < 3; j++) {
        f3 p = corner_pos(lx, ly, lz, face_corner(f, h, j));
        tv[j] = f3{p.x + I.off[0], p.y + I.off[1], p.z + I.off[2]};
    }
}

// computeNeePdf (nee_pdf.rs:240-279)
__device__ float nee_pdf_of(const DevScene &sc, f3 point, f3 normal, f3 dir, uint32_t ii, uint32_t leaf, float b1,
                            float b2) {
    f3 tv[3];
    light_tri_world(sc, ii, leaf, tv);
    f3 p = add3(add3(lscl3(b1, tv[0]), lscl3(b2, tv[1])), lscl3((1.0f - b1) - b2, tv[2]));
    float light_distance = len3(sub3(p, point));
    float light_area = 0.5f * len3(cross3(sub3(tv[0], tv[1]), sub3(tv[2], tv[1])));
    float cos_theta = dot3(normal, dir);
    float ppp = light_distance * light_distance / (cos_theta * light_area);
    float P = reverse_walk(sc, point, normal, ii, leaf);
    return P * ppp;
}

constexpr int LIGHT_LIST = 32;
constexpr uint32_t FULL = 0xffffffffu;

__device__ __forceinline__ void st3(float *a, size_t i, f3 v) {
    a[3 * i] = v.x;
    a[3 * i + 1] = v.y;
    a[3 * i + 2] = v.z;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// raygen (raygen.rs:84-111): pixel corner, jitter multiplied by 0.00
__device__ __forceinline__ f3 ray_col(const ViewDev &V, uint32_t x) {
    const float u = 2.0f * (float)x / (float)V.W - 1.0f;
    const float aspect = (float)V.W / (float)V.H;
    return scl3(lscl3(u, V.right), aspect);
}
__device__ __forceinline__ f3 ray_row(const ViewDev &V, uint32_t y) {
    return lscl3(2.0f * (float)y / (float)V.H - 1.0f, V.up);
}
__device__ __forceinline__ void raygen(const ViewDev &V, uint32_t x, uint32_t y, f3 &o, f3 &d) {
    o = V.eye;
    d = norm3(add3(add3(ld3(__ldg(V.ray_x + x)), ld3(__ldg(V.ray_y + y))), V.front));
}

// Start of a frame: clears the counters and fills every view's primary-ray
// tables (W + H entries; the terms take three divisions and nine products per
// ray when the closest hit and the shading work them out each for themselves;
// with the integer divisions and the materials' R / pi gone too, the 1080p
// frame in flight went from 1014 to 995 us).  blockIdx.y is the view.
template <bool BATCH>
__global__ void __launch_bounds__(128) k_frame_begin(const __grid_constant__ FrameArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y == 0 && i < CNT_WORDS && i / 2 != CNT_STAMP / 2 + ST_BEGIN) a.counters[i] = 0;
    if (blockIdx.y == 0) stamp_start(a, ST_BEGIN);
    const ViewDev &V = BATCH ? a.views[blockIdx.y] : a.v0;
    if (i < V.W) {
        const f3 c = ray_col(V, i);
        V.ray_x[i] = make_float4(c.x, c.y, c.z, 0.0f);
    } else if (i < V.W + V.H) {
        const f3 c = ray_row(V, i - V.W);
        V.ray_y[i - V.W] = make_float4(c.x, c.y, c.z, 0.0f);
    }
}

// the slab test's offsets of the near and far planes, the boxes widened by m
__device__ __forceinline__ void slab_offsets(f3 o, f3 inv, float m, f3 &oin, f3 &oif) {
    const f3 oi = f3{-o.x * inv.x, -o.y * inv.y, -o.z * inv.z};
    const f3 w = f3{m * fabsf(inv.x), m * fabsf(inv.y), m * fabsf(inv.z)};
    oin = sub3(oi, w);
    oif = add3(oi, w);
}

// Pops the next pending child whose box starts at or before best_t (boxes
// are culled only when strictly beyond it); false when none is left.
__device__ __forceinline__ bool pop_near(const int2 *stack, int &sp, float best_t, int &node) {
    while (sp > 0) {
        const int2 e = stack[--sp];  // (ref, entry distance bits)
        if (__int_as_float(e.y) <= best_t) {
            node = e.x;
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ void cswap(float &ta, int &ra, float &tb, int &rb) {
    if (tb < ta) {
        const float t = ta; ta = tb; tb = t;
        const int r = ra; ra = rb; rb = r;
    }
}

// three-input min / max (sm_100+); NaN inputs are ignored as by fminf/fmaxf
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// v * m + c per component, each a single rounded FMA, two per instruction
// (fma.rn.f32x2).  The walks are bound by the instructions they issue: the
// packed form takes 12 of about 115 off a node's visit (the closest hits of a
// 960x540 frame: 95.0 -> 89.6 M warp instructions) and, with the registers
// capped at 64 so that 8 CTAs share an SM (71 and 7 before), the 1080p frame
// in flight goes from 1093 to 1060 us, a 3840x2160 one from 6060 to 5857.
// (Packed, but at 6 or 7 CTAs: 1081 and 1078 us.)
__device__ __forceinline__ float4 fma4(float4 v, float m, float c) {
    const float2 a = __ffma2_rn(make_float2(v.x, v.y), make_float2(m, m), make_float2(c, c));
    const float2 b = __ffma2_rn(make_float2(v.z, v.w), make_float2(m, m), make_float2(c, c));
    return make_float4(a.x, a.y, b.x, b.y);
}

// slab test of the 4 children of a 4-wide node; returns the entry distances
// sorted ascending (+inf for a miss) with their refs.  NX..FZ are the near and
// far planes per axis, picked per ray by the sign of its direction (so the
// per-axis min/max of the classic slab test is not needed).  For such a pick
// the near distance of a non-empty box is <= its far distance, exactly, since
// rounding is monotonic; a NaN distance (only possible for a direction
// component below 1e-30 in magnitude, whose inverse overflows) is ignored by
// min/max, which only keeps more boxes: the test stays conservative and the
// closest hit does not depend on it.  A component of exactly 0 has the finite
// inverse +-1e30 (slab_inv), so that axis culls like any other.  An unused
// slot holds the inverted box lo = +inf, hi = -inf: on an axis with a finite
// inverse its near distance is +inf, so the slot is never entered and needs
// no test of its ref.
__device__ __forceinline__ void slab4(float4 NX, float4 FX, float4 NY, float4 FY, float4 NZ, float4 FZ, float4 RF,
                                      f3 inv, f3 oin, f3 oif, float tmin, float tmax, float tk[4], int rk[4]) {
    const int rf[4] = {__float_as_int(RF.x), __float_as_int(RF.y), __float_as_int(RF.z), __float_as_int(RF.w)};
    const float4 ax = fma4(NX, inv.x, oin.x), ay = fma4(NY, inv.y, oin.y), az = fma4(NZ, inv.z, oin.z);
    const float4 bx = fma4(FX, inv.x, oif.x), by = fma4(FY, inv.y, oif.y), bz = fma4(FZ, inv.z, oif.z);
    const float nx[4] = {ax.x, ax.y, ax.z, ax.w}, ny[4] = {ay.x, ay.y, ay.z, ay.w}, nz[4] = {az.x, az.y, az.z, az.w};
    const float fx[4] = {bx.x, bx.y, bx.z, bx.w}, fy[4] = {by.x, by.y, by.z, by.w}, fz[4] = {bz.x, bz.y, bz.z, bz.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float tn = fmax3(nx[i], ny[i], fmaxf(nz[i], tmin));
        const float tf = fmin3(fx[i], fy[i], fminf(fz[i], tmax));
        tk[i] = (tn <= tf) ? tn : INFINITY;
        rk[i] = rf[i];
    }
    // sorting network for 4
    cswap(tk[0], rk[0], tk[1], rk[1]);
    cswap(tk[2], rk[2], tk[3], rk[3]);
    cswap(tk[0], rk[0], tk[2], rk[2]);
    cswap(tk[1], rk[1], tk[3], rk[3]);
    cswap(tk[1], rk[1], tk[2], rk[2]);
}

// Work distribution of the persistent walks.  A returning atomicAdd by one
// lane per warp on one word takes 0.66 ns chip-wide and, with every warp of
// the chip queueing for it, 3.2 us each (311 K of them in 205 us).  So a warp
// does not fetch at every refill: it owns a range of the queue and refills its
// lanes from it.  Its first 32 entries are its static share (no atomic; a warp
// past the queue's end leaves at once), then it takes chunks that shrink with
// what is left (a quarter of its even share, 32 to 256 entries), so that the
// last warps finish together.  The closest hits of a 640x480 frame's bounces:
// 40 + 94 + 62 -> 33 + 70 + 45 us; of a 1080p frame's 125 + 332 + 382 -> 132 +
// 269 + 361 us (chunks of at most 32: 134 + 274 + 358; at 3840x2160 548 + 1307
// + 1657 us against 638 + 1376 + 1812 with 32).
struct WarpRange {
    uint32_t cur, end, last;  // the entries [cur, end) in hand; the end of the last chunk taken
    bool more;                // the queue may hold entries past it
};
constexpr uint32_t CHUNK_MAX = 256;

// Entries of a warp's static share: 32, or one where the queue holds fewer
// entries than there are resident warps: a warp's divergent lanes follow one
// another, and such a queue's kernel lasts as long as its slowest warp (64x64
// pixels: closest hits 22 -> 18 us, the frame 132 -> 128).  Longer queues keep
// whole warps: spread at 8 entries per warp and more, a 957x541 frame in flight
// took 288 us, not 270.
__device__ __forceinline__ uint32_t first_share(uint32_t n_in, uint32_t all) {
    return n_in >= all ? 32u : 1u;
}

__device__ __forceinline__ WarpRange range_first(uint32_t n_in) {
    const uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), all = gridDim.x * (blockDim.x >> 5);
    const uint32_t share = first_share(n_in, all);
    WarpRange r;
    r.cur = min(share * w, n_in);
    r.end = min(share * w + share, n_in);
    r.last = share * all;
    r.more = r.last < n_in;
    return r;
}

// the next chunk (all lanes; fetch counts the entries past the static shares)
__device__ __forceinline__ void range_next(WarpRange &r, uint32_t n_in, uint32_t *fetch) {
    const uint32_t all = gridDim.x * (blockDim.x >> 5);
    const uint32_t size = min(((n_in - r.last) / (128u * all) + 1u) * 32u, CHUNK_MAX);
    uint32_t base = 0;
    if ((threadIdx.x & 31u) == 0) base = atomicAdd(fetch, size);
    base = first_share(n_in, all) * all + __shfl_sync(0xffffffffu, base, 0);
    r.cur = min(base, n_in);
    r.last = r.end = min(base + size, n_in);
    r.more = r.end < n_in;
}

// Adds each warp's totals to N u64 counters, one atomic per CTA and counter:
// the CTA's last warp to finish publishes the sums (s_sum: N + 1 words of
// shared memory, zeroed before the walk); true for the lane that did.
template <int N>
__device__ __forceinline__ bool publish_totals(uint32_t *s_sum, uint32_t *counters, const int (&at)[N],
                                               const uint32_t (&v)[N]) {
    if ((threadIdx.x & 31u) != 0) return false;
#pragma unroll
    for (int k = 0; k < N; k++)
        if (v[k]) atomicAdd(s_sum + k, v[k]);
    __threadfence_block();
    if (atomicAdd(s_sum + N, 1u) != (blockDim.x >> 5) - 1u) return false;
    __threadfence_block();
#pragma unroll
    for (int k = 0; k < N; k++) {
        const uint32_t t = atomicAdd(s_sum + k, 0u);
        if (t) atomicAdd(reinterpret_cast<unsigned long long *>(counters + at[k]), (unsigned long long)t);
    }
    return true;
}

// ---------------------------------------------------------------------------
// k_trace: closest hit over the voxel faces (replaces getIntersectionInfo,
// raytrace.rs:354-388).  Persistent warps; each lane owns one ray and, when
// its traversal ends, takes a new ray from its warp's range of the bounce queue
// (once a.refill_trace lanes are idle), so a warp does not wait for its
// longest ray.  The result is independent of traversal order: ties on t go
// to the smaller (instance, triangle) key and boxes are culled only when
// strictly beyond the current best t.  In a batched frame each lane reads the
// scene of its ray's view when it takes the ray.
// ---------------------------------------------------------------------------
template <bool BATCH, bool MESH>
__global__ void __launch_bounds__(128, 8) k_trace(const __grid_constant__ FrameArgs a, uint32_t b) {
    __shared__ uint32_t s_sum[4];
    const int REFILL = (int)a.refill_trace;
    const uint32_t n_in = (b == 0) ? a.n0 : a.counters[a.qsel ? CNT_TQUEUE : CNT_QUEUE + b];
    const uint32_t *qin = a.qsel ? a.tq : a.queue[(b + 1) & 1];
    uint32_t *fetch = a.counters + (a.qsel ? CNT_TFETCH : CNT_FETCH + b);
    uint32_t *err = a.counters + CNT_ERROR;
    const float4 *wide = a.v0.sc.geo_wide;
    const int4 *recs = a.v0.sc.geo_rec;
    const float4 *tris = a.v0.sc.tri_rec;
    uint32_t nblk = a.v0.sc.n_blk_rec;
    float extent = a.v0.sc.extent;
    int root = a.v0.sc.geo_root;
    if (threadIdx.x < 4) s_sum[threadIdx.x] = 0;
    __syncthreads();
    WarpRange range = range_first(n_in);
    bool has = false;
    uint32_t p = 0, steps = 0, traced = 0, n_nodes = 0, n_leaves = 0;
    f3 o = f3{0, 0, 0}, d = f3{0, 0, 0}, inv = f3{0, 0, 0}, oin = f3{0, 0, 0}, oif = f3{0, 0, 0};
    float best_t = 0.0f, hb1 = 0.0f, hb2 = 0.0f;
    uint64_t best_key = 0;
    int node = 0, sp = 0, hrec = -1;
    uint32_t hfh = 0;
    int px = 0, py = 2, pz = 4;  // float4 index of the near plane per axis (the far one is next to it)
    // pending children with their entry distances: a popped entry whose box
    // starts beyond the current best t is dropped unvisited (every box below
    // it starts no nearer, so each would be culled by its own test)
    int2 stack[TRAV_STACK];
    while (true) {
        const uint32_t need = __ballot_sync(FULL, !has);
        if ((range.cur < range.end || range.more) && need && (__popc(need) >= REFILL || need == FULL)) {
            if (range.cur == range.end) range_next(range, n_in, fetch);
            const uint32_t base = range.cur;
            range.cur = min(base + (uint32_t)__popc(need), range.end);
            if (!has) {
                const uint32_t idx = base + (uint32_t)__popc(need & lanemask_lt());
                uint32_t x = 0, y = 0;
                if (idx < range.end &&
                    (b == 0 ? bounce0_pixel(view_of_tile<BATCH>(a, idx >> 5), idx, p, x, y) : (p = qin[idx], true))) {
                    has = true;
                    traced++;
                    const ViewDev &V = view_of<BATCH>(a, p);
                    if constexpr (BATCH) {
                        wide = V.sc.geo_wide;
                        recs = V.sc.geo_rec;
                        tris = V.sc.tri_rec;
                        nblk = V.sc.n_blk_rec;
                        extent = V.sc.extent;
                        root = V.sc.geo_root;
                    }
                    if (b == 0) raygen(V, x, y, o, d);
                    else {
                        float4 ro, rd;
                        ld2(a.ray + 2 * (size_t)p, ro, rd);
                        o = ld3(ro);
                        d = ld3(rd);
                    }
                    inv = f3{slab_inv(d.x), slab_inv(d.y), slab_inv(d.z)};
                    slab_offsets(o, inv, ray_margin(extent, o), oin, oif);
                    px = signbit(inv.x) ? 1 : 0;
                    py = signbit(inv.y) ? 3 : 2;
                    pz = signbit(inv.z) ? 5 : 4;
                    best_t = 1000.0f;
                    best_key = ~0ull;
                    node = root;
                    sp = 0;
                    hrec = -1;
                    steps = 0;
                }
            }
        }
        if (!__any_sync(FULL, has)) {
            if (range.cur < range.end || range.more) continue;
            break;
        }
        // descend through 4-wide inner nodes to the next leaf
        bool done = has && (node == EMPTY_ROOT);
        while (true) {
            const bool inner = has && !done && node >= 0;
            if (!__any_sync(FULL, inner)) break;
            if (inner) {
                const float4 *w = wide + 8 * (size_t)node;
                const float4 NX = __ldg(w + px), FX = __ldg(w + (px ^ 1)), NY = __ldg(w + py);
                const float4 FY = __ldg(w + (py ^ 1)), NZ = __ldg(w + pz), FZ = __ldg(w + (pz ^ 1));
                const float4 RF = __ldg(w + 6);
                float tk[4];
                int rk[4];
                slab4(NX, FX, NY, FY, NZ, FZ, RF, inv, oin, oif, EPS_TRACE, best_t, tk, rk);
                // tk sorted ascending (misses at +inf)
                if (tk[0] == INFINITY) {
                    done = !pop_near(stack, sp, best_t, node);
                } else {
                    node = rk[0];
                    if (sp + 3 <= TRAV_STACK) {
                        if (tk[3] != INFINITY) stack[sp++] = make_int2(rk[3], __float_as_int(tk[3]));
                        if (tk[2] != INFINITY) stack[sp++] = make_int2(rk[2], __float_as_int(tk[2]));
                        if (tk[1] != INFINITY) stack[sp++] = make_int2(rk[1], __float_as_int(tk[1]));
                    } else {
                        atomicOr(err, ERR_STACK);
                    }
                }
                if (++steps > TRAV_GUARD) {  // only reachable with a malformed layout
                    atomicOr(err, ERR_GUARD);
                    done = true;
                }
            }
        }
        if (has && (done || node < 0)) {
            if (MESH && !done && (uint32_t)(~node) >= nblk) {  // leaf: one world-space mesh triangle
                const float4 *tr = tris + 3 * (size_t)((uint32_t)(~node) - nblk);
                const float4 A = __ldg(tr), B = __ldg(tr + 1), C = __ldg(tr + 2);
                n_leaves++;
                TriHit th;
                if (tri_test(ld3(A), ld3(B), ld3(C), o, d, EPS_TRACE, best_t, th)) {
                    const uint64_t key = ((uint64_t)__float_as_uint(A.w) << 32) | __float_as_uint(B.w);
                    if (th.t < best_t || key < best_key) {
                        best_t = th.t;
                        best_key = key;
                        hrec = ~node;
                        hfh = 0;
                        hb1 = th.b1;
                        hb2 = th.b2;
                    }
                }
                done = !pop_near(stack, sp, best_t, node);
            } else if (!done) {  // leaf: the exposed faces of one surface block
                const int4 r = __ldg(recs + (~node));
                n_leaves++;
                const int wx = rec_wx(r), wy = rec_wy(r), wz = rec_wz(r);
                const uint32_t mask = ((uint32_t)r.z >> 15) & 63u;
                const uint64_t ikey = (uint64_t)rec_inst(r) << 32;
                for (uint32_t m = mask; m; m &= m - 1u) {
                    const int f = __ffs(m) - 1;
                    FaceHit fh;
                    if (face_test(wx, wy, wz, f, o, d, inv, EPS_TRACE, best_t, fh)) {
                        const uint32_t rank = __popc(mask & ((1u << f) - 1u));
                        const uint64_t key = ikey | ((uint32_t)r.w + 2u * rank + (uint32_t)fh.half);
                        if (fh.t < best_t || key < best_key) {
                            best_t = fh.t;
                            best_key = key;
                            hrec = ~node;
                            hfh = (uint32_t)f | ((uint32_t)fh.half << 3);
                            hb1 = fh.b1;
                            hb2 = fh.b2;
                        }
                    }
                }
                done = !pop_near(stack, sp, best_t, node);
            }
            if (done) {
                n_nodes += steps;
                a.hits[p] = make_int4(hrec, (int)hfh, __float_as_int(hb1), __float_as_int(hb2));
                has = false;
            }
        }
    }
    for (int off = 16; off; off >>= 1) {
        traced += __shfl_xor_sync(FULL, traced, off);
        n_nodes += __shfl_xor_sync(FULL, n_nodes, off);
        n_leaves += __shfl_xor_sync(FULL, n_leaves, off);
    }
    if (publish_totals<3>(s_sum, a.counters, {CNT_RAYS, CNT_NODES, CNT_LEAVES}, {traced, n_nodes, n_leaves}))
        stamp_end(a, ST_TRACED + b);
}

// Shading of one path vertex (raytrace.rs:405-577): the hit's material
// (constant slot colours or the texture atlas), emission, and the sampled
// continuation (mirror, transmission, or Lambertian with light-BVH NEE
// sampling).
struct ShadeOut {
    f3 n, E, R, new_o, new_d;
    float mis, pdf;
    int face, half;
    int4 rc;
};

// need_dir false: the path ends at this vertex (its last bounce, or a cache
// frame's query vertex of a path that does not train; no capture) and only
// its emission (or the cache's prediction) reaches the image: the outgoing radiance of the last
// vertex is E + (R * 0) * w = E for any finite R >= 0 and w > 0, and the
// vertex position keeps its offset; the Lambertian continuation (light-BVH
// descent and direction sampling) is skipped, with mis 0 and pdf 1.
template <bool MESH>
__device__ __forceinline__ void shade_vertex(const DevScene &S, uint32_t nee_type, uint32_t b, uint32_t seed, f3 o,
                                             f3 d, int4 hv, bool need_dir, ShadeOut &out) {
    f3 n, E, R, new_o, new_d;
    float mis = 0.0f, pdf = 1.0f;
    int face = 0, half = 0;
    int4 rc = make_int4(0, 0, 0, 0);
    if (hv.x < 0) {
        new_o = add3(o, scl3(d, 5000.0f));
        new_d = f3{0.0f, 0.0f, 0.0f};
        n = f3{0.0f, 0.0f, 0.0f};
        const float sky = (dot3(d, f3{0.0f, 1.0f, 0.0f}) > 0.9f) ? 50.0f : 0.0f;
        E = f3{sky, sky, sky};
        R = f3{0.0f, 0.0f, 0.0f};
    } else {
        const float b1 = __int_as_float(hv.z), b2 = __int_as_float(hv.w);
        const float b0 = (1.0f - b1) - b2;
        f3 t0, t1, t2;
        Frame fr;                    // the tangent and bitangent where the direction needs them
        const float4 *ft = nullptr;  // a voxel face's row of d_faces
        uint32_t slot;
        float u = 0.0f, v = 0.0f;  // the texture coordinate (read with an atlas only)
        if (MESH && (uint32_t)hv.x >= S.n_blk_rec) {
            // a mesh triangle: its world-space vertices and material slot;
            // localCoordinateSystem of the triangle (raytrace.rs:319-331);
            // face carries bit 31 | its record (the normal of the light-pdf walk)
            const uint32_t tr = (uint32_t)hv.x - S.n_blk_rec;
            const float4 *q = S.tri_rec + 3 * (size_t)tr;
            const float4 A = __ldg(q), B = __ldg(q + 1), C = __ldg(q + 2);
            t0 = ld3(A);
            t1 = ld3(B);
            t2 = ld3(C);
            fr.n = tri_frame(t0, t1, t2).n;
            slot = __float_as_uint(C.w);
            face = (int)(0x80000000u | tr);
            rc = make_int4((int)__float_as_uint(A.w), (int)__float_as_uint(B.w), -1, 0);
            if (S.atlas) {  // uv = v0.uv * b0 + v1.uv * b1 + v2.uv * b2 (raytrace.rs:457)
                const float *uv = S.inst[rc.x].uv + 6 * (size_t)rc.y;
                u = ((__ldg(uv) * b0) + (__ldg(uv + 2) * b1)) + (__ldg(uv + 4) * b2);
                v = ((__ldg(uv + 1) * b0) + (__ldg(uv + 3) * b1)) + (__ldg(uv + 5) * b2);
            }
        } else {
            rc = __ldg(S.geo_rec + hv.x);
            face = hv.y & 7;
            half = (hv.y >> 3) & 1;
            const int wx = rec_wx(rc), wy = rec_wy(rc), wz = rec_wz(rc);
            ft = d_faces + FACE_ROW * (2 * face + half);
            const float4 q = __ldg(ft);
            const uint32_t cb = __float_as_uint(q.w);
            fr.n = ld3(q);
            t0 = corner_pos(wx, wy, wz, cb & 7u);
            t1 = corner_pos(wx, wy, wz, (cb >> 3) & 7u);
            t2 = corner_pos(wx, wy, wz, cb >> 6);
            const uint32_t blk_id = ((uint32_t)rc.z >> 21) & 0xFFu;
            slot = 6u * blk_id + (uint32_t)face;
            if (S.atlas) {  // gen_mesh's corner uvs
                const uint32_t q0 = face_uv(face, half, 0), q1 = face_uv(face, half, 1),
                               q2 = face_uv(face, half, 2);
                u = (((float)(q0 & 1u) * b0) + ((float)(q1 & 1u) * b1)) + ((float)(q2 & 1u) * b2);
                v = (((float)(q0 >> 1) * b0) + ((float)(q1 >> 1) * b1)) + ((float)(q2 >> 1) * b2);
            }
        }
        n = fr.n;
        new_o = add3(add3(scl3(t0, b0), scl3(t1, b1)), scl3(t2, b2));
        const float ndd = -dot3(d, n);
        float alpha, metal;
        if (S.atlas) {
            // texture atlas: the three maps at the interpolated uv
            // (raytrace.rs:457-480), nearest texel clamped to the edge
            const int aw = (int)S.atlas_w, ah = (int)S.atlas_h;
            const int ix = min(max((int)floorf(u * (float)aw), 0), aw - 1);
            const int iy = min(max((int)floorf(v * (float)ah), 0), ah - 1);
            const size_t texel = (size_t)slot * 3 * aw * ah + (size_t)iy * aw + ix, map = (size_t)aw * ah;
            const uchar4 x0 = __ldg(S.atlas + texel), x1 = __ldg(S.atlas + texel + map),
                         x2 = __ldg(S.atlas + texel + 2 * map);
            const float *lin = S.srgb;
            R = f3{__ldg(lin + x0.x), __ldg(lin + x0.y), __ldg(lin + x0.z)};
            alpha = (float)x0.w / 255.0f;
            E = f3{(1000.0f * __ldg(lin + x1.x)) * ndd, (1000.0f * __ldg(lin + x1.y)) * ndd,
                   (1000.0f * __ldg(lin + x1.z)) * ndd};
            metal = __ldg(lin + x2.x);
        } else {
            // (reflectivity, alpha), (emission, metallic)
            const float4 *m = reinterpret_cast<const float4 *>(S.mats + slot);
            const float4 ra = __ldg(m), em = __ldg(m + 1);
            R = ld3(ra);
            alpha = ra.w;
            E = f3{em.x * ndd, em.y * ndd, em.z * ndd};
            metal = em.w;
        }
        const float r0 = mm_rand(mm_combine(seed, 0));
        if (r0 < metal) {
            pdf = 1.0f;
            new_d = sub3(d, lscl3(2.0f * dot3(n, d), n));
        } else if (r0 < metal + (1.0f - alpha)) {
            new_d = d;
            R = f3{1.0f, 1.0f, 1.0f};
            pdf = 1.0f;
        } else {
            new_o = add3(new_o, lscl3(EPS_TRACE * 1.5f, n));
            if (S.atlas) R = f3{R.x / PI_F, R.y / PI_F, R.z / PI_F};
            else R = ld3(__ldg(S.lambert + slot));
            if (!need_dir) {
                new_d = f3{0.0f, 0.0f, 0.0f};
                goto done;
            }
            Descent res;
            res.success = false;
            res.importance = 0.0f;
            if (nee_type == 1 || (nee_type == 2 && b == 1))
                res = light_descent(S, new_o, n, mm_combine(seed, 2));
            if (res.success && res.importance > 0.0f) mis = 0.3f;
            const float mis_rand = mm_rand(mm_combine(seed, 3));
            float ux = mm_rand(mm_combine(seed, 4)), uy = mm_rand(mm_combine(seed, 5));
            if (mis_rand < mis) {
                f3 lt[3];
                light_tri_world(S, res.inst, res.leaf, lt);
                if (ux + uy > 1.0f) { ux = 1.0f - ux; uy = 1.0f - uy; }  // triangleSample
                const float bx = (1.0f - ux) - uy;
                const f3 sp = add3(add3(lscl3(bx, lt[0]), lscl3(ux, lt[1])), lscl3(uy, lt[2]));
                new_d = norm3(sub3(sp, new_o));
            } else {
                float s, c;
                sincos_turns(ux, &s, &c);
                const float vv = sqrtf(fmaxf(0.0f, 1.0f - uy * uy));
                const f3 hs = f3{vv * c, uy, vv * s};
                if (!MESH || ft) {
                    float4 ta, bi;
                    ldg2(ft + 2, ta, bi);
                    fr.t = ld3(ta);
                    fr.b = ld3(bi);
                } else {  // (worked out again here, not carried through the descent)
                    const float4 *q = S.tri_rec + 3 * (size_t)((uint32_t)face & 0x7FFFFFFFu);
                    fr = tri_frame(ld3(__ldg(q)), ld3(__ldg(q + 1)), ld3(__ldg(q + 2)));
                }
                new_d = norm3(add3(add3(lscl3(hs.x, fr.t), lscl3(hs.y, fr.n)), lscl3(hs.z, fr.b)));
            }
            pdf = dot3(new_d, n) / PI_F;
        }
    }
done:
    out.n = n;
    out.E = E;
    out.R = R;
    out.new_o = new_o;
    out.new_d = new_d;
    out.mis = mis;
    out.pdf = pdf;
    out.face = face;
    out.half = half;
    out.rc = rc;
}

// ---------------------------------------------------------------------------
// k_shade: shading of the hit, light-BVH descent and direction sampling
// (raytrace.rs:405-577).  Rays whose light pdf is needed are queued for
// k_anyhit; the others get their (E, w) (R, q) record here.
// ---------------------------------------------------------------------------
constexpr uint32_t SHADE_BATCH = 4;  // queue entries per lane of a surface-first shading batch

// the bounces whose shading takes its queue in routed batches (k_shade)
__host__ __device__ __forceinline__ bool shade_split(const FrameArgs &a, uint32_t b) {
    return b > 0 && b + 1 < a.nb;
}

// A cache frame's query vertex continues on one path in 16: the training
// paths, picked by a hash of the frame and the view's pixel.
__device__ __forceinline__ bool want_train_of(const ViewDev &V, uint32_t lp) {
    return (mm_finalize(mm_combine(V.frame * 0x9E3779B9u + 0x7a11u, lp)) & 15u) == 0u;
}

template <bool CAPTURE, bool BATCH, bool MESH, bool SPLIT>
__global__ void __launch_bounds__(128, 8) k_shade(const __grid_constant__ FrameArgs a, uint32_t b) {
    // per warp: the batch's pixels, surface hits first
    __shared__ uint32_t s_route[SPLIT ? 4 : 1][SPLIT ? 32 * SHADE_BATCH : 1];
    const int lane = threadIdx.x & 31;
    const uint32_t P = a.P, nb = a.nb;
    const uint32_t n_in = (b == 0) ? a.n0 : a.counters[a.qsel ? CNT_TQUEUE : CNT_QUEUE + b];
    const uint32_t *qin = a.qsel ? a.tq : a.queue[(b + 1) & 1];
    uint32_t *qout = a.queue[b & 1];
    // the bounce before a split query bounce: training candidates go to tq
    const bool to_tq = a.tq_split && b + 2 == a.nb_render;
    const float inv2pi = 1.0f / (2.0f * PI_F);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t wid = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    // SPLIT (secondary bounces that continue): each warp takes SHADE_BATCH x
    // 32 queue entries and shades first those that sample a continuation (the
    // light-BVH descent and the direction), 32 at a time, then the others, so
    // that a lane with little to do does not sit out its neighbours'
    // descents.  Those are the surface hits, and at a cache frame's query
    // vertex (without capture) the surface hits of the training paths; the
    // others are the sky misses, and the query vertices that end into the
    // cache.  Every pixel's results are independent of the order of shading.
    const bool split = SPLIT && shade_split(a, b);
    const bool route_train = !CAPTURE && a.cache && b + 1 == a.nb_render;
    // (Batches of 128 entries when every warp gets two of them, of 64 or 32
    // for shorter queues, whose batches of 128 would leave most warps idle:
    // 128 K entries took 47 us in batches of 128 on 1988 of 4864 warps, 20 us
    // in batches of 32.)
    const uint32_t per = !split                                     ? 1u
                         : n_in >= 2u * SHADE_BATCH * 32u * warps ? SHADE_BATCH
                         : n_in >= 2u * 64u * warps               ? 2u
                                                                  : 1u;
    const uint32_t span = split ? 32u * per : first_share(n_in, warps);
    uint32_t *route = s_route[threadIdx.x >> 5];
    for (uint32_t base = wid * span; base < n_in; base += warps * span) {
        uint32_t n_route = 0;
        if (split) {
            uint32_t pk[SHADE_BATCH], surf[SHADE_BATCH], valid[SHADE_BATCH];
            uint32_t n_surf = 0;
#pragma unroll
            for (uint32_t k = 0; k < SHADE_BATCH; k++) {
                const uint32_t i = base + 32 * k + lane;
                const bool v = k < per && i < n_in;
                pk[k] = v ? qin[i] : 0u;
                bool sf = v && a.hits[pk[k]].x >= 0;
                if (sf && route_train) {
                    const ViewDev &V = view_of<BATCH>(a, pk[k]);
                    sf = want_train_of(V, pk[k] - V.pix_off);
                }
                surf[k] = __ballot_sync(FULL, sf);
                valid[k] = __ballot_sync(FULL, v);
                n_surf += __popc(surf[k]);
            }
            uint32_t before_s = 0, before_m = n_surf;
#pragma unroll
            for (uint32_t k = 0; k < SHADE_BATCH; k++) {
                const uint32_t miss = valid[k] & ~surf[k];
                if ((surf[k] >> lane) & 1u) route[before_s + __popc(surf[k] & lanemask_lt())] = pk[k];
                else if ((miss >> lane) & 1u) route[before_m + __popc(miss & lanemask_lt())] = pk[k];
                before_s += __popc(surf[k]);
                before_m += __popc(miss);
            }
            n_route = before_m;
            __syncwarp();
        }
        const uint32_t passes = split ? (n_route + 31u) / 32u : 1u;
        for (uint32_t pass = 0; pass < passes; pass++) {
            uint32_t p = 0, px = 0, py = 0;
            bool active;
            if (split) {
                const uint32_t r = 32 * pass + lane;
                active = r < n_route;
                if (active) p = route[r];
            } else {
                const uint32_t i = base + lane;
                active = (uint32_t)lane < span && i < n_in &&
                         (b == 0 ? bounce0_pixel(view_of_tile<BATCH>(a, i >> 5), i, p, px, py) : (p = qin[i], true));
            }
            bool cont = false, anyj = false, qhit = false, want_train = false;
            const bool at_query = a.cache && b + 1 == a.nb_render;
            f3 stash_E = f3{0, 0, 0}, stash_R = f3{0, 0, 0}, stash_n = f3{0, 0, 0};
            float stash_mis = 0.0f;
            int4 stash_hit = make_int4(-1, 0, 0, 0), stash_rc = make_int4(0, 0, 0, 0);
            int stash_half = 0;
            f3 new_o = f3{0, 0, 0}, new_d = f3{0, 0, 0};
            float pdf = 1.0f;
            int face = 0;
            if (active) {
                const ViewDev &V = view_of<BATCH>(a, p);
                const uint32_t lp = p - V.pix_off;
                f3 o, d;
                if (b == 0) {
                    raygen(V, px, py, o, d);
                    if (CAPTURE) {
                        st3(a.c_origin, p, o);
                        st3(a.c_dir, p, d);
                    }
                } else {
                    float4 ro, rd;
                    ld2(a.ray + 2 * (size_t)p, ro, rd);
                    o = ld3(ro);
                    d = ld3(rd);
                }
                const uint32_t seed = mm_combine(V.frame * nb + b, lp);  // interactive_rendering.rs:1189
                const int4 hv = a.hits[p];
                // A cache frame's query vertex continues only on its training paths
                // (one in 16): on the others the cache's prediction replaces the
                // vertex's outgoing radiance, and its record, direction and light
                // pdf are never read, so they skip the continuation as a last
                // vertex does.
                if (at_query || to_tq) want_train = want_train_of(V, lp);
                ShadeOut so;
                shade_vertex<MESH>(V.sc, a.nee_type, b, seed, o, d, hv,
                                   CAPTURE || (b + 1 < nb && (!at_query || want_train)), so);
                const f3 n = so.n, E = so.E;
                f3 R = so.R;
                const float mis = so.mis;
                const int half = so.half;
                const int4 rc = so.rc;
                new_o = so.new_o;
                new_d = so.new_d;
                pdf = so.pdf;
                face = so.face;
                // the light pdf of the chosen direction (nee_pdf pass, bounce nb-1 never computed)
                if (hv.x >= 0) anyj = (b + 1 < nb) && mis != 0.0f && len3(new_d) != 0.0f;
                // radiance cache: the vertex where rendered paths end into the cache
                // (every pixel's flag is cleared at bounce 0, so a path that ends
                // before the query vertex never reads a stale one)
                if (a.cache && b == 0 && !at_query) a.qflag[p] = 0;
                if (at_query) {
                    qhit = hv.x >= 0;
                    a.qflag[p] = qhit ? 1 : 0;
                    if (qhit) {
                        // the cache's normal: a face index, or a mesh normal packed in 32 bits
                        a.q_pos[p] = make_float4(new_o.x, new_o.y, new_o.z,
                                                 face >= 0 ? __int_as_float(face) : __uint_as_float(pack_normal10(so.n)));
                        a.q_dir[p] = make_float4(d.x, d.y, d.z, 0.0f);
                    }
                }
                // stash for the second half (after the warp-level training-slot grant)
                stash_E = E;
                stash_R = R;
                stash_n = n;
                stash_mis = mis;
                stash_hit = hv;
                stash_rc = rc;
                stash_half = half;
            }
            // training paths: up to train_cap per frame, granted per warp
            bool is_train = false;
            if (at_query) {
                const uint32_t tm = __ballot_sync(FULL, active && qhit && want_train);
                const uint32_t im = __ballot_sync(FULL, active && qhit);
                uint32_t tb = 0, ib = 0;
                if (lane == 0) {
                    if (tm) tb = atomicAdd(&a.counters[CNT_TRAIN], (uint32_t)__popc(tm));
                    if (im) ib = atomicAdd(&a.counters[CNT_INFER], (uint32_t)__popc(im));
                }
                tb = __shfl_sync(FULL, tb, 0);
                ib = __shfl_sync(FULL, ib, 0);
                if (active && qhit) a.infer_list[ib + __popc(im & lanemask_lt())] = p;
                if (active && qhit && want_train) {
                    const uint32_t slot = tb + __popc(tm & lanemask_lt());
                    if (slot < a.train_cap) {
                        a.train_list[slot] = p;
                        is_train = true;
                    }
                }
                if (!is_train) anyj = false;  // the record of this bounce is replaced by the cache
            }
            if (active) {
                const f3 E = stash_E, R = stash_R, n = stash_n;
                const float mis = stash_mis;
                const int4 hv = stash_hit, rc = stash_rc;
                const int half = stash_half;
                // the record without a light hit; a light-pdf job whose ray crosses
                // lights gets its q and w from k_hit_eval / k_hit_sum
                const float q = 0.0f * mis + (1.0f - mis) * inv2pi;
                const float w = pdf / q;
                st2(a.rec + 2 * ((size_t)b * P + p), make_float4(E.x, E.y, E.z, w), make_float4(R.x, R.y, R.z, q));
                if (b < 2) {
                    const int nw = hv.x < 0 ? NORMAL_NONE : face < 0 ? face : 2 * face + half;
                    (b == 0 ? a.xv : a.xs)[p] = make_float4(new_o.x, new_o.y, new_o.z, __int_as_float(nw));
                }
                cont = !zero3(new_d) && (b + 1 < nb) && (!at_query || is_train);
                if (cont) {
                    // .w of the ray carries the face and the bsdf pdf to k_anyhit
                    st2(a.ray + 2 * (size_t)p, make_float4(new_o.x, new_o.y, new_o.z, __int_as_float(face)),
                        make_float4(new_d.x, new_d.y, new_d.z, pdf));
                } else {
                    a.nlive[p] = (uint8_t)(b + 1);
                }
                if (CAPTURE) {
                    const size_t s1 = (size_t)(b + 1) * P + p, s0 = (size_t)b * P + p;
                    st3(a.c_origin, s1, new_o);
                    st3(a.c_dir, s1, new_d);
                    st3(a.c_normal, s0, n);
                    st3(a.c_emis, s0, E);
                    st3(a.c_refl, s0, R);
                    a.c_mis[s0] = mis;
                    a.c_pdf[s0] = pdf;
                    a.c_nee[s0] = 0.0f;
                    uint4 hw;
                    if (face < 0) {  // a mesh triangle: (instance, triangle)
                        hw = make_uint4((uint32_t)rc.x, (uint32_t)rc.y, INVALID, 0u);
                    } else if (hv.x >= 0) {
                        const uint32_t mask = ((uint32_t)rc.z >> 15) & 63u;
                        hw.x = rec_inst(rc);
                        hw.y = (uint32_t)rc.w + 2u * __popc(mask & ((1u << face) - 1u)) + (uint32_t)half;
                        hw.z = (uint32_t)rc.z & 0x7FFFu;
                        hw.w = (uint32_t)face | ((uint32_t)half << 8);
                    } else {
                        hw = make_uint4(INVALID, INVALID, INVALID, INVALID);
                    }
                    reinterpret_cast<uint4 *>(a.c_hit)[s0] = hw;
                }
            }
            // compaction: continuing rays into the next bounce queue, light-pdf jobs
            // into the any-hit queue (one ballot + one atomic per warp each)
            const bool cont_t = cont && to_tq && want_train;  // a training candidate's ray
            const uint32_t cm = __ballot_sync(FULL, cont && !cont_t);
            const uint32_t am = __ballot_sync(FULL, anyj);
            uint32_t qb = 0, ab = 0;
            if (lane == 0) {
                if (cm) qb = atomicAdd(&a.counters[CNT_QUEUE + b + 1], (uint32_t)__popc(cm));
                if (am) ab = atomicAdd(&a.counters[CNT_AQUEUE + b], (uint32_t)__popc(am));
            }
            qb = __shfl_sync(FULL, qb, 0);
            ab = __shfl_sync(FULL, ab, 0);
            if (cont && !cont_t) qout[qb + __popc(cm & lanemask_lt())] = p;
            if (to_tq) {
                const uint32_t tm = __ballot_sync(FULL, cont_t);
                uint32_t tb = 0;
                if (lane == 0 && tm) tb = atomicAdd(&a.counters[CNT_TQUEUE], (uint32_t)__popc(tm));
                tb = __shfl_sync(FULL, tb, 0);
                if (cont_t) a.tq[tb + __popc(tm & lanemask_lt())] = p;
            }
            if (anyj) {
                const uint32_t j = ab + __popc(am & lanemask_lt());
                a.aqueue[b & 1][j] = p;
                st2(a.ajob[b & 1] + 2 * (size_t)j, make_float4(new_o.x, new_o.y, new_o.z, __int_as_float(face)),
                    make_float4(new_d.x, new_d.y, new_d.z, pdf));
            }
        }
        // (the warp's end; behind the loop the same stamp made every shading 1%
        // slower, written or not)
        if (lane == 0 && n_in - base <= warps * span) stamp_end(a, ST_SHADED + b);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// The nee_pdf pass (nee_pdf.rs:281-337) for the queued rays, in three passes
// so that each runs with coherent lanes:
//   k_anyhit     every light triangle the ray crosses in [1e-4, 1000] is
//                collected in ascending (instance, leaf) order; a ray that
//                crosses none (69% at 1080p) keeps the record its shading
//                wrote for that case;
//   k_hit_eval   one thread per hit: computeNeePdf (nee_pdf.rs:240-279) with
//                its reverse walk up the light BVH; a job's only hit (26% of
//                the jobs) completes the bounce record: q and w = bsdf_pdf / q;
//   k_hit_sum    one thread per job with several hits (5%): the sum in key
//                order, then the record.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void finish_job(const FrameArgs &a, uint32_t b, uint32_t p, float pdf, float nee) {
    const float inv2pi = 1.0f / (2.0f * PI_F);
    const float mis = 0.3f;
    const float q = nee * mis + (1.0f - mis) * inv2pi;
    const float w = pdf / q;
    float4 *rec = a.rec + 2 * ((size_t)b * a.P + p);
    rec[0].w = w;
    rec[1].w = q;
}

// a job's hits in ascending key order
struct HitList {
    uint64_t key[LIGHT_LIST];
    float b1[LIGHT_LIST], b2[LIGHT_LIST];
};
__device__ __forceinline__ void hit_insert(HitList &L, int &nh, uint64_t key, float b1, float b2, uint32_t *err) {
    if (nh >= LIGHT_LIST) {
        atomicOr(err, ERR_LIGHT_LIST);
        return;
    }
    int j = nh++;
    while (j > 0 && L.key[j - 1] > key) {
        L.key[j] = L.key[j - 1];
        L.b1[j] = L.b1[j - 1];
        L.b2[j] = L.b2[j - 1];
        j--;
    }
    L.key[j] = key;
    L.b1[j] = b1;
    L.b2[j] = b2;
}

// Light-hit collection.  Every crossed light counts, so the order of the walk
// is free: the walk visits inner nodes only and puts the lamps it reaches
// aside; they are tested when the warp's walks have ended (or a lane's list is
// full), and the hits of the jobs that ended take their slots with one atomic
// per warp.  (Tested where they were found, with one atomic per job, the pass
// ran 7.6 of 32 lanes per instruction.)
constexpr int LAMP_LIST = 12;  // lamps a lane puts aside; a node adds up to 4

template <bool CAPTURE, bool BATCH>
__global__ void __launch_bounds__(128, 8) k_anyhit(const __grid_constant__ FrameArgs a, uint32_t b) {
    __shared__ uint32_t s_sum[4];
    const int lane = threadIdx.x & 31;
    const int REFILL = (int)a.refill_any;
    const uint32_t n_in = a.counters[CNT_AQUEUE + b];
    uint32_t *err = a.counters + CNT_ERROR;
    const float4 *wide = a.v0.sc.lamp_wide;
    const int4 *recs = a.v0.sc.lamp_rec;
    const uint32_t *table = a.v0.sc.lamp_table;
    const float4 *tris = a.v0.sc.tri_rec;
    int root = a.v0.sc.lamp_root;
    float extent = a.v0.sc.extent;
    const float tmin = EPS_NEE, tmax = 1000.0f;
    bool has = false;
    uint32_t p = 0, idx = 0, steps = 0, n_nodes = 0, n_leaves = 0, n_hits = 0;
    f3 o = f3{0, 0, 0}, d = f3{0, 0, 0}, inv = f3{0, 0, 0}, oin = f3{0, 0, 0}, oif = f3{0, 0, 0};
    int node = EMPTY_ROOT, sp = 0, nh = 0, nl = 0;  // node < 0: the walk has ended
    int px = 0, py = 2, pz = 4;  // near-plane float4 per axis, picked by the ray's direction signs
    int stack[TRAV_STACK], lamps[LAMP_LIST];
    HitList hits;
    stamp_start(a, ST_WALK + b);
    if (blockIdx.x == 0 && threadIdx.x == 0 && n_in)
        atomicAdd(reinterpret_cast<unsigned long long *>(a.counters + CNT_ANY), (unsigned long long)n_in);
    if (threadIdx.x < 4) s_sum[threadIdx.x] = 0;
    __syncthreads();
    WarpRange range = range_first(n_in);
    while (true) {
        const uint32_t need = __ballot_sync(FULL, !has);
        if ((range.cur < range.end || range.more) && need && (__popc(need) >= REFILL || need == FULL)) {
            if (range.cur == range.end) range_next(range, n_in, &a.counters[CNT_AFETCH + b]);
            const uint32_t base = range.cur;
            range.cur = min(base + (uint32_t)__popc(need), range.end);
            if (!has) {
                idx = base + (uint32_t)__popc(need & lanemask_lt());
                if (idx < range.end) {
                    has = true;
                    p = a.aqueue[b & 1][idx];
                    if constexpr (BATCH) {
                        const ViewDev &V = view_of<BATCH>(a, p);
                        wide = V.sc.lamp_wide;
                        recs = V.sc.lamp_rec;
                        table = V.sc.lamp_table;
                        tris = V.sc.tri_rec;
                        root = V.sc.lamp_root;
                        extent = V.sc.extent;
                    }
                    float4 ro, rd;
                    ld2(a.ajob[b & 1] + 2 * (size_t)idx, ro, rd);
                    o = ld3(ro);
                    d = ld3(rd);
                    inv = f3{slab_inv(d.x), slab_inv(d.y), slab_inv(d.z)};
                    slab_offsets(o, inv, ray_margin(extent, o), oin, oif);
                    px = signbit(inv.x) ? 1 : 0;
                    py = signbit(inv.y) ? 3 : 2;
                    pz = signbit(inv.z) ? 5 : 4;
                    node = root;
                    sp = 0;
                    nh = 0;
                    nl = 0;
                    steps = 0;
                    if (root < 0 && root != EMPTY_ROOT) {  // one lamp, no inner node
                        lamps[nl++] = ~root;
                        node = EMPTY_ROOT;
                    }
                }
            }
        }
        if (!__any_sync(FULL, has)) {
            if (range.cur < range.end || range.more) continue;
            break;
        }
        while (true) {
            const bool inner = has && node >= 0 && nl <= LAMP_LIST - 4;
            if (!__any_sync(FULL, inner)) break;
            if (inner) {
                const float4 *w = wide + 8 * (size_t)node;
                const float4 NX = __ldg(w + px), FX = __ldg(w + (px ^ 1)), NY = __ldg(w + py);
                const float4 FY = __ldg(w + (py ^ 1)), NZ = __ldg(w + pz), FZ = __ldg(w + (pz ^ 1));
                const float4 RF = __ldg(w + 6);
                const int rf[4] = {__float_as_int(RF.x), __float_as_int(RF.y), __float_as_int(RF.z),
                                   __float_as_int(RF.w)};
                const float4 ax = fma4(NX, inv.x, oin.x), ay = fma4(NY, inv.y, oin.y), az = fma4(NZ, inv.z, oin.z);
                const float4 bx = fma4(FX, inv.x, oif.x), by = fma4(FY, inv.y, oif.y), bz = fma4(FZ, inv.z, oif.z);
                const float nx[4] = {ax.x, ax.y, ax.z, ax.w}, ny[4] = {ay.x, ay.y, ay.z, ay.w};
                const float nz[4] = {az.x, az.y, az.z, az.w}, fx[4] = {bx.x, bx.y, bx.z, bx.w};
                const float fy[4] = {by.x, by.y, by.z, by.w}, fz[4] = {bz.x, bz.y, bz.z, bz.w};
                int next = EMPTY_ROOT;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float tn = fmax3(nx[i], ny[i], fmaxf(nz[i], tmin));
                    const float tf = fmin3(fx[i], fy[i], fminf(fz[i], tmax));
                    if (tn <= tf) {  // (an unused slot's inverted box is never entered)
                        if (rf[i] < 0) {
                            lamps[nl++] = ~rf[i];
                        } else if (next == EMPTY_ROOT) {
                            next = rf[i];
                        } else if (sp < TRAV_STACK) {
                            stack[sp++] = rf[i];
                        } else {
                            atomicOr(err, ERR_STACK);
                        }
                    }
                }
                if (next == EMPTY_ROOT && sp > 0) next = stack[--sp];
                node = next;
                if (++steps > TRAV_GUARD) {  // only reachable with a malformed layout
                    atomicOr(err, ERR_GUARD);
                    node = EMPTY_ROOT;
                }
            }
        }
        while (has && nl > 0) {  // one lamp; each emissive face hit names one light triangle
            n_leaves++;
            const int4 r = __ldg(recs + lamps[--nl]);
            const int wx = rec_wx(r), wy = rec_wy(r), wz = rec_wz(r);
            const uint64_t ikey = (uint64_t)rec_inst(r) << 32;
            if (r.z < 0) {  // a mesh light triangle: (leaf, world-space triangle record) in the table
                const uint32_t leaf = __ldg(table + r.w), t = __ldg(table + r.w + 1);
                const float4 *q = tris + 3 * (size_t)t;
                TriHit th;
                if (tri_test(ld3(__ldg(q)), ld3(__ldg(q + 1)), ld3(__ldg(q + 2)), o, d, tmin, tmax, th))
                    hit_insert(hits, nh, ikey | leaf, th.b1, th.b2, err);
                continue;
            }
            for (uint32_t fm = (uint32_t)r.z; fm; fm &= fm - 1u) {
                const int f = __ffs(fm) - 1;
                FaceHit fh;
                if (!face_test(wx, wy, wz, f, o, d, inv, tmin, tmax, fh)) continue;
                const uint32_t leaf = __ldg(table + r.w + 2 * f + fh.half);
                if (leaf != INVALID) hit_insert(hits, nh, ikey | leaf, fh.b1, fh.b2, err);
            }
        }
        const bool done = has && node < 0;
        const uint32_t cnt = done ? (uint32_t)nh : 0u;
        const uint32_t multi = __ballot_sync(FULL, cnt > 1);
        if (__any_sync(FULL, cnt > 0)) {
            uint32_t incl = cnt;
#pragma unroll
            for (int k = 1; k < 32; k <<= 1) {
                const uint32_t up = __shfl_up_sync(FULL, incl, k);
                if (lane >= k) incl += up;
            }
            unsigned long long at = 0;
            if (lane == 31)
                at = atomicAdd(reinterpret_cast<unsigned long long *>(a.counters + CNT_HITS + 2 * b),
                               ((unsigned long long)__popc(multi) << 32) | incl);
            at = __shfl_sync(FULL, at, 31);
            const uint32_t hb = (uint32_t)at + incl - cnt;
            const bool fits = hb + cnt <= a.hit_cap;
            if (!fits) atomicOr(err, ERR_LIGHT_LIST);
            for (uint32_t j = 0; j < cnt && hb + j < a.hit_cap; j++) {
                st2(reinterpret_cast<float4 *>(a.hitbuf) + 2 * (size_t)(hb + j),
                    as_float4(make_uint4(p, (uint32_t)(hits.key[j] >> 32), (uint32_t)hits.key[j],
                                         __float_as_uint(hits.b1[j]))),
                    as_float4(make_uint4(__float_as_uint(hits.b2[j]), idx, fits ? cnt : 0u, 0u)));
            }
            // the jobs with several hits, for the sum (a job past the hit
            // buffer's end has none to sum)
            if (cnt > 1)
                a.jmeta[(uint32_t)(at >> 32) + __popc(multi & lanemask_lt())] = make_uint2(hb, fits ? cnt : 0u);
            n_hits += cnt;
        }
        if (done) {
            n_nodes += steps;
            has = false;
        }
    }
    n_nodes = __reduce_add_sync(FULL, n_nodes);
    n_leaves = __reduce_add_sync(FULL, n_leaves);
    n_hits = __reduce_add_sync(FULL, n_hits);
    publish_totals<3>(s_sum, a.counters, {CNT_ANODES, CNT_ALEAVES, CNT_AHITS}, {n_nodes, n_leaves, n_hits});
}

template <bool CAPTURE, bool BATCH>
__global__ void __launch_bounds__(128) k_hit_eval(const __grid_constant__ FrameArgs a, uint32_t b) {
    const uint32_t n = min(a.counters[CNT_HITS + 2 * b], a.hit_cap);
    for (uint32_t h = blockIdx.x * blockDim.x + threadIdx.x; h < n; h += gridDim.x * blockDim.x) {
        float4 h0, h1;
        ld2(reinterpret_cast<const float4 *>(a.hitbuf) + 2 * (size_t)h, h0, h1);
        const uint4 A = as_uint4(h0), B = as_uint4(h1);
        if (B.z == 0) continue;  // of a job that did not fit the hit buffer
        const uint32_t p = A.x;
        float4 ro, rd;
        ld2(a.ajob[b & 1] + 2 * (size_t)B.y, ro, rd);
        const DevScene &sc = view_of<BATCH>(a, p).sc;
        // the shading normal of the job's vertex: a voxel face's, or a mesh
        // triangle's, recomputed as its shading computed it
        const int fw = __float_as_int(ro.w);
        f3 n3;
        if (fw >= 0) {
            n3 = ld3(__ldg(d_faces + 2 * FACE_ROW * fw));
        } else {
            const float4 *q = sc.tri_rec + 3 * (size_t)((uint32_t)fw & 0x7FFFFFFFu);
            n3 = tri_frame(ld3(__ldg(q)), ld3(__ldg(q + 1)), ld3(__ldg(q + 2))).n;
        }
        const float v = nee_pdf_of(sc, ld3(ro), n3, ld3(rd), A.y, A.z, __uint_as_float(A.w), __uint_as_float(B.x));
        if (B.z > 1) {
            a.hitval[h] = v;
        } else {
            const float nee = 0.0f + v;  // the sum from 0 in key order
            finish_job(a, b, p, rd.w, nee);
            if (CAPTURE) a.c_nee[(size_t)b * a.P + p] = nee;
        }
    }
}

template <bool CAPTURE>
__global__ void __launch_bounds__(128) k_hit_sum(const __grid_constant__ FrameArgs a, uint32_t b) {
    const uint32_t n = a.counters[CNT_HITS + 2 * b + 1];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 m = a.jmeta[i];
        if (m.y == 0) continue;
        const uint32_t p = a.hitbuf[2 * (size_t)m.x].x, idx = a.hitbuf[2 * (size_t)m.x + 1].y;
        float nee = 0.0f;
        for (uint32_t j = 0; j < m.y; j++) nee += a.hitval[m.x + j];
        finish_job(a, b, p, a.ajob[b & 1][2 * (size_t)idx + 1].w, nee);
        if (CAPTURE) a.c_nee[(size_t)b * a.P + p] = nee;
    }
    // (of the warps that had a job, and the first)
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    if ((threadIdx.x & 31u) == 0 && (first < n || first == 0)) stamp_end(a, ST_WALKED + b);
}

}  // namespace

vrg_status upload_frames(cudaStream_t s, const float4 **table) {
    float4 t[12 * FACE_ROW] = {};
    for (int f = 0; f < 6; f++)
        for (int h = 0; h < 2; h++) {
            const Frame fr = face_frame(f, h);
            const uint32_t bits = face_corner(f, h, 0) | face_corner(f, h, 1) << 3 | face_corner(f, h, 2) << 6;
            float4 *q = t + FACE_ROW * (2 * f + h);
            q[0] = make_float4(fr.n.x, fr.n.y, fr.n.z, 0.0f);
            memcpy(&q[0].w, &bits, 4);
            q[2] = make_float4(fr.t.x, fr.t.y, fr.t.z, 0.0f);
            q[3] = make_float4(fr.b.x, fr.b.y, fr.b.z, 0.0f);
        }
    VRG_CUDA_TRY(cudaMemcpyToSymbolAsync(d_faces, t, sizeof(t), 0, cudaMemcpyHostToDevice, s));
    VRG_CUDA_TRY(cudaGetSymbolAddress((void **)table, d_faces));
    return VRG_OK;
}

static int occupancy_grid(const void *fn, int threads) {
    int dev = 0, sms = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, 0);
    return std::max(1, sms) * std::max(1, n);
}

// full-occupancy grids of the persistent bounce kernels, [single view,
// batched] (set once, before any stream capture)
static int g_trace[2] = {0, 0}, g_shade[2] = {0, 0}, g_any[2] = {0, 0};
static int g_sms = 1;
static std::once_flag g_grids_once;

static void init_grids_once() {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    g_sms = std::max(1, g_sms);
    g_shade[0] = occupancy_grid((const void *)k_shade<false, false, false, false>, 128);
    g_shade[1] = occupancy_grid((const void *)k_shade<false, true, false, false>, 128);
    g_any[0] = occupancy_grid((const void *)k_anyhit<false, false>, 128);
    g_any[1] = occupancy_grid((const void *)k_anyhit<false, true>, 128);
    g_trace[1] = occupancy_grid((const void *)k_trace<true, false>, 128);
    g_trace[0] = occupancy_grid((const void *)k_trace<false, false>, 128);
}

// (thread-safe: renderers may be created from several threads)
static void init_grids() { std::call_once(g_grids_once, init_grids_once); }

// resident CTAs per SM at full occupancy of (closest hit, shading, light
// hits), the bound of a tuned persistent grid; and the SM count
void bounce_occupancy(bool batch, int occ[3], int *sms) {
    init_grids();
    const int v = batch ? 1 : 0;
    occ[0] = std::max(1, g_trace[v] / g_sms);
    occ[1] = std::max(1, g_shade[v] / g_sms);
    occ[2] = std::max(1, g_any[v] / g_sms);
    *sms = g_sms;
}

// A bounce in two launches groups.  A batched frame (a.views set) runs the
// variants that look up each pixel's view.  max_rays > 0 bounds the rays of the
// bounce (a cache frame's training paths): the persistent grids then shrink to
// one lane per ray, leaving the other SMs to the work that runs beside them.
static void bounce_grids(const FrameArgs &a, uint32_t max_rays, int &gt, int &gs, int &ga) {
    init_grids();
    const int v = a.views ? 1 : 0;
    gt = a.grid_trace ? std::min((int)a.grid_trace, g_trace[v]) : g_trace[v];
    gs = a.grid_shade ? std::min((int)a.grid_shade, g_shade[v]) : g_shade[v];
    ga = a.grid_any ? std::min((int)a.grid_any, g_any[v]) : g_any[v];
    if (max_rays) {
        const int cap = (int)std::max<uint32_t>(1u, (max_rays + 127) / 128);
        gt = std::min(gt, cap);
        gs = std::min(gs, cap);
        ga = std::min(ga, cap);
    }
}

// the frame's counters cleared and its ray tables filled
vrg_status launch_frame_begin(cudaStream_t s, const FrameArgs &a, uint32_t max_entries) {
    const dim3 g((std::max(max_entries, (uint32_t)CNT_WORDS) + 127) / 128, a.views ? a.n_views : 1);
    if (a.views) k_frame_begin<true><<<g, 128, 0, s>>>(a);
    else k_frame_begin<false><<<g, 128, 0, s>>>(a);
    VRG_CUDA_TRY(cudaGetLastError());
    return VRG_OK;
}

// closest hit of bounce b
vrg_status launch_trace(cudaStream_t s, const FrameArgs &a, uint32_t b, uint32_t max_rays) {
    int gt, gs, ga;
    bounce_grids(a, max_rays, gt, gs, ga);
    // the mesh-capable builds only for frames whose scenes hold meshes
    if (a.views) {
        if (a.mesh) k_trace<true, true><<<gt, 128, 0, s>>>(a, b);
        else k_trace<true, false><<<gt, 128, 0, s>>>(a, b);
    } else if (a.mesh) {
        k_trace<false, true><<<gt, 128, 0, s>>>(a, b);
    } else {
        k_trace<false, false><<<gt, 128, 0, s>>>(a, b);
    }
    VRG_CUDA_TRY(cudaGetLastError());
    return VRG_OK;
}

template <bool CAPTURE, bool BATCH, bool MESH>
static void shade_launch(int gs, cudaStream_t s, const FrameArgs &a, uint32_t b, bool split) {
    if (split) k_shade<CAPTURE, BATCH, MESH, true><<<gs, 128, 0, s>>>(a, b);
    else k_shade<CAPTURE, BATCH, MESH, false><<<gs, 128, 0, s>>>(a, b);
}

// shading of bounce b
vrg_status launch_shade(cudaStream_t s, const FrameArgs &a, uint32_t b, uint32_t max_rays) {
    int gt, gs, ga;
    bounce_grids(a, max_rays, gt, gs, ga);
    // (not for the few rays of a cache frame's training bounces, bounded by
    // max_rays: batches of 128 per warp would leave most of the grid idle)
    const bool split = shade_split(a, b) && max_rays == 0;
    if (a.mesh) {
        if (a.views) shade_launch<false, true, true>(gs, s, a, b, split);
        else if (a.capture) shade_launch<true, false, true>(gs, s, a, b, split);
        else shade_launch<false, false, true>(gs, s, a, b, split);
    } else {
        if (a.views) shade_launch<false, true, false>(gs, s, a, b, split);
        else if (a.capture) shade_launch<true, false, false>(gs, s, a, b, split);
        else shade_launch<false, false, false>(gs, s, a, b, split);
    }
    VRG_CUDA_TRY(cudaGetLastError());
    return VRG_OK;
}

// closest hit and shading of bounce b
vrg_status launch_trace_shade(cudaStream_t s, const FrameArgs &a, uint32_t b, uint32_t max_rays) {
    if (a.views && a.capture) {
        set_error("capture is not available for batched frames");
        return VRG_ERR_UNSUPPORTED;
    }
    VRG_TRY(launch_trace(s, a, b, max_rays));
    return launch_shade(s, a, b, max_rays);
}

// the light-pdf walk of bounce b's jobs (bounces before the last): it reads only
// the jobs' own ray copies, so it may run beside bounce b + 1
vrg_status launch_light_pdf(cudaStream_t s, const FrameArgs &a, uint32_t b, uint32_t max_rays) {
    if (b + 1 >= a.nb) return VRG_OK;
    const bool batch = a.views != nullptr;
    int gt, gs, ga;
    bounce_grids(a, max_rays, gt, gs, ga);
    if (batch) k_anyhit<false, true><<<ga, 128, 0, s>>>(a, b);
    else if (a.capture) k_anyhit<true, false><<<ga, 128, 0, s>>>(a, b);
    else k_anyhit<false, false><<<ga, 128, 0, s>>>(a, b);
    if (batch) k_hit_eval<false, true><<<gs, 128, 0, s>>>(a, b);
    else if (a.capture) k_hit_eval<true, false><<<gs, 128, 0, s>>>(a, b);
    else k_hit_eval<false, false><<<gs, 128, 0, s>>>(a, b);
    if (a.capture) k_hit_sum<true><<<gs, 128, 0, s>>>(a, b);
    else k_hit_sum<false><<<gs, 128, 0, s>>>(a, b);
    VRG_CUDA_TRY(cudaGetLastError());
    return VRG_OK;
}

}  // namespace vrg
