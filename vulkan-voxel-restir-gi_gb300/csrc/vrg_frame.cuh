// Per-frame kernel arguments shared by the wavefront stages.
#pragma once

#include "vrg_device.cuh"

namespace vrg {

// counters[] layout (u32 words)
constexpr int CNT_QUEUE = 0;     // [0..7]  rays queued for bounce b
constexpr int CNT_FETCH = 8;     // [8..15] closest-hit work-fetch cursor of bounce b
constexpr int CNT_ERROR = 16;    // error word
constexpr int CNT_RAYS = 18;     // u64 at words 18-19: closest-hit queries
constexpr int CNT_TQUEUE = 22;   // a cache frame's training candidates queued for its query bounce (FrameArgs::tq)
constexpr int CNT_TFETCH = 23;   // their closest-hit work-fetch cursor
constexpr int CNT_ANY = 20;      // u64 at words 20-21: light any-hit queries
constexpr int CNT_AQUEUE = 24;   // [24..31] any-hit jobs queued by bounce b
constexpr int CNT_AFETCH = 32;   // [32..39] any-hit work-fetch cursor of bounce b
constexpr int CNT_NODES = 50;    // u64 at words 50-51: inner nodes fetched by k_trace
constexpr int CNT_LEAVES = 52;   // u64 at words 52-53: leaf records tested by k_trace
constexpr int CNT_HITS = 64;     // [64..79] per bounce b, one u64: light hits collected by k_anyhit (word 64 + 2b)
                                 // and jobs with several (word 65 + 2b)
constexpr int CNT_ANODES = 56;   // u64 at words 56-57: 4-wide lamp nodes fetched by k_anyhit
constexpr int CNT_ALEAVES = 58;  // u64 at words 58-59: lamp-block records tested by k_anyhit
constexpr int CNT_AHITS = 60;    // u64 at words 60-61: light hits collected by k_anyhit
constexpr int CNT_INFER = 48;    // radiance-cache queries of the frame
constexpr int CNT_TRAIN = 49;    // radiance-cache training paths of the frame
constexpr int MAX_BOUNCES = 8;
// A vertex's normal in one word: 2 * face + half of a voxel face, bit 31 | its
// record of a mesh triangle, or NORMAL_NONE (a miss).  (The two halves' normals
// differ in the sign of zeros.)
constexpr int NORMAL_NONE = 12;
constexpr int FACE_ROW = 4;

// The frame's stage times, written by its kernels: u64 nanoseconds of the
// device's global timer from word CNT_STAMP on (0: the stage did not run).
// Starts are written by a kernel's first thread, ends are the latest of its
// CTAs (of its warps that had work in the shading and k_hit_sum; 0 for the
// shading of an empty queue).  About 20 timing events between the stages held
// the frame up: with these times in their place a 64x64 frame with stats went
// from 129 to 106 us, a 640x480 one from 287 to 260.
constexpr int CNT_STAMP = 80;
constexpr int ST_BEGIN = 0;                        // the frame (start)
constexpr int ST_SPATIAL = 1;                      // spatial (start)
constexpr int ST_TRACED = 2;                       // + b: closest hit of bounce b (end)
constexpr int ST_SHADED = ST_TRACED + MAX_BOUNCES; // + b: its shading (end)
constexpr int ST_WALK = ST_SHADED + MAX_BOUNCES;   // + b: its light-pdf walk (start)
constexpr int ST_WALKED = ST_WALK + MAX_BOUNCES;   // + b: its light-pdf walk (end)
constexpr int ST_COUNT = ST_WALKED + MAX_BOUNCES;
constexpr int CNT_WORDS = CNT_STAMP + 2 * ST_COUNT;

// One camera view of one scene.  A frame renders either one view (the
// FrameArgs::v0 fields, passed as kernel parameters) or a batch of views whose
// pixels are numbered view after view in one pixel space (FrameArgs::views in
// device memory, so that a captured launch sequence reads each frame's
// cameras, seeds and scenes from there).  Pixel streams and reservoir
// neighbourhoods use the view-local pixel index p - pix_off, so a view renders
// the same image alone or inside a batch.
struct ViewDev {
    DevScene sc;
    f3 eye, front, right, up;
    uint32_t W, H, pix_off, pix_end;
    uint32_t frame, temporal_seed, spatial_seed;
    uint32_t w_magic;             // div_magic(W)
    // the primary rays' direction terms of the frame's camera per column and
    // per row (k_frame_begin): d = normalize((ray_x[x] + ray_y[y]) + front)
    float4 *ray_x, *ray_y;
    // its 8x4-pixel tiles: [tile_off, tile_end) of the frame's tiles, tiles_x per row
    uint32_t tile_off, tile_end, tiles_x, tile_magic;  // tile_magic: div_magic(tiles_x)
};

// n / d and n % d for any 32-bit n by one high product and a correction, with
// m = floor(2^32 / d) from the host (the quotient is short by at most 1; cf.
// Granlund and Montgomery, PLDI 1994): 5 instructions, an integer division
// with its remainder about 25.
inline uint32_t div_magic(uint32_t d) { return d <= 1 ? 0xFFFFFFFFu : (uint32_t)((1ull << 32) / d); }
__host__ __device__ __forceinline__ void div_mod(uint32_t n, uint32_t d, uint32_t m, uint32_t &q, uint32_t &rem) {
    q = (uint32_t)(((uint64_t)n * m) >> 32);
    rem = n - q * d;
    if (rem >= d) {
        q++;
        rem -= d;
    }
}

constexpr int TILE_SHIFT = 3;  // ttab entry per 8 tiles: the view of the group's first tile
constexpr int VIEW_SHIFT = 8;  // vtab entry per 256 pixels: the view of the group's first pixel

struct FrameArgs {
    ViewDev v0;                   // the view of a single-view frame
    const ViewDev *views;         // batched frame: the views (device), else null
    const uint16_t *vtab;         // batched frame: view of pixel group p >> VIEW_SHIFT
    uint32_t n_views;
    uint32_t mesh;                // a scene of the frame holds mesh triangles (the bounce kernels
                                  // built with mesh support run; voxel-only frames run without it)
    uint32_t P;                   // pixels of the frame (all views)
    uint32_t n0;                  // bounce-0 slots: 32 per 8x4-pixel tile (bounce0_pixel)
    const uint16_t *ttab;         // batched frame: view of tile group t >> TILE_SHIFT
    uint32_t nb, nee_type;
    uint32_t mode, spatial_iters;
    float spatial_radius;
    uint32_t m_cap, debug_view, accumulate, pack;
    // launch configuration (scheduling only, never a result): idle lanes that
    // trigger a warp's refill, persistent grids (CTAs), per-pixel CTA size
    uint32_t refill_trace, refill_any;
    // supersampling (Renderer.scale): the frame is traced at scale x the
    // output extent; k_downsample packs out_w x out_h pixels
    uint32_t scale, out_w, out_h;
    uint8_t *out_bgra;
    float *out_radiance;
    uint32_t grid_trace, grid_shade, grid_any, stream_block;
    // wavefront state
    float4 *ray;                  // [P][2]: (origin, face), (direction, bsdf pdf)
    uint32_t *queue[2];
    // A single-view cache frame traces its query bounce in two launches: the
    // training candidates (one pixel in 16) first, so that the training
    // branch forks early, then the other paths.  tq_split: the shading of the
    // bounce before the query bounce queues the candidates' rays in tq
    // (CNT_TQUEUE) instead of queue[]; qsel: this launch of the query bounce
    // takes its rays from tq.
    uint32_t *tq;
    uint32_t tq_split, qsel;
    uint32_t timed;               // the kernels write the stage times (CNT_STAMP)
    // light-pdf jobs of bounce b in [b & 1] (double-buffered by bounce parity:
    // the jobs of bounce b are walked while bounce b + 1 traces and shades):
    // the pixel, and a copy of its ray (origin | face, direction | bsdf pdf)
    uint32_t *aqueue[2];
    float4 *ajob[2];              // 2 float4 per job
    uint4 *hitbuf;                // light hits: (pixel, instance, leaf, b1 bits), then (b2 bits, job, the job's hits, 0)
    float *hitval;                // light-sampling pdf of each hit
    uint2 *jmeta;                 // per any-hit job with several hits: (first hit, hit count)
    uint32_t hit_cap;
    int4 *hits;                   // closest hit per pixel: (~record or -1, face|half<<3, b1, b2)
    uint32_t *counters;
    uint8_t *nlive;
    float4 *rec;                  // [nb][P][2]: (E.xyz, w), (R.xyz, q)
    float4 *xv, *xs;              // the first two vertices: position, normal word
    const float4 *faces;          // face frames: FACE_ROW float4 per 2 * face + half, the normal first
    float4 *plain;                // L[0], for the views that show it (debug_view 0)
    float4 *res;                  // temporal ring slot (res_pair in restir.cu)
    float4 *spatial;              // likewise (written when capture)
    float4 *final_t;              // [P] (written when capture)
    uint8_t *bgra;
    float *radiance;
    double *accum;
    // radiance cache (VRG_RENDER_CACHE): paths end into the cache after
    // nb_render bounces; 1/16 of them (up to train_cap) trace to nb and train it
    uint32_t nb_render, cache, train_cap, restir;  // restir: reservoirs (two bounces or more)
    float4 *q_pos, *q_dir, *pred, *target;
    uint32_t *infer_list, *train_list;
    uint8_t *qflag;
    // capture (reference SoA layout, for parity readback)
    uint32_t capture;
    float *c_origin, *c_dir, *c_normal, *c_emis, *c_refl, *c_mis, *c_pdf, *c_nee, *c_L, *c_q;
    uint32_t *c_hit;
};

#ifdef __CUDACC__
// Two float4 at a 32-byte boundary in one access.  The stages are bound by the
// requests they put to the L1 and by the sectors they touch: a path's ray, its
// record, a job and a hit are one sector and one request each.  (As pairs of
// arrays or of 16-byte accesses: 1080p in flight 837 us, not 829, with 8 bounces
// 1776, not 1724; 3840x2160 4854, not 4792.)
__device__ __forceinline__ void ld2(const float4 *p, float4 &a, float4 &b) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}
// (of data no kernel running beside writes)
__device__ __forceinline__ void ldg2(const float4 *p, float4 &a, float4 &b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}
__device__ __forceinline__ uint4 as_uint4(float4 v) {
    return make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
}
__device__ __forceinline__ float4 as_float4(uint4 v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ void st2(float4 *p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
// (frames without stats write no times: with them, mostly by the ends'
// atomics, 1080p frames in flight took 871 us, not 867)
__device__ __forceinline__ unsigned long long *stamp_at(const FrameArgs &a, uint32_t stage) {
    return reinterpret_cast<unsigned long long *>(a.counters + CNT_STAMP) + stage;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// the kernel's first thread: its start
__device__ __forceinline__ void stamp_start(const FrameArgs &a, uint32_t stage) {
    if (a.timed && blockIdx.x == 0 && threadIdx.x == 0) *stamp_at(a, stage) = global_ns();
}
// one thread of each CTA: its end
__device__ __forceinline__ void stamp_end(const FrameArgs &a, uint32_t stage) {
    if (a.timed) atomicMax(stamp_at(a, stage), global_ns());
}
#endif

// The view that owns pixel p of the frame.
template <bool BATCH>
__device__ __forceinline__ const ViewDev &view_of(const FrameArgs &a, uint32_t p) {
    if constexpr (BATCH) {
        uint32_t v = a.vtab[p >> VIEW_SHIFT];
        while (p >= a.views[v].pix_end) v++;  // views smaller than a pixel group
        return a.views[v];
    } else {
        (void)p;
        return a.v0;
    }
}

// The view that owns tile t of the frame.
template <bool BATCH>
__device__ __forceinline__ const ViewDev &view_of_tile(const FrameArgs &a, uint32_t t) {
    if constexpr (BATCH) {
        uint32_t v = a.ttab[t >> TILE_SHIFT];
        while (t >= a.views[v].tile_end) v++;
        return a.views[v];
    } else {
        (void)t;
        return a.v0;
    }
}

// Bounce 0 takes a view's pixels in 8x4 tiles, so that a warp's primary rays,
// and through the queue order the secondary rays they spawn, start close
// together.  Slot i (< n0) of view V is pixel p = (x, y), or no pixel in the
// part of an edge tile outside the view.
__device__ __forceinline__ bool bounce0_pixel(const ViewDev &V, uint32_t i, uint32_t &p, uint32_t &x, uint32_t &y) {
    const uint32_t t = (i >> 5) - V.tile_off, k = i & 31u;
    uint32_t tx, ty;
    div_mod(t, V.tiles_x, V.tile_magic, ty, tx);
    x = tx * 8u + (k & 7u);
    y = ty * 4u + (k >> 3);
    p = V.pix_off + y * V.W + x;
    return x < V.W && y < V.H;
}

}  // namespace vrg
