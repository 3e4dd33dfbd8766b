// GPU chunk meshing and light-primitive extraction, batched over chunks.
//
// Replaces, per chunk, the reference's CPU pipeline chunk::gen_mesh
// (chunk.rs:158-292) -> SceneUploader::upload_object (scene.rs:547-725) ->
// build_bl_bvh (build.rs:249-372): a face of a non-air block is exposed when
// the neighbouring block (inside the chunk or in the neighbour chunk's
// boundary plane) is air or translucent; exposed faces become two triangles
// each, numbered in gen_mesh's scan order (x, y, z, then faces left, right,
// down, up, back, front); a triangle is a light when its face material has
// luminance > 0, with power luminance * area.  The geometry primitives are
// the surface blocks (>= 1 exposed face) with AABB [x, x+1]^3.
//
// One CTA of 1024 threads per chunk; thread t owns the 32 consecutive block
// indices 32t..32t+31 (x = t/32, y = t%32, z = 0..31), so a CTA-wide
// exclusive scan of per-thread counts gives gen_mesh's numbering directly.
#include "vrg_internal.h"

namespace vrg {

namespace {

constexpr int CHUNK_BYTES = VRG_CHUNK_BLOCKS + 6 * 1024;  // blocks + 6 neighbour planes

// Masks of a chunk's rows: a row is the 32 blocks z = 0..31 of (x, y), one
// thread's share, and its masks are 32-bit words with bit z.
struct ExtractArgs {
    const uint8_t *in;           // [n_chunks][CHUNK_BYTES]
    uint32_t *rows;              // [n_chunks][6][1024]: exposed faces f of row x * 32 + y
    uint32_t *counts;            // [n_chunks][4]: faces, light faces, surface blocks, lamp blocks
    const vrg_material *mats;
    uint32_t air;
};

// which of a row's 32 blocks (16-byte aligned) are translucent (air is), and
// which are air; tbits: the translucent block ids
__device__ __forceinline__ uint32_t row_translucent(const uint8_t *row, const uint32_t *tbits, uint32_t air,
                                                    uint32_t *is_air) {
    const uint4 a = *reinterpret_cast<const uint4 *>(row), b = *reinterpret_cast<const uint4 *>(row + 16);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t t = 0, e = 0;
#pragma unroll
    for (int z = 0; z < 32; z++) {
        const uint32_t id = (w[z >> 2] >> (8 * (z & 3))) & 255u;
        t |= ((tbits[id >> 5] >> (id & 31u)) & 1u) << z;
        e |= (id == air ? 1u : 0u) << z;
    }
    if (is_air) *is_air = e;
    return t;
}

__device__ __forceinline__ uint32_t block_reduce_add(uint32_t v, uint32_t *sh) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    uint32_t r = 0;
    if (w == 0) {
        r = sh[lane];
        for (int o = 16; o; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (lane == 0) sh[32] = r;
    }
    __syncthreads();
    r = sh[32];
    __syncthreads();
    return r;
}

// exclusive scan over the 1024 threads of the CTA
__device__ __forceinline__ uint32_t block_exscan(uint32_t v, uint32_t *sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t s = sh[lane];
        uint32_t si = s;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, si, o);
            if (lane >= o) si += t;
        }
        sh[lane] = si - s;  // exclusive warp offsets
    }
    __syncthreads();
    uint32_t r = sh[w] + inc - v;
    __syncthreads();
    return r;
}

// The exposed faces (chunk.rs:170-205) of a chunk, a thread per row: a face is
// exposed when the block across it is translucent, so a row's faces are word
// operations on its own and its four neighbour rows' translucency masks, and
// shifts of its own along z.  (Block by block, with six byte loads each, the
// kernel took 54 us for one chunk, the latency of its loads; now 13.)
__global__ void __launch_bounds__(1024) k_extract_masks(ExtractArgs a) {
    __shared__ uint32_t sh[33], s_tbits[8], s_rows[1024];
    __shared__ uint8_t s_lum[256];  // per block id: its luminous faces
    const uint8_t *in = a.in + (size_t)blockIdx.x * CHUNK_BYTES;
    const uint8_t *slabs = in + VRG_CHUNK_BLOCKS;
    uint32_t *rows = a.rows + (size_t)blockIdx.x * 6 * 1024;
    const int t = threadIdx.x, x = t >> 5, y = t & 31;
    if (t < 256) {
        const bool known = (uint32_t)t < a.air;
        const uint32_t m = __ballot_sync(0xffffffffu, (uint32_t)t == a.air ||
                                                          (known && (a.mats[6u * t].flags & VRG_MAT_TRANSLUCENT)));
        if ((t & 31) == 0) s_tbits[t >> 5] = m;
        uint32_t l = 0;
        if (known)
            for (uint32_t f = 0; f < 6; f++) l |= (a.mats[6u * t + f].luminance > 0.0f ? 1u : 0u) << f;
        s_lum[t] = (uint8_t)l;
    }
    __syncthreads();
    uint32_t air = 0;
    const uint32_t own = row_translucent(in + t * 32, s_tbits, a.air, &air);
    s_rows[t] = own;
    __syncthreads();
    const uint32_t back = slabs[4 * 1024 + t], front = slabs[5 * 1024 + t];
    uint32_t m[6];
    m[0] = x == 0 ? row_translucent(slabs + y * 32, s_tbits, a.air, nullptr) : s_rows[t - 32];
    m[1] = x == 31 ? row_translucent(slabs + 1024 + y * 32, s_tbits, a.air, nullptr) : s_rows[t + 32];
    m[2] = y == 0 ? row_translucent(slabs + 2 * 1024 + x * 32, s_tbits, a.air, nullptr) : s_rows[t - 1];
    m[3] = y == 31 ? row_translucent(slabs + 3 * 1024 + x * 32, s_tbits, a.air, nullptr) : s_rows[t + 1];
    m[4] = (own << 1) | ((s_tbits[back >> 5] >> (back & 31u)) & 1u);
    m[5] = (own >> 1) | (((s_tbits[front >> 5] >> (front & 31u)) & 1u) << 31);
    uint32_t any = 0, faces = 0, lfaces = 0, lamps = 0;
#pragma unroll
    for (int f = 0; f < 6; f++) {
        m[f] &= ~air;
        rows[f * 1024 + t] = m[f];
        any |= m[f];
        faces += __popc(m[f]);
    }
    for (uint32_t s = any; s; s &= s - 1u) {
        const int z = __ffs(s) - 1;
        uint32_t l = s_lum[in[t * 32 + z]];
#pragma unroll
        for (int f = 0; f < 6; f++) l &= ~((~m[f] >> z & 1u) << f);
        lfaces += __popc(l);
        lamps += l ? 1u : 0u;
    }
    const uint32_t F = block_reduce_add(faces, sh);
    const uint32_t Lf = block_reduce_add(lfaces, sh);
    const uint32_t S = block_reduce_add(__popc(any), sh);
    const uint32_t Lb = block_reduce_add(lamps, sh);
    if (t == 0) {
        a.counts[4 * blockIdx.x + 0] = F;
        a.counts[4 * blockIdx.x + 1] = Lf;
        a.counts[4 * blockIdx.x + 2] = S;
        a.counts[4 * blockIdx.x + 3] = Lb;
    }
}

struct WriteArgs {
    const uint8_t *in;
    const uint32_t *rows;
    const vrg_material *mats;
    uint32_t air;
    const uint32_t *geo_off;     // [n_chunks] prim offset of the chunk's geometry prims
    const uint32_t *light_off;   // [n_chunks] prim offset of the chunk's light prims
    const uint32_t *loc_off;     // [n_chunks] offset into geo_local / light_tri
    const uint32_t *lloc_off;
    // builder inputs
    float4 *lo, *hi, *cen;
    uint32_t *id;
    // persistent per-object outputs
    int2 *geo_local;
    uint32_t *light_tri;
};

__global__ void __launch_bounds__(1024) k_extract_write(WriteArgs a) {
    __shared__ uint32_t sh[33];
    const uint32_t c = blockIdx.x;
    const uint8_t *in = a.in + (size_t)c * CHUNK_BYTES;
    const int t = threadIdx.x;
    uint32_t row[6], any = 0, faces = 0, lfaces = 0;
    for (int f = 0; f < 6; f++) {
        row[f] = a.rows[((size_t)c * 6 + f) * 1024 + t];
        any |= row[f];
        faces += __popc(row[f]);
    }
    auto mask_at = [&](int z) {
        uint32_t m = 0;
#pragma unroll
        for (int f = 0; f < 6; f++) m |= ((row[f] >> z) & 1u) << f;
        return m;
    };
    for (uint32_t s = any; s; s &= s - 1u) {
        const int z = __ffs(s) - 1;
        const uint32_t b = in[t * 32 + z];
        for (uint32_t m = mask_at(z); m; m &= m - 1u)
            if (a.mats[6u * b + (uint32_t)__ffs(m) - 1u].luminance > 0.0f) lfaces++;
    }
    uint32_t face_base = block_exscan(faces, sh);
    uint32_t lface_base = block_exscan(lfaces, sh);
    uint32_t surf_base = block_exscan(__popc(any), sh);
    const int x = t >> 5, y = t & 31;
    const uint32_t goff = a.geo_off[c], loff = a.light_off[c], gl = a.loc_off[c], ll = a.lloc_off[c];
    for (uint32_t s = any; s; s &= s - 1u) {
        const int z = __ffs(s) - 1;
        const uint32_t bi = (uint32_t)(t * 32 + z), m = mask_at(z), b = in[bi];
        uint32_t first_tri = 2u * face_base;
        // geometry prim: block AABB, centroid (min+max)/2 (build.rs:391-400)
        {
            uint32_t g = goff + surf_base;
            float lx = (float)x, ly = (float)y, lz = (float)z;
            float hx = (float)(x + 1), hy = (float)(y + 1), hz = (float)(z + 1);
            a.lo[g] = make_float4(lx, ly, lz, 0.0f);
            a.hi[g] = make_float4(hx, hy, hz, 0.0f);
            a.cen[g] = make_float4((lx + hx) / 2.0f, (ly + hy) / 2.0f, (lz + hz) / 2.0f, 0.0f);
            a.id[g] = bi;
            a.geo_local[gl + surf_base] = make_int2((int)(bi | (m << 15) | (b << 21)), (int)first_tri);
        }
        uint32_t rank = 0;
        for (int f = 0; f < 6; f++) {
            if (!((m >> f) & 1u)) continue;
            float L = a.mats[6u * b + (uint32_t)f].luminance;
            if (L > 0.0f) {
                for (int h = 0; h < 2; h++) {
                    uint32_t lp = 2u * lface_base + (uint32_t)h;
                    uint32_t g = loff + lp;
                    f3 v0 = corner_pos(x, y, z, face_corner(f, h, 0));
                    f3 v1 = corner_pos(x, y, z, face_corner(f, h, 1));
                    f3 v2 = corner_pos(x, y, z, face_corner(f, h, 2));
                    // Aabb::from_points (aabb.rs:10-22)
                    float mnx = fminf(fminf(fminf(v0.x, v0.x), v1.x), v2.x);
                    float mny = fminf(fminf(fminf(v0.y, v0.y), v1.y), v2.y);
                    float mnz = fminf(fminf(fminf(v0.z, v0.z), v1.z), v2.z);
                    float mxx = fmaxf(fmaxf(fmaxf(v0.x, v0.x), v1.x), v2.x);
                    float mxy = fmaxf(fmaxf(fmaxf(v0.y, v0.y), v1.y), v2.y);
                    float mxz = fmaxf(fmaxf(fmaxf(v0.z, v0.z), v1.z), v2.z);
                    // centroid (v0+v1+v2)/3 (build.rs:267-270); power = lum*area (scene.rs:560-571)
                    f3 s = add3(add3(v0, v1), v2);
                    float area = len3(cross3(sub3(v1, v0), sub3(v2, v0))) / 2.0f;
                    a.lo[g] = make_float4(mnx, mny, mnz, 0.0f);
                    a.hi[g] = make_float4(mxx, mxy, mxz, 0.0f);
                    a.cen[g] = make_float4(s.x / 3.0f, s.y / 3.0f, s.z / 3.0f, L * area);
                    a.id[g] = first_tri + 2u * rank + (uint32_t)h;
                    a.light_tri[ll + lp] = (uint32_t)x | ((uint32_t)y << 5) | ((uint32_t)z << 10) |
                                           ((uint32_t)f << 15) | ((uint32_t)h << 18);
                }
                lface_base++;
            }
            rank++;
        }
        face_base += __popc(m);
        surf_base++;
    }
}

// A chunk's trees in the flush's arrays: nodes (INVALID: none) and first prims
// of its geometry and light trees, light nodes, and its light_tri offset.
struct ChunkTrees {
    uint32_t node_off[2], prim_off[2], n_light_nodes, light_off, payload_off, pad;
};
// What the host keeps of a tree's root (build_bl_bvh return convention,
// build.rs:359-371): of a leaf root, its prim's own bounds and power.
struct RootSummary {
    float lo[3], hi[3], power;
};

// per light node: the triangle of the leaf's prim; blockIdx.y is the chunk,
// whose first two threads also sum up its roots
__global__ void __launch_bounds__(256) k_chunk_finish(const ChunkTrees *trees, const vrg_bvh_node *nodes,
                                                      const uint32_t *leaf_prim, const uint32_t *light_tri,
                                                      SahInputs in, uint32_t *payload, RootSummary *roots) {
    const ChunkTrees C = trees[blockIdx.y];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < C.n_light_nodes) {
        const uint32_t p = leaf_prim[C.node_off[1] + i];
        payload[C.payload_off + i] = (p == INVALID) ? INVALID : light_tri[C.light_off + p];
    }
    if (i < 2 && C.node_off[i] != INVALID) {
        const vrg_bvh_node n = nodes[C.node_off[i]];
        RootSummary r;
        if (n.left_node_idx == INVALID) {
            const float4 l = in.lo[C.prim_off[i]], h = in.hi[C.prim_off[i]];
            r = RootSummary{{l.x, l.y, l.z}, {h.x, h.y, h.z}, in.cen[C.prim_off[i]].w};
        } else {
            r = RootSummary{{n.min[0], n.min[1], n.min[2]}, {n.max[0], n.max[1], n.max[2]}, n.power};
        }
        roots[2 * blockIdx.y + i] = r;
    }
}

}  // namespace

vrg_status extract_and_build(Context *ctx, std::vector<Object *> &batch) {
    if (batch.empty()) return VRG_OK;
    cudaStream_t s = ctx->stream;
    const uint32_t nc = (uint32_t)batch.size();
    if (nc > 65535) {
        set_error("too many chunks in one flush (%u)", nc);
        return VRG_ERR_UNSUPPORTED;
    }
    // stage blocks + neighbour planes; the same page-locked buffer takes the
    // counts, the trees' places and the roots (all copies in and out of one
    // flush, ended by its last synchronization)
    const size_t in_bytes = (size_t)nc * CHUNK_BYTES, cnt_bytes = 16 * (size_t)nc;
    const size_t plan_bytes = nc * (16 + sizeof(ChunkTrees)), out_bytes = 2 * nc * sizeof(RootSummary) + 16;
    const size_t stage_bytes = in_bytes + cnt_bytes + plan_bytes + out_bytes;
    struct Pinned {
        cudaStream_t s;
        uint8_t *alloc(size_t n) {
            void *p = nullptr;
            if (cudaMallocHost(&p, n) == cudaSuccess) return (uint8_t *)p;
            cudaGetLastError();
            return nullptr;
        }
        void release(uint8_t *p) { cudaFreeHost(p); }
        void wait() { cudaStreamSynchronize(s); }
    };
    std::vector<SahTree> trees;  // (copied from here until the last synchronization: outlives the lease)
    StagingLease<Pinned> lease(ctx->stage, Pinned{s}, Context::STAGE_KEEP);
    uint8_t *h_in = lease.take(stage_bytes);
    if (!h_in) {
        set_error("%zu bytes of page-locked staging are not to be had", stage_bytes);
        return VRG_ERR_CUDA;
    }
    for (uint32_t c = 0; c < nc; c++) {
        memcpy(h_in + (size_t)c * CHUNK_BYTES, batch[c]->blocks.data(), VRG_CHUNK_BLOCKS);
        memcpy(h_in + (size_t)c * CHUNK_BYTES + VRG_CHUNK_BLOCKS, batch[c]->slabs.data(), 6 * 1024);
    }
    DevBufPtr tmp;
    VRG_TRY(dev_alloc(ctx, in_bytes + (size_t)nc * 6 * 1024 * 4 + cnt_bytes, tmp));
    uint8_t *d_in = (uint8_t *)tmp->ptr;
    uint32_t *d_rows = (uint32_t *)(d_in + in_bytes);
    uint32_t *d_counts = d_rows + (size_t)nc * 6 * 1024;
    VRG_CUDA_TRY(cudaMemcpyAsync(d_in, h_in, in_bytes, cudaMemcpyHostToDevice, s));
    ExtractArgs ea{d_in, d_rows, d_counts, (const vrg_material *)ctx->d_mats->ptr, ctx->n_types};
    k_extract_masks<<<nc, 1024, 0, s>>>(ea);
    VRG_CUDA_TRY(cudaGetLastError());
    uint32_t *h_counts = (uint32_t *)(h_in + in_bytes);
    VRG_CUDA_TRY(cudaMemcpyAsync(h_counts, d_counts, cnt_bytes, cudaMemcpyDeviceToHost, s));
    VRG_CUDA_TRY(cudaStreamSynchronize(s));

    // layout of the batch: persistent arrays per object + builder inputs (temp)
    uint64_t tot_geo = 0, tot_light = 0, tot_geo_nodes = 0, tot_light_nodes = 0;
    std::vector<uint32_t> geo_off(nc), light_off(nc);
    for (uint32_t c = 0; c < nc; c++) {
        uint32_t F = h_counts[4 * c], Lf = h_counts[4 * c + 1], S = h_counts[4 * c + 2];
        ChunkSummary &cs = batch[c]->sum;
        memset(&cs, 0, sizeof(cs));
        cs.n_faces = F;
        cs.n_tris = 2 * F;
        cs.n_light = 2 * Lf;
        cs.n_geo = S;
        cs.n_lamps = h_counts[4 * c + 3];
        geo_off[c] = (uint32_t)tot_geo;
        light_off[c] = (uint32_t)tot_light;
        tot_geo += S;
        tot_light += 2 * Lf;
        if (S) tot_geo_nodes += 2 * (uint64_t)S - 1;
        if (Lf) tot_light_nodes += 4 * (uint64_t)Lf - 1;
    }
    if (tot_geo + tot_light > 0x7FFFFFFFull) {
        set_error("flush too large");
        return VRG_ERR_UNSUPPORTED;
    }
    const uint64_t n_prims = tot_geo + tot_light;
    const uint64_t n_nodes = tot_geo_nodes + tot_light_nodes;
    auto al = [](uint64_t x) { return (x + 255) & ~255ull; };
    uint64_t o = 0;
    uint64_t o_geo_local = o; o += al(tot_geo * 8);
    uint64_t o_light_tri = o; o += al(tot_light * 4);
    uint64_t o_nodes = o; o += al(n_nodes * sizeof(vrg_bvh_node));
    uint64_t o_perm = o; o += al(n_prims * 4);
    uint64_t o_leaf = o; o += al(n_nodes * 4);
    uint64_t o_payload = o; o += al(tot_light_nodes * 4);
    uint64_t persist_bytes = o;
    DevBufPtr batch_buf;
    VRG_TRY(dev_alloc(ctx, std::max<uint64_t>(persist_bytes, 256), batch_buf));
    uint8_t *B = (uint8_t *)batch_buf->ptr;
    DevBufPtr bin;
    uint64_t ob = 0;
    uint64_t o_lo = ob; ob += al(n_prims * 16);
    uint64_t o_hi = ob; ob += al(n_prims * 16);
    uint64_t o_cen = ob; ob += al(n_prims * 16);
    uint64_t o_id = ob; ob += al(n_prims * 4);
    uint64_t o_plan = ob; ob += al(plan_bytes);
    uint64_t o_out = ob; ob += al(out_bytes);
    VRG_TRY(dev_alloc(ctx, std::max<uint64_t>(ob, 256), bin));
    uint8_t *I = (uint8_t *)bin->ptr;
    // Prim index space: geometry prims first, then light prims.  One batched
    // SAH build: geometry trees (build_tl_bvh semantics over block AABBs) and
    // light trees (build_bl_bvh over light triangles).
    uint32_t *offs = (uint32_t *)(h_in + in_bytes + cnt_bytes);
    ChunkTrees *ct = (ChunkTrees *)(offs + 4 * (size_t)nc);
    uint64_t node_cursor = 0;
    uint32_t max_light_nodes = 0;
    for (int k = 0; k < 2; k++)
        for (uint32_t c = 0; c < nc; c++) {
            const ChunkSummary &cs = batch[c]->sum;
            const uint32_t n = k ? cs.n_light : cs.n_geo, first = k ? (uint32_t)tot_geo + light_off[c] : geo_off[c];
            ct[c].node_off[k] = n ? (uint32_t)node_cursor : INVALID;
            ct[c].prim_off[k] = first;
            if (k) {
                ct[c].n_light_nodes = n ? 2 * n - 1 : 0;
                ct[c].light_off = light_off[c];
                ct[c].payload_off = (uint32_t)(node_cursor - tot_geo_nodes);
                ct[c].pad = 0;
                max_light_nodes = std::max(max_light_nodes, ct[c].n_light_nodes);
            }
            if (!n) continue;
            trees.push_back(SahTree{n, first, (uint32_t)node_cursor, k ? SAH_POWER : 0u});
            node_cursor += 2 * (uint64_t)n - 1;
        }
    for (uint32_t c = 0; c < nc; c++) {
        offs[c] = geo_off[c];
        offs[nc + c] = (uint32_t)tot_geo + light_off[c];
        offs[2 * nc + c] = geo_off[c];
        offs[3 * nc + c] = light_off[c];
    }
    uint32_t *d_offs = (uint32_t *)(I + o_plan);
    const ChunkTrees *d_ct = (const ChunkTrees *)(d_offs + 4 * (size_t)nc);
    RootSummary *d_roots = (RootSummary *)(I + o_out);
    uint32_t *d_levels = (uint32_t *)(d_roots + 2 * (size_t)nc);
    VRG_CUDA_TRY(cudaMemcpyAsync(d_offs, offs, plan_bytes, cudaMemcpyHostToDevice, s));
    VRG_CUDA_TRY(cudaMemsetAsync(d_levels, 0, 4, s));
    WriteArgs wa;
    wa.in = d_in;
    wa.rows = d_rows;
    wa.mats = (const vrg_material *)ctx->d_mats->ptr;
    wa.air = ctx->n_types;
    wa.geo_off = d_offs;
    wa.light_off = d_offs + nc;
    wa.loc_off = d_offs + 2 * nc;
    wa.lloc_off = d_offs + 3 * nc;
    wa.lo = (float4 *)(I + o_lo);
    wa.hi = (float4 *)(I + o_hi);
    wa.cen = (float4 *)(I + o_cen);
    wa.id = (uint32_t *)(I + o_id);
    wa.geo_local = (int2 *)(B + o_geo_local);
    wa.light_tri = (uint32_t *)(B + o_light_tri);
    k_extract_write<<<nc, 1024, 0, s>>>(wa);
    VRG_CUDA_TRY(cudaGetLastError());

    SahInputs sin{wa.lo, wa.hi, wa.cen, wa.id};
    SahOutputs sout{(vrg_bvh_node *)(B + o_nodes), (uint32_t *)(B + o_perm), (uint32_t *)(B + o_leaf)};
    uint32_t levels = 0;
    VRG_TRY(sah_build(ctx, trees, (uint32_t)n_prims, (uint32_t)n_nodes, sin, sout, &levels, d_levels));
    k_chunk_finish<<<dim3((std::max(2u, max_light_nodes) + 255) / 256, nc), 256, 0, s>>>(
        d_ct, sout.nodes, sout.leaf_prim, wa.light_tri, sin, (uint32_t *)(B + o_payload), d_roots);
    VRG_CUDA_TRY(cudaGetLastError());
    const RootSummary *roots = (const RootSummary *)(h_in + in_bytes + cnt_bytes + plan_bytes);
    VRG_CUDA_TRY(cudaMemcpyAsync((void *)roots, d_roots, out_bytes, cudaMemcpyDeviceToHost, s));
    VRG_CUDA_TRY(cudaStreamSynchronize(s));
    lease.settled();
    uint32_t lv_dev;
    memcpy(&lv_dev, roots + 2 * (size_t)nc, 4);
    levels = std::max(levels, lv_dev);
    for (uint32_t c = 0; c < nc; c++) {
        Object *ob = batch[c];
        ChunkSummary &cs = ob->sum;
        ob->batch = batch_buf;
        ob->geo_local = (const int2 *)(B + o_geo_local) + geo_off[c];
        ob->light_tri = (const uint32_t *)(B + o_light_tri) + light_off[c];
        if (cs.n_geo) {
            const uint32_t off = ct[c].node_off[0];
            ob->geo_nodes = sout.nodes + off;
            ob->geo_leaf = sout.leaf_prim + off;
            ob->geo_perm = sout.perm + geo_off[c];
            memcpy(cs.geo_lo, roots[2 * c].lo, 12);
            memcpy(cs.geo_hi, roots[2 * c].hi, 12);
        }
        if (cs.n_light) {
            const uint32_t off = ct[c].node_off[1];
            ob->light_nodes = sout.nodes + off;
            ob->light_leaf = sout.leaf_prim + off;
            ob->light_perm = sout.perm + tot_geo + light_off[c];
            ob->light_leaf_tri = (const uint32_t *)(B + o_payload) + (off - tot_geo_nodes);
            memcpy(cs.light_lo, roots[2 * c + 1].lo, 12);
            memcpy(cs.light_hi, roots[2 * c + 1].hi, 12);
            cs.light_power = roots[2 * c + 1].power;
        }
        ob->levels = levels;
        ob->flushed = true;
        ob->blocks.clear();
        ob->blocks.shrink_to_fit();
        ob->slabs.clear();
        ob->slabs.shrink_to_fit();
    }
    return VRG_OK;
}

}  // namespace vrg
