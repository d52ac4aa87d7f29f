// fiber_prepass.cu — work preparation (the reference's work_preparation_pass,
// src/nodes/prepass.rs:27-233 -> run_prepass, src/pipelines/prepass.rs:818-1397).
//
// Stage map (reference entry point -> kernel here):
//   reduce_opaque_depth (opaque_depth_reduce.wgsl:36-86)                -> k_opaque_reduce
//   broad_prepass + broad_strand_prepass (strand_prepass.wgsl:684-782) -> k_broad, folded into k_fine
//   coarse_interval_pass + build_depth_warp_lut (:835-1014)           -> k_lut
//   fine_prepass (:1016-1140)                                           -> k_fine (single-pass compaction)
//   mark_coarse_count_pages_pass (:1928-1932)                           -> k_visit (+ visit records)
//   allocate_coarse_count_pages (:1934-1969)                            -> k_alloc_pages (ordered)
//   binning_queue_pass (:1986-1990)                                     -> k_count_visits | k_traverse<kCount>
//   prefix_fine_pages (:2051-2143)                                      -> k_prefix_pages
//   fill_fine_seg_refs (:2190-2194)                                     -> k_fill_visits | k_traverse<kFill>
//   prefix_active_tile_blocks + compact_active_tiles (:2581-2676)       -> k_compact_active (+ work bases)
//   emit_raster_work (:2678-2834)                                       -> k_emit (canonical cell order: k_sort_cells)
// The finalize_* indirect-argument kernels disappear: every consumer is a
// persistent or grid-stride kernel that reads its item count on the device.
// Append orders that the reference takes from atomics are replaced by
// decoupled look-back scans, so every output is deterministic.
#include <algorithm>

#include "fiber_kernels.cuh"

namespace fiber {

// ===========================================================================
// K0 opaque depth reduce: per camera fine tile, whether every pixel holds
// opaque depth (reversed-Z: > 0 after the min over the pixel's samples) and
// the farthest such depth (the min), quantised. One warp per tile; lanes
// stride over the tile's pixels so a warp reads whole image rows. The result
// is a count and a min, so the lane order cannot change it.
// ===========================================================================
__global__ void __launch_bounds__(256) k_opaque_reduce(const FrameParams* __restrict__ Pp, PrepassArgs A,
                                                       const float* __restrict__ depth, uint32_t pitch,
                                                       uint32_t samples, bool stamp) {
    if (stamp) stamp_start(A.stamps, kStampBroad);
    const fiber_frustum_desc& d = Pp->frusta[0];
    const uint32_t tx = (d.screen_width + d.froxel_size_x - 1u) / d.froxel_size_x;
    const uint32_t ty = (d.screen_height + d.froxel_size_y - 1u) / d.froxel_size_y;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    if (blockIdx.x == 0 && threadIdx.x == 0) A.counters->opaque_bound = 1u;
    for (uint32_t t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tx * ty; t += warps) {
        const uint32_t x0 = (t % tx) * d.froxel_size_x, y0 = (t / tx) * d.froxel_size_y;
        const uint32_t w = min(x0 + d.froxel_size_x, d.screen_width) - x0;
        const uint32_t n = w * (min(y0 + d.froxel_size_y, d.screen_height) - y0);
        uint32_t covered = 0u;
        float farthest = 1.0f;
        for (uint32_t p = lane; p < n; p += 32u) {
            const uint32_t x = x0 + p % w, y = y0 + p / w;
            const float* px = reinterpret_cast<const float*>(reinterpret_cast<const char*>(depth) + (size_t)y * pitch) +
                              (size_t)x * samples;
            float z = __ldg(px);
            for (uint32_t q = 1u; q < samples; ++q) z = wmin(z, __ldg(px + q));
            if (z > 0.0f) {
                ++covered;
                farthest = wmin(farthest, z);
            }
        }
        covered = __reduce_add_sync(0xFFFFFFFFu, covered);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) farthest = wmin(farthest, __shfl_xor_sync(0xFFFFFFFFu, farthest, o));
        if (lane == 0u) A.opaque_tiles[t] = make_uint2(covered == n && n > 0u ? 1u : 0u, quantize_depth01(farthest));
    }
}

// ===========================================================================
// K1 broad prepass: coarse range + keep probabilities per (instance, frustum)
// ===========================================================================
struct CornerScan {
    float sminx, sminy, smaxx, smaxy, zmin, zmax;
    bool any, near_clip;
};

__device__ CornerScan scan_corners(const float4* corners, const float* clip, float vw, float vh) {
    CornerScan s{1e30f, 1e30f, -1e30f, -1e30f, 1.0f, 0.0f, false, false};
    for (int i = 0; i < 8; ++i) {
        float4 c = matvec(clip, corners[i].x, corners[i].y, corners[i].z, corners[i].w);
        if (c.w <= 1e-6f) { s.near_clip = true; continue; }
        float nx = c.x / c.w, ny = c.y / c.w, nz = c.z / c.w;
        if (nz < 0.0f) s.near_clip = true;
        float rx = 0.0f + (nx * 0.5f + 0.5f) * vw;
        float ry = 0.0f + (ny * -0.5f + 0.5f) * vh;
        s.any = true;
        s.sminx = wmin(s.sminx, rx);
        s.sminy = wmin(s.sminy, ry);
        s.smaxx = wmax(s.smaxx, rx);
        s.smaxy = wmax(s.smaxy, ry);
        float z = normalize_depth01(nz);
        s.zmin = wmin(s.zmin, z);
        s.zmax = wmax(s.zmax, z);
    }
    return s;
}

// A warp per instance, a lane per frustum: an (instance, frustum) pair is a
// serial chain of eight projected corners, which a thread per instance paid
// once per frustum. With k_lut: 16 views 158 -> 39 us, 4 frusta 22 -> 18, tiny
// 15 -> 11.
__global__ void __launch_bounds__(128) k_broad(const FrameParams* __restrict__ Pp, const InstanceView* __restrict__ inst,
                                               PrepassArgs A, bool stamp) {
    if (stamp) stamp_start(A.stamps, kStampBroad);
    const FrameParams& P = *Pp;
    const uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (i >= P.I) return;
    const InstanceView& in = inst[i];
    bool visible = false;
    float keep_max = 0.0f;
    float4 corners[8];
    if (in.valid) {
        const float* mn = in.aabb.min;
        const float* mx = in.aabb.max;
        const float cx[8][3] = {{mn[0], mn[1], mn[2]}, {mn[0], mn[1], mx[2]}, {mn[0], mx[1], mn[2]},
                                {mn[0], mx[1], mx[2]}, {mx[0], mn[1], mn[2]}, {mx[0], mn[1], mx[2]},
                                {mx[0], mx[1], mn[2]}, {mx[0], mx[1], mx[2]}};
#pragma unroll
        for (int c = 0; c < 8; ++c) corners[c] = matvec(in.world_from_local, cx[c][0], cx[c][1], cx[c][2], 1.0f);
    }
    for (uint32_t f = lane; f < P.F; f += 32u) {
        const fiber_frustum_desc& d = P.frusta[f];
        float k = 0.0f;
        const uint32_t slot = i * P.F + f;
        bool vis = false;
        // A frustum of another view of a multi-view frame does not see it.
        if (in.valid && d.kind <= 1u && P.fview[f] == in.view && d.coarse_depth_tile_count != 0u &&
            !(d.kind == 1u && light_layer(P, f) == kInvalid)) {
            // emit_coarse_asset_range_for_aabb (strand_prepass.wgsl:575-682)
            const float vw = u2f(d.screen_width), vh = u2f(d.screen_height);
            CornerScan s = scan_corners(corners, P.clip[f], vw, vh);
            if (s.near_clip) {
                s.sminx = 0.0f; s.sminy = 0.0f;
                s.smaxx = vw - 1.0f; s.smaxy = vh - 1.0f;
                s.zmax = 1.0f;
                if (!s.any) s.zmin = 0.0f;
                s.any = true;
            }
            if (s.any && !(s.smaxx < 0.0f || s.smaxy < 0.0f || s.sminx >= vw || s.sminy >= vh) &&
                !(s.zmax < 0.0f || s.zmin > 1.0f)) {
                const uint32_t cpx = max(1u, d.froxel_size_x * kCoarseExtent);
                const uint32_t cpy = max(1u, d.froxel_size_y * kCoarseExtent);
                const float cminx = wclamp(s.sminx, 0.0f, vw - 1.0f), cminy = wclamp(s.sminy, 0.0f, vh - 1.0f);
                const float cmaxx = wclamp(s.smaxx, 0.0f, vw - 1.0f), cmaxy = wclamp(s.smaxy, 0.0f, vh - 1.0f);
                fiber_coarse_asset_range r;
                r.geo_id = i;
                r.frustum_id = f;
                r.min_x = min(f2u(cminx) / cpx, d.coarse_tiles_x - 1u);
                r.max_x = min(f2u(cmaxx) / cpx, d.coarse_tiles_x - 1u);
                r.min_y = min(f2u(cminy) / cpy, d.coarse_tiles_y - 1u);
                r.max_y = min(f2u(cmaxy) / cpy, d.coarse_tiles_y - 1u);
                r.z_min_q = quantize_depth01(s.zmin);
                r.z_max_q = quantize_depth01(s.zmax);
                A.ranges[slot] = r;
                vis = true;
                if (A.tel) {  // FRUSTUM_TELEMETRY_VISIBLE_* (:735-738)
                    atomicAdd(tel_frustum(A.tel, f, kTelVisibleInstances), 1u);
                    atomicAdd(tel_frustum(A.tel, f, kTelVisibleStrands), in.strand_count);
                }
                // aabb_projected_screen_area (:295-362) of a box that is in view
                const float area = s.near_clip ? vw * vh : wmax(cmaxx - cminx, 1.0f) * wmax(cmaxy - cminy, 1.0f);
                // stochastic_{camera,shadow}_keep_probability (:364-392)
                if (P.stochastic_cull_enabled == 0u) k = 1.0f;
                else if (area < 0.0f) k = 0.0f;
                else {
                    const float density = wmax(P.target_strands_per_pixel, 1e-5f);
                    const float min_keep = wclamp(P.min_keep_probability, 0.0f, 1.0f);
                    const float area_keep = wclamp(area * density / wmax(u2f(in.strand_count), 1.0f), min_keep, 1.0f);
                    if (d.kind == 0u) k = area_keep;
                    else {
                        const float cap = wclamp(P.shadow_keep_probability, 0.0f, 1.0f);
                        const float curved = area_keep * area_keep;
                        const float scale = 1.0f / exp2f(u2f(d.cascade_index));
                        k = wclamp(curved * scale * cap, min_keep, 1.0f);
                    }
                }
            }
        }
        A.range_valid[slot] = vis ? 1u : 0u;
        A.keep[slot] = k;
        visible = visible || vis;
        keep_max = wmax(keep_max, k);
    }
    visible = __any_sync(0xFFFFFFFFu, visible);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) keep_max = wmax(keep_max, __shfl_xor_sync(0xFFFFFFFFu, keep_max, o));
    if (lane == 0u) {
        A.inst_visible[i] = visible ? 1u : 0u;
        A.inst_keep[i] = keep_max;
    }
}

// ===========================================================================
// K4 + K5: per coarse tile, merge the depth intervals of the ranges covering
// it (instance order) and split 16 LUT slices across them.
// ===========================================================================
__global__ void k_lut(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    const FrameParams& P = *Pp;
    uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.total_coarse_tiles) return;
    fiber_coarse_depth_lut_entry* out = A.lut + (size_t)t * kDepthSlices;
    uint32_t f = frustum_for_tile(P, t);
    uint32_t mins[kDepthSlices], maxs[kDepthSlices];
    uint32_t count = 0;
    if (f != kInvalid) {
        const fiber_frustum_desc& d = P.frusta[f];
        uint32_t local = t - d.coarse_depth_tile_base;
        uint32_t cx = local % d.coarse_tiles_x, cy = local / d.coarse_tiles_x;
        for (uint32_t i = 0; i < P.I; ++i) {
            uint32_t slot = i * P.F + f;
            if (!A.range_valid[slot]) continue;
            fiber_coarse_asset_range r = A.ranges[slot];
            if (r.max_x < r.min_x || r.max_y < r.min_y) continue;
            if (cx < r.min_x || cx > r.max_x || cy < r.min_y || cy > r.max_y) continue;
            uint32_t zmin = min(r.z_min_q, r.z_max_q), zmax = max(r.z_min_q, r.z_max_q);
            bool merged = false;
            for (uint32_t k = 0; k < count; ++k) {
                if (zmin <= maxs[k] + 1u && zmax + 1u >= mins[k]) {
                    mins[k] = min(mins[k], zmin);
                    maxs[k] = max(maxs[k], zmax);
                    merged = true;
                }
            }
            if (merged) continue;
            if (count < kDepthSlices) {
                mins[count] = zmin;
                maxs[count] = zmax;
                ++count;
            } else {
                uint32_t best = 0, best_gap = 0xFFFFFFFFu;
                for (uint32_t k = 0; k < kDepthSlices; ++k) {
                    uint32_t g = maxs[k] < zmin ? zmin - maxs[k] : (zmax < mins[k] ? mins[k] - zmax : 0u);
                    if (g < best_gap) { best_gap = g; best = k; }
                }
                mins[best] = min(mins[best], zmin);
                maxs[best] = max(maxs[best], zmax);
            }
        }
    }
    for (uint32_t k = 1; k < count; ++k) {
        uint32_t j = k, kmin = mins[k], kmax = maxs[k];
        while (j != 0 && mins[j - 1] > kmin) {
            mins[j] = mins[j - 1];
            maxs[j] = maxs[j - 1];
            --j;
        }
        mins[j] = kmin;
        maxs[j] = kmax;
    }
    uint32_t out_slice = 0;
    // simple: all 16 entries populated, each start <= end, each end below the
    // next start (the lookup in lut_slices may then binary-search).
    bool simple = true;
    uint32_t prev_end = 0u;
    for (uint32_t k = 0; k < count; ++k) {
        uint32_t base_slices = max(1u, kDepthSlices / count);
        uint32_t rem = kDepthSlices % count;
        uint32_t slices = base_slices + (k < rem ? 1u : 0u);
        uint32_t span = max(1u, maxs[k] - mins[k] + 1u);
        for (uint32_t s = 0; s < slices && out_slice < kDepthSlices; ++s) {
            uint32_t start = mins[k] + (span * s) / slices;
            uint32_t excl_end = mins[k] + (span * (s + 1u)) / slices;
            uint32_t end = min(excl_end > start ? excl_end - 1u : start, maxs[k]);
            simple = simple && start <= end && (out_slice == 0u || prev_end < start);
            prev_end = end;
            out[out_slice++] = fiber_coarse_depth_lut_entry{start, end, start, max(1u, end - start + 1u)};
        }
    }
    for (uint32_t k = out_slice; k < kDepthSlices; ++k) out[k] = fiber_coarse_depth_lut_entry{0u, 0u, 0u, 0u};
    // The search tree of a simple LUT (read back from this thread's own
    // entries); word 0 = kInvalid marks a LUT that takes the linear lookup.
    uint4* tree = reinterpret_cast<uint4*>(A.lut_tree + (size_t)t * kLutTreeWords);
    if (simple && out_slice == kDepthSlices) {
        tree[0] = make_uint4(out[0].z_min_q, out[4].z_min_q, out[8].z_min_q, out[12].z_min_q);
        for (uint32_t g = 0; g < 4u; ++g) {
            const fiber_coarse_depth_lut_entry* e = out + 4u * g;
            tree[1u + 2u * g] = make_uint4(e[0].z_min_q, e[1].z_min_q, e[2].z_min_q, e[3].z_min_q);
            tree[2u + 2u * g] = make_uint4(e[0].z_max_q, e[1].z_max_q, e[2].z_max_q, e[3].z_max_q);
        }
    } else {
        tree[0] = make_uint4(kInvalid, kInvalid, kInvalid, kInvalid);
    }
}

// ===========================================================================
// K2 + K6 fine prepass: a warp per strand (a lane per segment), each warp
// taking fine_per_warp consecutive strands (at most 8), one block per (frustum,
// 8 fine_per_warp-strand tile) in frustum-major order. Pass A counts
// every strand's clipped segments; the block takes its output offset from a
// decoupled look-back; pass B projects again and writes BinningTask +
// ProjectedSegment in (frustum, inst, strand, seg) order — the binning
// queue's canonical order, produced without a sort. A tile of 64 strands
// spends one look-back (and two block barriers) on 64 strands' work.
// ===========================================================================
constexpr int kFineThreads = 256;
constexpr int kFineWarps = kFineThreads / 32;
static_assert(kFineWarps == (int)kFineTileWarps, "fine tile shape");

struct SegOut {
    uint32_t seg;
    uint32_t p0, p1, dz;
    float4 r0, r1;  // world_to_screen_raw of both end points, kept for the rasters
};

// world_to_screen_raw (common.wgsl:93-107) of the strand point at index
// position `pos` after the instance transform.
__device__ __forceinline__ float4 fine_vertex(const FrameParams& P, const InstanceView& in, uint32_t f, uint32_t pos) {
    const fiber_frustum_desc& d = P.frusta[f];
    const float4 a = __ldg(in.vertices + __ldg(in.indices + pos));
    const float4 w = matvec(in.world_from_local, a.x, a.y, a.z, 1.0f);
    return world_to_screen_raw(w, P.clip[f], u2f(d.screen_width), u2f(d.screen_height));
}

// A segment from its two projected end points: normalised depth, clip to the
// screen box, quantise (fine_prepass, strand_prepass.wgsl:1016-1140).
__device__ __forceinline__ bool fine_segment(const FrameParams& P, uint32_t f, uint32_t seg, float4 r0, float4 r1,
                                             SegOut& o) {
    const fiber_frustum_desc& d = P.frusta[f];
    const float vw = u2f(d.screen_width), vh = u2f(d.screen_height);
    F3 p0 = f3(r0.x, r0.y, normalize_depth01(r0.z)), p1 = f3(r1.x, r1.y, normalize_depth01(r1.z));
    F3 c0, c1;
    if (!clip_segment(p0, p1, f3(0.0f, 0.0f, 0.0f), f3(wmax(0.0f, vw - 1e-3f), wmax(0.0f, vh - 1e-3f), 1.0f), c0, c1))
        return false;
    float ssx = wmax(1.0f, vw), ssy = wmax(1.0f, vh);
    o.seg = seg;
    o.r0 = r0;
    o.r1 = r1;
    // Quotients by 1 .. 16384; a numerator too small for its residual is far
    // below the 16-bit step.
    const float yx = rcp_exact(ssx), yy = rcp_exact(ssy);
    o.p0 = pack2x16unorm(wclamp(div_by_rcp(c0.x, ssx, yx), 0.0f, 1.0f), wclamp(div_by_rcp(c0.y, ssy, yy), 0.0f, 1.0f));
    o.p1 = pack2x16unorm(wclamp(div_by_rcp(c1.x, ssx, yx), 0.0f, 1.0f), wclamp(div_by_rcp(c1.y, ssy, yy), 0.0f, 1.0f));
    o.dz = pack2x16unorm(wclamp(c0.z, 0.0f, 1.0f), wclamp(c1.z, 0.0f, 1.0f));
    return true;
}

// Segments c .. c + 30 of a strand, one per lane 0..30: lane l projects point
// c + l once and takes its segment's far end point from lane l + 1 (a point
// shared by two segments is projected once, by the same operations).
constexpr uint32_t kFineChunk = 31;
__device__ __forceinline__ bool fine_chunk(const FrameParams& P, const InstanceView& in, uint32_t f,
                                           uint32_t first, uint32_t nseg, uint32_t c, uint32_t lane, SegOut& o) {
    const uint32_t pos = first + c + lane;
    const bool has_point = c + lane <= nseg && pos < in.n_indices;
    float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (has_point) r = fine_vertex(P, in, f, pos);
    float4 r1;
    r1.x = __shfl_down_sync(0xFFFFFFFFu, r.x, 1);
    r1.y = __shfl_down_sync(0xFFFFFFFFu, r.y, 1);
    r1.z = __shfl_down_sync(0xFFFFFFFFu, r.z, 1);
    r1.w = __shfl_down_sync(0xFFFFFFFFu, r.w, 1);
    const bool seg_ok = lane < kFineChunk && c + lane < nseg && pos + 1u < in.n_indices;
    return seg_ok && fine_segment(P, f, pos, r, r1, o);
}

// The strand g of frustum f: instance, local strand, segment count, first
// index and the task's packed field; nseg = 0 when the keep tests drop it.
struct FineStrand {
    uint32_t i, s, nseg, meta_offset, packed, material;
    bool ordered;  // its segments follow the previous strand's in the index slab
    __device__ __forceinline__ FineStrand of_lane(int k) const {
        FineStrand r;
        r.i = __shfl_sync(0xFFFFFFFFu, i, k);
        r.s = __shfl_sync(0xFFFFFFFFu, s, k);
        r.nseg = __shfl_sync(0xFFFFFFFFu, nseg, k);
        r.meta_offset = __shfl_sync(0xFFFFFFFFu, meta_offset, k);
        r.packed = __shfl_sync(0xFFFFFFFFu, packed, k);
        r.material = __shfl_sync(0xFFFFFFFFu, material, k);
        r.ordered = true;
        return r;
    }
};

__device__ __forceinline__ FineStrand fine_strand(const FrameParams& P, const InstanceView* __restrict__ inst,
                                                  const PrepassArgs& A, uint32_t f, uint32_t g, uint32_t g_end) {
    FineStrand r{0u, 0u, 0u, 0u, 0u, 0u, true};
    if (g >= g_end) return r;
    uint32_t lo = 0, hi = P.I;  // last instance with strand_base <= g
    while (hi - lo > 1u) {
        uint32_t mid = (lo + hi) >> 1;
        if (inst[mid].strand_base <= g) lo = mid; else hi = mid;
    }
    r.i = lo;
    r.s = g - inst[lo].strand_base;
    const InstanceView& in = inst[lo];
    const fiber_frustum_desc& d = P.frusta[f];
    // The keep hash takes the instance's id inside its view, so a view keeps
    // the same strands in a multi-view frame as alone (one view: the id).
    const uint32_t local_i = lo - P.view_inst0[P.fview[f]];
    const float h = hash_to_unit_float(wang_hash((local_i * 16777619u) ^ r.s));
    bool ok = in.valid && in.view == P.fview[f] && A.inst_visible[lo] != 0u && r.s < in.strand_count &&
              !(h > A.inst_keep[lo]);
    ok = ok && d.kind <= 1u && r.s < in.n_meta;
    if (in.valid && r.s > 0u && r.s < in.strand_count) {
        const fiber_strand_meta a = in.meta[r.s - 1u];
        r.ordered = (uint64_t)a.offset + max(a.count, 1u) - 1u <= (uint64_t)in.meta[r.s].offset;
    }
    if (ok) {
        const fiber_strand_meta m = in.meta[r.s];
        ok = m.count >= 2u && !(h > A.keep[lo * P.F + f]) && !(d.kind == 1u && light_layer(P, f) == kInvalid);
        if (ok) {
            r.nseg = m.count - 1u;
            r.meta_offset = m.offset;
            r.material = m.material_idx;
            r.packed = ((d.kind == 1u ? 1u : 0u) << 2u) | (f << 3u);
        }
    }
    return r;
}

__global__ void __launch_bounds__(kFineThreads, 4) k_fine(const FrameParams* __restrict__ Pp,
                                                       const InstanceView* __restrict__ inst, PrepassArgs A) {
    stamp_start(A.stamps, kStampFine);
    const FrameParams& P = *Pp;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp_count[kFineWarps];
    __shared__ uint32_t s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // Each frustum's tiles cover its view's strands (every strand of a
    // single-view frame): fine_tile_base is their prefix over frusta.
    const uint32_t n_tiles = P.fine_tile_base[P.F], per_warp = P.fine_per_warp;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(A.tile_counter, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= n_tiles) break;
        uint32_t f = 0, fhi = P.F;  // last frustum whose tiles start at or before tile
        while (fhi - f > 1u) {
            const uint32_t mid = (f + fhi) >> 1;
            if (P.fine_tile_base[mid] <= tile) f = mid; else fhi = mid;
        }
        const uint32_t lt = tile - P.fine_tile_base[f];
        const uint32_t v = P.fview[f];
        const uint32_t g_end = P.view_strand0[v] + P.view_strands[v];
        const uint32_t g0 = P.view_strand0[v] + (lt * kFineWarps + (uint32_t)warp) * per_warp;
        // Lane k looks up the warp's strand k, once for both passes.
        FineStrand own{0u, 0u, 0u, 0u, 0u, 0u, true};
        if (lane < (int)per_warp) own = fine_strand(P, inst, A, f, g0 + lane, g_end);
        if (!own.ordered) A.counters->seg_unordered = 1u;
        // FRUSTUM_TELEMETRY_RETAINED_STRANDS (:1085): every strand the keep
        // tests pass.
        if (A.tel && own.nseg > 0u) atomicAdd(tel_frustum(A.tel, f, kTelRetainedStrands), 1u);
        // Pass A: count the clipped segments of the warp's strands.
        uint32_t count = 0;
        for (uint32_t k = 0; k < per_warp; ++k) {
            const FineStrand fs = own.of_lane((int)k);
            for (uint32_t c = 0; c < fs.nseg; c += kFineChunk) {
                SegOut o;
                const bool ok = fine_chunk(P, inst[fs.i], f, fs.meta_offset, fs.nseg, c, lane, o);
                count += __popc(__ballot_sync(0xFFFFFFFFu, ok));
            }
        }
        if (lane == 0) s_warp_count[warp] = count;
        __syncthreads();
        if (threadIdx.x < 32u) {
            uint32_t agg = 0;
            for (int w = 0; w < kFineWarps; ++w) agg += s_warp_count[w];
            uint32_t base = lb_exclusive_warp(A.lb_status, tile, P.epoch, agg, &A.counters->error, lb_limit(P),
                                              lb_withheld(P, kStageFine));
            if (threadIdx.x == 0) {
                s_base = base;
                if (lt == 0u) A.counters->frustum_task_base[f] = base;
                if (tile == n_tiles - 1u) {
                    A.counters->tasks = base + agg;
                    A.counters->frustum_task_base[P.F] = base + agg;
                }
            }
        }
        __syncthreads();
        uint32_t out = s_base;
        for (int w = 0; w < warp; ++w) out += s_warp_count[w];
        // Pass B: project again and write in segment order.
        for (uint32_t k = 0; k < per_warp; ++k) {
            const FineStrand fs = own.of_lane((int)k);
            for (uint32_t c = 0; c < fs.nseg; c += kFineChunk) {
                SegOut o;
                const bool ok = fine_chunk(P, inst[fs.i], f, fs.meta_offset, fs.nseg, c, lane, o);
                const uint32_t mask = __ballot_sync(0xFFFFFFFFu, ok);
                if (ok) {
                    const uint32_t dst = out + __popc(mask & ((1u << lane) - 1u));
                    if (dst < P.task_capacity) {
                        reinterpret_cast<uint4*>(A.tasks)[dst] = make_uint4(fs.i, fs.s, o.seg, fs.packed);
                        fiber_projected_segment ps{o.p0, o.p1, o.dz};
                        A.projected[dst] = ps;
                        A.task_key[dst] = (o.dz & 0xFFFFu) + (o.dz >> 16u);
                        float4* rec = A.task_rec + (size_t)kTaskRec * dst;
                        rec[0] = o.r0;
                        rec[1] = o.r1;
                        reinterpret_cast<uint4*>(rec)[2] = make_uint4(fs.i, o.seg, fs.material, 0u);
                    } else {
                        atomicOr(&A.counters->overflow, 1u);
                    }
                }
                out += __popc(mask);
            }
        }
        __syncthreads();
    }
}

// ===========================================================================
// K7 / K9 / K11 traversal: coarse-tile 2-D DDA, LUT slices, then the fine
// 3-D DDA inside each page (strand_prepass.wgsl:1251-1696,1894-1926).
//
// The walk is written once; what a pass does at a page-table slot that
// survives the depth clip, and at each fine cell the 3-D DDA visits, is a sink:
//   VisitSink  k_visit: marks the slot (mark_coarse_count_pages_pass) and
//              records the visit (slot << 8 | cell) in a per-thread buffer
//   SpillSink  k_visit: re-walks a task with more visits than the buffer and
//              writes the visits past it
//   CountSink, FillSink  the walking form of binning_queue_pass and
//              fill_fine_seg_refs, used only when the visit records did not fit
// With the records, the count and fill passes stream over visits instead of
// walking every task again (k_count_visits, k_fill_visits).
// ===========================================================================
enum : int { kCount = 1, kFill = 2 };
constexpr uint32_t kVisitThreads = 256;
constexpr uint32_t kVisitSlots = 16;  // buffered visits per coarse tile of a task
// Cell sort sizes: a thread sorts a cell of up to 8 references, a warp one of
// up to 256 (32 lanes x 8 registers), a block anything longer.
constexpr uint32_t kThreadSortMax = 8;
constexpr uint32_t kQuadSortMax = 16;   // 4 lanes x 4 registers: eight cells per warp
constexpr uint32_t kGroupSortMax = 32;  // 8 lanes x 4 registers: four cells per warp
constexpr uint32_t kWarpSortMax = 256;

// lut_slices for one end point of a LUT whose 16 entries are all populated,
// each start <= end and each end below the next start: at most one entry
// holds the quantised depth q, and the nearest entry otherwise is a neighbour
// of the gap q falls in, so the last entry whose start is <= q (the starts
// increase strictly) answers what the linear scan answers (first holding
// entry, else first nearest). The search reads the LUT's tree: the quarter
// starts (piv, shared by both end points), then the quarter's starts and ends.
__device__ __forceinline__ uint32_t lut_slice_tree(const uint4* tree, const uint4& piv, float z) {
    const uint32_t q = quantize_depth01(z);
    if (piv.x > q) return 0u;  // no entry starts at or below q: the first is nearest
    const uint32_t g = (piv.y <= q ? 1u : 0u) + (piv.z <= q ? 1u : 0u) + (piv.w <= q ? 1u : 0u);
    const uint4 st = __ldg(tree + 1u + 2u * g), en = __ldg(tree + 2u + 2u * g);
    const uint32_t r = (st.y <= q ? 1u : 0u) + (st.z <= q ? 1u : 0u) + (st.w <= q ? 1u : 0u);
    const uint32_t lo = 4u * g + r;
    const uint32_t end = r == 0u ? en.x : (r == 1u ? en.y : (r == 2u ? en.z : en.w));
    if (q <= end || lo == kDepthSlices - 1u) return lo;
    const uint32_t next_piv = g == 0u ? piv.y : (g == 1u ? piv.z : piv.w);
    const uint32_t next_start = r == 0u ? st.y : (r == 1u ? st.z : (r == 2u ? st.w : next_piv));
    return (q - end <= next_start - q) ? lo : lo + 1u;
}

// lut_slice for both clipped end points at once: per end point, the first
// populated slice whose [z_min_q, z_max_q] holds its quantised depth, else the
// first populated slice nearest to it, else kInvalid. One unrolled pass over
// the 16 entries without an early exit, so their loads issue together.
__device__ __forceinline__ void lut_slices(const fiber_coarse_depth_lut_entry* e, float za, float zb, uint32_t& sa,
                                           uint32_t& sb) {
    const uint32_t qa = quantize_depth01(za), qb = quantize_depth01(zb);
    uint32_t fa = kInvalid, fb = kInvalid, ba = kInvalid, bb = kInvalid, da = 0xFFFFFFFFu, db = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t i = 0; i < kDepthSlices; ++i) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(e) + i);  // z_min_q, z_max_q, -, virtual_count_q
        if (x.w == 0u) continue;
        if (qa >= x.x && qa <= x.y && fa == kInvalid) fa = i;
        if (qb >= x.x && qb <= x.y && fb == kInvalid) fb = i;
        const uint32_t ea = qa > x.y ? qa - x.y : x.x - qa;  // meaningful only while nothing holds qa
        const uint32_t eb = qb > x.y ? qb - x.y : x.x - qb;
        if (ea < da) { da = ea; ba = i; }
        if (eb < db) { db = eb; bb = i; }
    }
    sa = fa != kInvalid ? fa : ba;
    sb = fb != kInvalid ? fb : bb;
}

// Sinks. page_slot(pti) returns whether to walk the slot's fine cells.
// kTel: count the task as a candidate of the slot (telemetry); a task visits
// each slot once.
template <bool kTel>
struct VisitSink {
    uint32_t* page_table;
    uint32_t* buf;  // this lane's column of the warp's buffer (stride 32)
    uint32_t cur, n;
    bool records;
    uint32_t* tel_slots;
    __device__ __forceinline__ bool page_slot(uint32_t pti) {
        page_table[pti] = kMarked;
        if (kTel) atomicAdd(tel_slots + pti, 1u);
        cur = pti << 8;
        return records;
    }
    __device__ __forceinline__ void cell(uint32_t c) {
        if (n < kVisitSlots) buf[n * 32u] = cur | c;
        ++n;
    }
};

struct SpillSink {
    uint32_t* rec;
    uint32_t* task;
    uint32_t at, k, lim, cur, n;  // lim: visits the first walk counted (the room reserved)
    __device__ __forceinline__ bool page_slot(uint32_t pti) {
        cur = pti << 8;
        return true;
    }
    __device__ __forceinline__ void cell(uint32_t c) {
        if (n >= kVisitSlots && n < lim) {
            rec[at + n] = cur | c;
            task[at + n] = k;
        }
        ++n;
    }
};

struct CountSink {
    const uint32_t* page_table;
    uint32_t* counts;
    uint32_t page;
    __device__ __forceinline__ bool page_slot(uint32_t pti) {
        uint32_t h = page_table[pti];
        if (h == 0u || h == kMarked) return false;
        page = h - 1u;
        return true;
    }
    __device__ __forceinline__ void cell(uint32_t c) { atomicAdd(counts + (size_t)page * kPageSize + c, 1u); }
};

struct FillSink {
    const PrepassArgs* A;
    uint32_t page, base, count, task;
    __device__ __forceinline__ bool page_slot(uint32_t pti) {
        uint32_t h = A->page_table[pti];
        if (h == 0u || h == kMarked) return false;
        page = h - 1u;
        const fiber_fine_page_meta pm = A->page_meta[page];
        base = pm.seg_ref_base;
        count = pm.seg_ref_count;
        return count != 0u;
    }
    __device__ __forceinline__ void cell(uint32_t c) {
        const uint32_t dst = atomicAdd(A->cursors + (size_t)page * kPageSize + c, 1u);
        if (dst - base >= count) return;
        A->ref_task[dst] = task;  // k_sort_cells orders the cell
    }
};

constexpr uint32_t kMaxCellSteps = kCoarseExtent + kCoarseExtent + kDepthSlices + 4u;  // cells of one slice's walk
// opq: the opaque fine tiles of the camera (null when none are bound); pd:
// the segment's clip direction (p1 - p0 and its reciprocals); (ccx, ccy): the
// coarse tile's column and row in the frustum.
template <class Sink>
__device__ __forceinline__ void walk_page(const PrepassArgs& A, F3 p0, const ClipDir& pd, const fiber_frustum_desc& d,
                                          uint32_t tile, uint32_t ccx, uint32_t ccy, const uint2* opq, Sink& sink) {
    // fine_tile_occluded_by_opaque (:551-573) applies to the camera only. The
    // opaque tiles hold the camera's fine tiles alone, so the camera's
    // fine_depth_tile_base (0) is not added.
    if (d.kind != 0u) opq = nullptr;
    uint32_t ftx = 0u, fty = 0u;
    if (opq) {
        ftx = (d.screen_width + d.froxel_size_x - 1u) / d.froxel_size_x;
        fty = (d.screen_height + d.froxel_size_y - 1u) / d.froxel_size_y;
    }
    uint32_t cpx = max(1u, d.froxel_size_x * kCoarseExtent);
    uint32_t cpy = max(1u, d.froxel_size_y * kCoarseExtent);
    float ox = u2f(ccx * cpx), oy = u2f(ccy * cpy);
    float tmx = wmin(ox + u2f(cpx), u2f(d.screen_width)) - 1e-3f;
    float tmy = wmin(oy + u2f(cpy), u2f(d.screen_height)) - 1e-3f;
    F3 bmax = f3(wmax(ox, tmx), wmax(oy, tmy), 1.0f);
    F3 c0, c1;
    if (!clip_segment_pre(p0, pd, f3(ox, oy, 0.0f), bmax, c0, c1)) return;
    const ClipDir cd = clip_dir(c0, c1);  // shared by the slice clips below
    const fiber_coarse_depth_lut_entry* lut = A.lut + (size_t)tile * kDepthSlices;
    const uint4* tree = reinterpret_cast<const uint4*>(A.lut_tree + (size_t)tile * kLutTreeWords);
    const uint4 piv = __ldg(tree);
    uint32_t z0s, z1s;
    if (piv.x != kInvalid) {
        z0s = lut_slice_tree(tree, piv, c0.z);
        z1s = lut_slice_tree(tree, piv, c1.z);
    } else {
        lut_slices(lut, c0.z, c1.z, z0s, z1s);
    }
    if (z0s == kInvalid || z1s == kInvalid) return;
    for (uint32_t cz = min(z0s, z1s); cz <= max(z0s, z1s); ++cz) {
        fiber_coarse_depth_lut_entry e = lut[cz];
        if (e.virtual_count_q == 0u) continue;
        float zmin = dequantize_depth01(e.z_min_q), zmax = dequantize_depth01(e.z_max_q);
        F3 d0, d1;
        if (!clip_segment_pre(c0, cd, f3(ox, oy, zmin), f3(bmax.x, bmax.y, zmax), d0, d1)) continue;
        if (!sink.page_slot(tile * kDepthSlices + cz)) continue;
        // The quotients below divide by 6e-8 .. 1 (zspan) and 1e-6 .. 16 (sd);
        // their numerators are zero or differences of screen coordinates, depths
        // and cell positions, which are multiples of 2^-60 at least.
        const float zspan = wmax(zmax - zmin, 1.0f / (float)kDepthQuantMax), zrcp = rcp_exact(zspan);
        const uint32_t fsx = d.froxel_size_x, fsy = d.froxel_size_y;
        float l0[3] = {div_by(d0.x - ox, fsx), div_by(d0.y - oy, fsy),
                       wclamp(div_by_rcp(d0.z - zmin, zspan, zrcp), 0.0f, 0.999999f) * 16.0f};
        float l1[3] = {div_by(d1.x - ox, fsx), div_by(d1.y - oy, fsy),
                       wclamp(div_by_rcp(d1.z - zmin, zspan, zrcp), 0.0f, 0.999999f) * 16.0f};
        // The walk's place as one word: the cell index, x + 4, y + 4 and z + 16
        // (in range: the field's top two bits are 01), and the steps taken, whose
        // limit carries into bit 31. A step along an axis is one addition.
        constexpr uint32_t kX = 1u << 10, kY = 1u << 14, kZ = 1u << 18, kStep = 1u << 26;
        constexpr uint32_t kTop = 12u * kX + 12u * kY + 48u * kZ + (1u << 31), kIn = 4u * kX + 4u * kY + 16u * kZ;
        uint32_t at = kIn + (32u - kMaxCellSteps) * kStep, end = kIn, move[3];
        float tm[3], dd[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int32_t hi = a == 2 ? 15 : 3;
            const uint32_t unit = a == 0 ? 1u + kX : (a == 1 ? 4u + kY : 16u + kZ);
            at += (uint32_t)iclamp(f2i(floorf(l0[a])), 0, hi) * unit;
            end += (uint32_t)iclamp(f2i(floorf(l1[a])), 0, hi) * unit;
            float dir = l1[a] - l0[a];
            const int32_t step = sgn_i32(dir);
            move[a] = (uint32_t)step * unit + kStep;
            float sd = fabsf(dir) < 1e-6f ? 1e-6f : dir;
            const float y = rcp_exact(sd);
            dd[a] = fabsf(y);
            float fl = floorf(l0[a]);
            tm[a] = div_by_rcp(step > 0 ? (fl + 1.0f) - l0[a] : fl - l0[a], sd, y);
            if (fabsf(dir) < 1e-6f) tm[a] = 1e38f;
        }
        for (;;) {
            // A covered fine tile whose farthest opaque depth is in front of
            // this slice's nearest depth (reversed-Z: z_max) hides the cell.
            bool occluded = false;
            if (opq) {
                const uint32_t fx = ccx * kCoarseExtent + (at / kX & 3u), fy = ccy * kCoarseExtent + (at / kY & 3u);
                if (fx < ftx && fy < fty) {
                    const uint2 o = __ldg(opq + (size_t)fy * ftx + fx);
                    occluded = o.x != 0u && zmax <= dequantize_depth01(o.y) - 1e-4f;
                }
            }
            if (!occluded) sink.cell(at & 0xFFu);
            if (((at ^ end) & (kStep - 1u)) == 0u) break;
            const float m = wmin(wmin(tm[0], tm[1]), tm[2]);  // canonical_min_mask
            if (tm[0] == m) { at += move[0]; tm[0] += dd[0]; }
            else if (tm[1] == m) { at += move[1]; tm[1] += dd[1]; }
            else { at += move[2]; tm[2] += dd[2]; }
            if (((at ^ kIn) & kTop) != 0u) break;
        }
    }
}

// One binning task's walk inputs (binning_queue_pass preamble, :1894-1926).
struct TaskWalk {
    F3 p0, p1;        // projected endpoints in pixels / depth01
    uint32_t f;       // frustum
    uint32_t min_cx, max_cx, min_cy, max_cy;
};

__device__ __forceinline__ bool task_walk(const FrameParams& P, const PrepassArgs& A, uint32_t k, TaskWalk& w) {
    const uint4 t = reinterpret_cast<const uint4*>(A.tasks)[k];
    const uint32_t f = t.w >> 3u;
    if (f >= P.F) return false;
    const uint32_t i = t.x;
    if (i >= P.I) return false;
    const fiber_frustum_desc& d = P.frusta[f];
    const fiber_projected_segment pr = A.projected[k];
    const float sw = u2f(d.screen_width), sh = u2f(d.screen_height);
    const float2 a = unpack2x16unorm(pr.p0_xy), b = unpack2x16unorm(pr.p1_xy), z = unpack2x16unorm(pr.depths);
    const F3 p0 = f3(a.x * sw, a.y * sh, z.x), p1 = f3(b.x * sw, b.y * sh, z.y);
    const uint32_t slot = i * P.F + f;
    if (!A.range_valid[slot]) return false;
    const fiber_coarse_asset_range r = A.ranges[slot];
    const uint32_t cpx = max(1u, d.froxel_size_x * kCoarseExtent);
    const uint32_t cpy = max(1u, d.froxel_size_y * kCoarseExtent);
    w.min_cx = max(r.min_x, min(f2u(wmax(wmin(p0.x, p1.x), 0.0f)) / cpx, d.coarse_tiles_x - 1u));
    w.max_cx = min(r.max_x, min(f2u(wmax(wmax(p0.x, p1.x), 0.0f)) / cpx, d.coarse_tiles_x - 1u));
    w.min_cy = max(r.min_y, min(f2u(wmax(wmin(p0.y, p1.y), 0.0f)) / cpy, d.coarse_tiles_y - 1u));
    w.max_cy = min(r.max_y, min(f2u(wmax(wmax(p0.y, p1.y), 0.0f)) / cpy, d.coarse_tiles_y - 1u));
    if (w.max_cx < w.min_cx || w.max_cy < w.min_cy) return false;
    w.p0 = p0;
    w.p1 = p1;
    w.f = f;
    return true;
}

// Coarse-tile 2-D DDA over the task's clipped range.
struct TileWalk {
    int32_t fx, fy, ex, ey, sx, sy;
    float tx, ty, ddx, ddy;
    uint32_t min_cx, max_cx, min_cy, max_cy, left;  // left: tiles the walk may still enter
    __device__ __forceinline__ bool begin(const FrameParams& P, const TaskWalk& w, const ClipDir& pd) {
        const fiber_frustum_desc& d = P.frusta[w.f];
        const float sw = u2f(d.screen_width), sh = u2f(d.screen_height);
        const uint32_t cpx = max(1u, d.froxel_size_x * kCoarseExtent);
        const uint32_t cpy = max(1u, d.froxel_size_y * kCoarseExtent);
        min_cx = w.min_cx, max_cx = w.max_cx, min_cy = w.min_cy, max_cy = w.max_cy;
        F3 bmin = f3(u2f(min_cx * cpx), u2f(min_cy * cpy), 0.0f);
        F3 bmax = f3(wmin(u2f((max_cx + 1u) * cpx), sw) - 1e-3f, wmin(u2f((max_cy + 1u) * cpy), sh) - 1e-3f, 1.0f);
        F3 c0, c1;
        if (!clip_segment_pre(w.p0, pd, bmin, bmax, c0, c1)) return false;
        float x0 = div_by(c0.x, cpx), y0 = div_by(c0.y, cpy), x1 = div_by(c1.x, cpx), y1 = div_by(c1.y, cpy);
        fx = iclamp(f2i(floorf(x0)), (int32_t)min_cx, (int32_t)max_cx);
        fy = iclamp(f2i(floorf(y0)), (int32_t)min_cy, (int32_t)max_cy);
        ex = iclamp(f2i(floorf(x1)), (int32_t)min_cx, (int32_t)max_cx);
        ey = iclamp(f2i(floorf(y1)), (int32_t)min_cy, (int32_t)max_cy);
        float dx = x1 - x0, dy = y1 - y0;
        sx = sgn_i32(dx), sy = sgn_i32(dy);
        float sdx = fabsf(dx) < 1e-6f ? 1e-6f : dx, sdy = fabsf(dy) < 1e-6f ? 1e-6f : dy;
        // |sdx|, |sdy| are 1e-6 to 16384 coarse tiles.
        const float rx = rcp_exact(sdx), ry = rcp_exact(sdy);
        ddx = fabsf(rx), ddy = fabsf(ry);
        float flx = floorf(x0), fly = floorf(y0);
        tx = div_by_rcp(sx > 0 ? (flx + 1.0f) - x0 : flx - x0, sdx, rx);
        ty = div_by_rcp(sy > 0 ? (fly + 1.0f) - y0 : fly - y0, sdy, ry);
        if (fabsf(dx) < 1e-6f) tx = 1e38f;
        if (fabsf(dy) < 1e-6f) ty = 1e38f;
        left = (max_cx - min_cx + 1u) + (max_cy - min_cy + 1u) + 3u;
        return true;
    }
    // Whether the walk is at a tile of its range.
    __device__ __forceinline__ bool here() const {
        return left != 0u && fx >= (int32_t)min_cx && fx <= (int32_t)max_cx && fy >= (int32_t)min_cy && fy <= (int32_t)max_cy;
    }
    // On to the next tile; false after the last.
    __device__ __forceinline__ bool advance() {
        if (fx == ex && fy == ey) return false;
        if (tx <= ty) { fx += sx; tx += ddx; } else { fy += sy; ty += ddy; }
        --left;
        return true;
    }
};

// Each coarse tile of the task is walked by walk_page.
template <class Sink>
__device__ __forceinline__ void walk_task(const FrameParams& P, const PrepassArgs& A, const TaskWalk& w,
                                          const uint2* opq, Sink& sink) {
    const fiber_frustum_desc& d = P.frusta[w.f];
    const ClipDir pd = clip_dir(w.p0, w.p1);  // shared by every coarse tile's clip
    TileWalk t;
    if (!t.begin(P, w, pd)) return;
    while (t.here()) {
        const uint32_t local = (uint32_t)t.fy * d.coarse_tiles_x + (uint32_t)t.fx;
        if (local < d.coarse_depth_tile_count)
            walk_page(A, w.p0, pd, d, d.coarse_depth_tile_base + local, (uint32_t)t.fx, (uint32_t)t.fy, opq, sink);
        if (!t.advance()) break;
    }
}

// Canonical order of the references in a cell as one 64-bit key: projected
// depth key (z0_16 + z1_16, 17 bits) descending, then instance, then segment.
__device__ __forceinline__ unsigned long long ref_sort_key(uint32_t key17, uint32_t inst, uint32_t seg) {
    return ((unsigned long long)(0x1FFFFu - (key17 & 0x1FFFFu)) << 47) |
           ((unsigned long long)(inst & 0x7FFFu) << 32) | (unsigned long long)seg;
}

__device__ __forceinline__ bool visits_unused(const PrepassArgs& A) {
    return *((volatile uint32_t*)&A.counters->visit_overflow) != 0u;
}

// K7: page marks + visit records. A warp takes 32 tasks at a time, a lane per
// task, and puts their coarse tiles into its queue; whenever 32 wait it walks
// them, a lane per tile. A tile's visits go to shared memory and from there to
// the warp's stage, which is written out with one reservation when it is full.
// Batches that do not fit it, or hold a tile of more than kVisitSlots visits
// (which is walked again to write the rest), are written directly. When the
// records do not fit (or slots exceed 24 bits) the pass still marks every page and
// raises visit_overflow, which hands count and fill to the walking kernels.
// Bound by instruction issue (62 % of the slots, 24 of 32 lanes) and the loads
// between them: a task has 1.5 coarse tiles on average and 2.8 in the longest of 32, so a lane that walked its own task's tiles (two clips, a
// slice lookup and a cell walk each) idled half of the time. Medium frame 674 ->
// 550 us, large 7.4 -> 6.5 ms, 16 views 3.3 -> 2.7, close-up 228 -> 175 us. What it
// takes: the reservations are atomics on one address, which the device takes at
// one per 3 ns (one per batch, without the stage: 960 us; a stage of 192 records
// 10 ms on the large frame), and tiles queued task by task (one tile of each of
// the 32 in turn: the fill's scattered accesses 257 -> 277 us). A queue of 128
// tiles left less L1 and took 575 us.
// kOpaque: the frame has opaque fine tiles (K0 ran); the variant without them
// carries no cull code. kTel: count page candidates for the telemetry.
constexpr uint32_t kTileQueue = 96;  // up to 31 left over and the 1.5 tiles per task of the next 32, mostly
constexpr uint32_t kVisitStage = 256;
struct VisitSmem {
    uint4 p[kTileQueue], q[kTileQueue];  // (p0, p1.x), (p1.yz, tile x, y)
    uint2 task[kTileQueue];              // (task, frustum)
    uint32_t buf[kVisitSlots * 32u];     // [slot][lane] visits of this lane's tile
    uint32_t stage_rec[kVisitStage], stage_task[kVisitStage];
};
constexpr size_t kVisitSmemBytes = sizeof(VisitSmem) * (kVisitThreads / 32u);
template <bool kOpaque, bool kTel>
__global__ void __launch_bounds__(kVisitThreads, 3) k_visit(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    stamp_start(A.stamps, kStampVisit);
    if (frame_failed(A.counters)) return;
    const FrameParams& P = *Pp;
    extern __shared__ VisitSmem s_visit[];
    VisitSmem& sm = s_visit[threadIdx.x >> 5];
    const uint32_t n = *((volatile uint32_t*)&A.counters->tasks);
    const uint32_t n_cap = min(n, P.task_capacity);
    const bool records = P.visit_records != 0u;
    const uint2* opq = kOpaque ? A.opaque_tiles : nullptr;
    if (!records && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&A.counters->visit_overflow, 1u);
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    // 16 tasks at a time if all of them still fit the warps: their tiles are one
    // batch then, not two (tiny frame 13 us against 18).
    const uint32_t warps = gridDim.x * (kVisitThreads / 32u), group = n_cap <= warps * 16u ? 16u : 32u;
    const uint32_t stride = warps * group;
    uint32_t k = (blockIdx.x * (kVisitThreads / 32u) + (threadIdx.x >> 5)) * group + lane;  // this lane's next task
    uint32_t head = 0u, queued = 0u;                        // ring of queued tiles
    bool more = false;                                      // the task has tiles left
    TaskWalk w;
    TileWalk t;
    uint32_t staged = 0u;
    auto ring = [](uint32_t at) { return at >= kTileQueue ? at - kTileQueue : at; };
    auto in_frustum = [&](const TileWalk& c) {
        const fiber_frustum_desc& d = P.frusta[w.f];
        return (uint32_t)c.fy * d.coarse_tiles_x + (uint32_t)c.fx < d.coarse_depth_tile_count;
    };
    // This lane's task at its tile into the queue.
    auto put = [&](uint32_t place) {
        const uint32_t at = ring(place);
        sm.p[at] = make_uint4(__float_as_uint(w.p0.x), __float_as_uint(w.p0.y), __float_as_uint(w.p0.z),
                              __float_as_uint(w.p1.x));
        sm.q[at] = make_uint4(__float_as_uint(w.p1.y), __float_as_uint(w.p1.z), (uint32_t)t.fx, (uint32_t)t.fy);
        sm.task[at] = make_uint2(k - stride, w.f);
    };
    // Room for n visits; kInvalid if they do not fit.
    auto reserve = [&](uint32_t n) -> uint32_t {
        uint32_t base = kInvalid;
        if (lane == 0u && n > 0u && !visits_unused(A)) {
            const unsigned long long b = atomicAdd(&A.counters->visits, (unsigned long long)n);
            if (b + n <= (unsigned long long)P.ref_capacity) base = (uint32_t)b;
            else atomicOr(&A.counters->visit_overflow, 1u);
        }
        return __shfl_sync(0xFFFFFFFFu, base, 0);
    };
    // Visit records are placed in reservation order; the count and fill passes
    // and the cell sort make the references independent of it. Streaming
    // stores: the records are read once, by the count pass.
    auto flush = [&] {
        const uint32_t base = reserve(staged);
        __syncwarp();
        if (base != kInvalid)
            for (uint32_t i = lane; i < staged; i += 32u) {
                __stcs(A.visit_rec + base + i, sm.stage_rec[i]);
                __stcs(A.visit_task + base + i, sm.stage_task[i]);
            }
        __syncwarp();
        staged = 0u;
    };
    for (;;) {
        while (queued < 32u) {
            if (!__any_sync(0xFFFFFFFFu, more)) {
                if (k - lane >= n_cap) break;  // the warp's tasks are done
                more = lane < group && k < n_cap && task_walk(P, A, k, w) && t.begin(P, w, clip_dir(w.p0, w.p1));
                k += stride;
                // Their tiles in task order, if the queue holds them all: the
                // visits of a strand's neighbouring segments stay together, and
                // so do the fill's accesses.
                uint32_t tiles = 0u;
                if (more) {
                    TileWalk c = t;
                    while (c.here()) {
                        tiles += in_frustum(c) ? 1u : 0u;
                        if (!c.advance()) break;
                    }
                }
                uint32_t incl = tiles;
#pragma unroll
                for (uint32_t o = 1; o < 32u; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += y;
                }
                const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
                if (queued + total <= kTileQueue) {
                    uint32_t at = head + queued + incl - tiles;
                    while (tiles) {
                        if (in_frustum(t)) {
                            put(at++);
                            --tiles;
                        }
                        t.advance();
                    }
                    queued += total;
                    more = false;
                    continue;
                }
            }
            bool push = false;
            if (more && t.here()) push = in_frustum(t);
            else more = false;
            const uint32_t pushed = __ballot_sync(0xFFFFFFFFu, push);
            if (push) put(head + queued + (uint32_t)__popc(pushed & below));
            queued += (uint32_t)__popc(pushed);
            if (more) more = t.advance();
        }
        // The staged visits are written before they would overflow, and at the end.
        if (queued == 0u) {
            flush();
            break;
        }
        __syncwarp();
        const uint32_t batch = min(queued, 32u);
        VisitSink<kTel> vs{A.page_table, sm.buf + lane, 0u, 0u, records, A.tel_slots};
        uint32_t task = 0u;
        // Walks this lane's tile of the batch.
        auto walk = [&](auto& sink) {
            const uint32_t at = ring(head + lane);
            const uint4 a = sm.p[at], b = sm.q[at];
            const uint2 c = sm.task[at];
            task = c.x;
            const fiber_frustum_desc& d = P.frusta[c.y];
            const F3 p0 = f3(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z));
            const F3 p1 = f3(__uint_as_float(a.w), __uint_as_float(b.x), __uint_as_float(b.y));
            walk_page(A, p0, clip_dir(p0, p1), d, d.coarse_depth_tile_base + b.w * d.coarse_tiles_x + b.z, b.z, b.w, opq, sink);
        };
        if (lane < batch) walk(vs);
        if (records) {
            uint32_t incl = vs.n;
#pragma unroll
            for (uint32_t o = 1; o < 32u; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            const bool spilled = __any_sync(0xFFFFFFFFu, vs.n > kVisitSlots);
            if (!spilled && total <= kVisitStage) {
                if (staged + total > kVisitStage) flush();
                const uint32_t at = staged + incl - vs.n;
                for (uint32_t j = 0; j < vs.n; ++j) {
                    sm.stage_rec[at + j] = sm.buf[j * 32u + lane];
                    sm.stage_task[at + j] = task;
                }
                staged += total;
            } else if (const uint32_t base = reserve(total); base != kInvalid && vs.n > 0u) {
                const uint32_t at = base + incl - vs.n;
                for (uint32_t j = 0; j < min(vs.n, kVisitSlots); ++j) {
                    __stcs(A.visit_rec + at + j, sm.buf[j * 32u + lane]);
                    __stcs(A.visit_task + at + j, task);
                }
                if (vs.n > kVisitSlots) {
                    SpillSink sp{A.visit_rec, A.visit_task, at, task, vs.n, 0u, 0u};
                    walk(sp);
                }
            }
        }
        __syncwarp();
        head = ring(head + batch);
        queued -= batch;
    }
}

// K9 over visit records: cell counts by atomics; each visit keeps its rank.
// Bound by the L2's scattered accesses, one per sector and instruction: a lane
// per visit keeps the neighbouring cells of one task in one instruction (four
// consecutive visits per lane took 0.24 ms against 0.18 on the medium frame).
__global__ void __launch_bounds__(256) k_count_visits(PrepassArgs A) {
    stamp_start(A.stamps, kStampCount);
    if (frame_failed(A.counters)) return;
    if (visits_unused(A)) return;
    const uint32_t n = (uint32_t)*((volatile unsigned long long*)&A.counters->visits);
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t rec = A.visit_rec[r];
        const uint32_t h = A.page_table[rec >> 8];
        uint32_t g = kInvalid, rank = 0u;
        if (h != 0u && h != kMarked) {
            g = (h - 1u) * kPageSize + (rec & 0xFFu);
            rank = atomicAdd(A.counts + g, 1u);
        }
        A.visit_rec[r] = g;
        A.visit_rank[r] = rank;
    }
}

// K11 over visit records: the visit's slot is its cell's first reference (the
// page prefix leaves it in `cursors`, kInvalid for a page that lost its
// references) + rank. A reference is its binning task's index (4 B, an array
// which a frame's L2 holds; 8 B words with the depth key beside it made the
// fill 0.43 ms on the medium frame against 0.25); k_sort_cells puts each cell's
// into canonical order.
__global__ void __launch_bounds__(256) k_fill_visits(PrepassArgs A) {
    stamp_start(A.stamps, kStampFill);
    if (frame_failed(A.counters)) return;
    if (visits_unused(A)) return;
    const uint32_t n = (uint32_t)*((volatile unsigned long long*)&A.counters->visits);
    // The visit records stream through once (evict-first loads), so L2 keeps
    // the scattered task-index lines until their sectors are complete.
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t g = __ldcs(A.visit_rec + r);
        const uint32_t task = __ldcs(A.visit_task + r), rank = __ldcs(A.visit_rank + r);
        if (g == kInvalid) continue;
        const uint32_t first = A.cursors[g];
        if (first != kInvalid) A.ref_task[first + rank] = task;
    }
}

// K9 / K11 walking form, for frames whose visit records did not fit.
template <int PASS, bool kOpaque>
__global__ void __launch_bounds__(256) k_traverse(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    if (frame_failed(A.counters)) return;
    if (!visits_unused(A)) return;
    const FrameParams& P = *Pp;
    const uint32_t n = *((volatile uint32_t*)&A.counters->tasks);
    const uint32_t n_cap = min(n, P.task_capacity);
    const uint2* opq = kOpaque ? A.opaque_tiles : nullptr;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_cap; k += gridDim.x * blockDim.x) {
        TaskWalk w;
        if (!task_walk(P, A, k, w)) continue;
        if (PASS == kCount) {
            CountSink cs{A.page_table, A.counts, 0u};
            walk_task(P, A, w, opq, cs);
        } else {
            FillSink fs{&A, 0u, 0u, 0u, k};
            walk_task(P, A, w, opq, fs);
        }
    }
}

// ===========================================================================
// K8: allocate marked pages in page-table order.
// ===========================================================================
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;

__global__ void __launch_bounds__(kScanThreads) k_alloc_pages(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    stamp_start(A.stamps, kStampAlloc);
    if (frame_failed(A.counters)) return;
    const FrameParams& P = *Pp;
    __shared__ uint32_t s_tile, s_base;
    __shared__ uint32_t s_warp[33];
    const uint32_t n = P.total_coarse_tiles * kDepthSlices;
    const uint32_t per_tile = kScanThreads * kScanItems;
    const uint32_t n_tiles = ceil_div(n, per_tile);
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(A.tile_counter, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= n_tiles) break;
        const uint32_t e0 = tile * per_tile + threadIdx.x * kScanItems;
        uint32_t flags[kScanItems], cnt = 0;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            flags[j] = (e0 + j < n && A.page_table[e0 + j] == kMarked) ? 1u : 0u;
            cnt += flags[j];
        }
        uint32_t total;
        uint32_t excl = block_exclusive_scan<kScanThreads>(cnt, s_warp, total);
        if (threadIdx.x < 32u) {
            uint32_t base = lb_exclusive_warp(A.lb_status, tile, P.epoch, total, &A.counters->error, lb_limit(P),
                                              lb_withheld(P, kStageAlloc));
            if (threadIdx.x == 0) {
                s_base = base;
                if (tile == n_tiles - 1u) A.counters->pages = min(base + total, P.page_capacity);
            }
        }
        __syncthreads();
        uint32_t idx = s_base + excl;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            if (!flags[j]) continue;
            uint32_t pti = e0 + j;
            if (idx >= P.page_capacity) {
                A.page_table[pti] = 0u;
                atomicOr(&A.counters->overflow, 2u);
            } else {
                A.page_meta[idx] = fiber_fine_page_meta{0u, 0u, 0u, 0u, pti / kDepthSlices, pti % kDepthSlices, 0u, 0u};
                A.page_table[pti] = idx + 1u;
            }
            ++idx;
        }
        __syncthreads();
    }
}

// The new pages' counts, over the whole grid (zeroed by the allocating blocks
// they took 13 us more on the small frame than this kernel's launch).
__global__ void k_zero_pages(PrepassArgs A) {
    const uint32_t pages = *((volatile uint32_t*)&A.counters->pages);
    const uint32_t n = pages * (kPageSize / 4u);
    uint4* c = reinterpret_cast<uint4*>(A.counts);
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        c[k] = make_uint4(0u, 0u, 0u, 0u);
    if (A.page_nvis)
        for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < pages; k += gridDim.x * blockDim.x)
            A.page_nvis[k] = 0u;
}

// ===========================================================================
// K10: per page exclusive scan of the 256 cell counts; page ref bases from a
// look-back over pages (page order); active fine-tile flags.
// ===========================================================================

// The page's cell offsets (this thread's cell count c in, its exclusive offset
// out), the page's reference base from a look-back over pages in page order,
// its metadata and overflow flag (s_flags) and base (s_pbase). Ends with a
// block barrier.
__device__ __forceinline__ uint32_t page_prefix(const FrameParams& P, const PrepassArgs& A, uint32_t page,
                                                uint32_t pages, uint32_t c, uint32_t* s_warp, uint32_t& s_flags,
                                                uint32_t& s_pbase) {
    const size_t g = (size_t)page * kPageSize + threadIdx.x;
    uint32_t total;
    const uint32_t excl = block_exclusive_scan<256>(c, s_warp, total);
    A.offsets[g] = excl;
    uint32_t base = 0u;
    if (threadIdx.x < 32u) base = lb_exclusive_warp(A.lb_status, page, P.epoch, total, &A.counters->error, lb_limit(P),
                                              lb_withheld(P, kStagePrefix));
    if (threadIdx.x == 0) {
        fiber_fine_page_meta pm = A.page_meta[page];
        uint32_t flags = 0u;
        if (total > 0u && (uint64_t)base + total > (uint64_t)P.ref_capacity) {
            flags = 1u;
            atomicOr(&A.counters->overflow, 4u);
        }
        pm.seg_ref_base = total > 0u ? base : 0u;
        pm.seg_ref_count = flags ? 0u : total;
        pm.flags = flags;
        A.page_meta[page] = pm;
        s_flags = flags;
        s_pbase = base;
        if (page == pages - 1u) A.counters->refs = base + total;
    }
    __syncthreads();
    return excl;
}

// Fine tile lt of a page has `work` work items (non-empty cells) in it: kept per
// page, and added to the tile's if it is on screen (a tile with any is active:
// append_active_fine_tile, :2207-2238).
__device__ __forceinline__ void add_tile_work(const FrameParams& P, const PrepassArgs& A, uint32_t page, uint32_t tile,
                                              uint32_t lt, uint32_t work) {
    A.page_items[(size_t)page * 16u + lt] = (uint8_t)work;  // at most 16
    if (work == 0u) return;
    const uint32_t f = frustum_for_tile(P, tile);
    if (f == kInvalid) return;
    const fiber_frustum_desc& d = P.frusta[f];
    const uint32_t lc = tile - d.coarse_depth_tile_base;
    const uint32_t fx = (lc % d.coarse_tiles_x) * kCoarseExtent + lt % kCoarseExtent;
    const uint32_t fy = (lc / d.coarse_tiles_x) * kCoarseExtent + lt / kCoarseExtent;
    if (fx < ceil_div(d.screen_width, d.froxel_size_x) && fy < ceil_div(d.screen_height, d.froxel_size_y))
        atomicAdd(A.tile_work + (size_t)tile * 16u + lt, work);
}

// The same for the 16 fine tiles of a page whose cell counts are in shared
// memory.
__device__ __forceinline__ void page_active_tiles(const FrameParams& P, const PrepassArgs& A, uint32_t page,
                                                  const uint32_t* s_counts) {
    if (threadIdx.x >= 16u) return;
    const uint32_t lt = threadIdx.x;
    uint32_t work = 0u;
    for (uint32_t z = 0; z < kDepthSlices; ++z) work += s_counts[z * 16u + lt] > 0u ? 1u : 0u;
    add_tile_work(P, A, page, A.page_meta[page].coarse_tile_id, lt, work);
}

// A page's cell counts as one warp holds them: lane l has cells 8 l .. 8 l + 7
// (one fine depth slice, fine tiles 8 (l & 1) .. + 7), their sum, and how many
// fall in each of the cell sort's size classes, 16 bits each.
struct PageCells {
    uint32_t c[8], sum, small_quad, mid_large;
    __device__ __forceinline__ PageCells(const uint32_t* counts, uint32_t page, uint32_t lane) {
        const size_t g0 = (size_t)page * kPageSize + lane * 8u;
        const uint4 ca = *reinterpret_cast<const uint4*>(counts + g0);
        const uint4 cb = *reinterpret_cast<const uint4*>(counts + g0 + 4u);
        c[0] = ca.x; c[1] = ca.y; c[2] = ca.z; c[3] = ca.w;
        c[4] = cb.x; c[5] = cb.y; c[6] = cb.z; c[7] = cb.w;
        sum = small_quad = mid_large = 0u;
#pragma unroll
        for (uint32_t k = 0; k < 8u; ++k) {
            sum += c[k];
            if (c[k] >= 2u && c[k] <= kThreadSortMax) small_quad += 1u;
            if (c[k] > kThreadSortMax && c[k] <= kQuadSortMax) small_quad += 1u << 16;
            if (c[k] > kQuadSortMax && c[k] <= kGroupSortMax) mid_large += 1u;
            if (c[k] > kGroupSortMax && c[k] <= kWarpSortMax) mid_large += 1u << 16;
        }
    }
};

// csr: a page-CSR frame, where k_build_pages does this work unless the visit
// records went unused. A warp per group of pages, claimed in page order: the
// group's sums first (one look-back and one reservation of list room per
// group), then page by page the cell offsets from a warp scan, with no block
// barrier. A group is the pages' share of a resident warp, at most eight. Bound
// by the latency of the look-back chain and of the list counters' atomics, which
// a group pays once: with a page per warp it took 28 us on the tiny frame (184
// pages), 53 on the small, 119 on the medium (23,195) and 566 on the large one
// (133,640), now 16, 37, 59 and 262 (at most four pages: 16, 37, 70, 307).
constexpr uint32_t kPageGroup = 8;
__global__ void __launch_bounds__(256) k_prefix_pages(const FrameParams* __restrict__ Pp, PrepassArgs A, bool csr) {
    stamp_start(A.stamps, kStampPrefix);
    if (frame_failed(A.counters)) return;
    if (csr && !visits_unused(A)) return;
    const FrameParams& P = *Pp;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t pages = *((volatile uint32_t*)&A.counters->pages);
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t per = min(kPageGroup, ceil_div(pages, warps));
    for (;;) {
        uint32_t group = 0u;
        if (lane == 0u) group = atomicAdd(A.tile_counter, 1u);
        group = __shfl_sync(0xFFFFFFFFu, group, 0);
        if ((uint64_t)group * per >= pages) break;
        const uint32_t first = group * per, end = min(first + per, pages);
        uint32_t total = 0u, small_quad = 0u, mid_large = 0u;
#pragma unroll
        for (uint32_t u = 0; u < kPageGroup; ++u) {
            if (first + u >= end) break;
            const PageCells pc(A.counts, first + u, lane);
            total += pc.sum;
            small_quad += pc.small_quad;
            mid_large += pc.mid_large;
        }
        total = __reduce_add_sync(0xFFFFFFFFu, total);
        small_quad = __reduce_add_sync(0xFFFFFFFFu, small_quad);  // at most 8 x 256 per class
        mid_large = __reduce_add_sync(0xFFFFFFFFu, mid_large);
        uint32_t base = lb_exclusive_warp(A.lb_status, group, P.epoch, total, &A.counters->error, lb_limit(P),
                                          lb_withheld(P, kStagePrefix));
        if (lane == 0u && end == pages) A.counters->refs = base + total;
        // Room in the cell sort's lists (lane = class), for the whole group
        // unless some of its pages may lose their references.
        const bool tight = (uint64_t)base + total > (uint64_t)P.ref_capacity;
        uint32_t room = 0u;
        auto reserve = [&](uint32_t sq, uint32_t ml) {
            const uint32_t w = lane < 2u ? sq : ml, want = lane & 1u ? w >> 16 : w & 0xFFFFu;
            if (lane < 4u && want) room = atomicAdd(&A.counters->list_cells[lane], want);
        };
        if (!tight) reserve(small_quad, mid_large);
        uint32_t shadow = 0u;
#pragma unroll 1
        for (uint32_t page = first; page < end; ++page) {
            const PageCells pc(A.counts, page, lane);
            uint32_t x = pc.sum, y = pc.small_quad, z = pc.mid_large;
#pragma unroll
            for (uint32_t o = 1; o < 32u; o <<= 1) {
                const uint32_t xa = __shfl_up_sync(0xFFFFFFFFu, x, o), ya = __shfl_up_sync(0xFFFFFFFFu, y, o);
                const uint32_t za = __shfl_up_sync(0xFFFFFFFFu, z, o);
                if (lane >= o) { x += xa; y += ya; z += za; }
            }
            const uint32_t refs = __shfl_sync(0xFFFFFFFFu, x, 31), sq = __shfl_sync(0xFFFFFFFFu, y, 31);
            const uint32_t ml = __shfl_sync(0xFFFFFFFFu, z, 31);
            uint32_t e[8];  // exclusive offsets inside the page
            e[0] = x - pc.sum;
#pragma unroll
            for (uint32_t k = 1; k < 8u; ++k) e[k] = e[k - 1] + pc.c[k - 1];
            const size_t g0 = (size_t)page * kPageSize + lane * 8u;
            *reinterpret_cast<uint4*>(A.offsets + g0) = make_uint4(e[0], e[1], e[2], e[3]);
            *reinterpret_cast<uint4*>(A.offsets + g0 + 4u) = make_uint4(e[4], e[5], e[6], e[7]);
            const uint32_t page_base = base;
            base += refs;
            const bool fits = refs == 0u || (uint64_t)page_base + refs <= (uint64_t)P.ref_capacity;
            // seg_ref_base, seg_ref_count; coarse_tile_id, coarse_z, -, flags
            uint4* meta = reinterpret_cast<uint4*>(A.page_meta + page);
            uint4 m = meta[1];
            __syncwarp();
            if (lane == 0u) {
                if (!fits) atomicOr(&A.counters->overflow, 4u);
                meta[0] = make_uint4(refs > 0u ? page_base : 0u, fits ? refs : 0u, 0u, 0u);
                m.w = fits ? 0u : 1u;
                meta[1] = m;
            }
            // Each cell's first reference, for the fill.
            const uint32_t lost = fits ? 0u : kInvalid;
#pragma unroll
            for (uint32_t k = 0; k < 8u; ++k) e[k] += page_base;
            *reinterpret_cast<uint4*>(A.cursors + g0) = make_uint4(e[0] | lost, e[1] | lost, e[2] | lost, e[3] | lost);
            *reinterpret_cast<uint4*>(A.cursors + g0 + 4u) = make_uint4(e[4] | lost, e[5] | lost, e[6] | lost, e[7] | lost);
            // A page that lost its references lists no cells and no work.
            if (!fits) {
                if (lane < 16u) A.page_items[(size_t)page * 16u + lane] = 0u;
                continue;
            }
            if (tight) reserve(sq, ml);
            // The page's cells for k_sort_cells, in cell order: 2..8 references
            // in the small list, 9..16 in the quad one, 17..32 in the middle one,
            // up to 256 in the large one (a single reference is in order); longer
            // ones, few if any, are queued for k_sort_big_cells one by one.
            uint32_t ks = __shfl_sync(0xFFFFFFFFu, room, 0) + ((y - pc.small_quad) & 0xFFFFu);
            uint32_t kq = __shfl_sync(0xFFFFFFFFu, room, 1) + ((y - pc.small_quad) >> 16);
            uint32_t km = __shfl_sync(0xFFFFFFFFu, room, 2) + ((z - pc.mid_large) & 0xFFFFu);
            uint32_t kl = __shfl_sync(0xFFFFFFFFu, room, 3) + ((z - pc.mid_large) >> 16);
#pragma unroll
            for (uint32_t k = 0; k < 8u; ++k) {
                const uint32_t n = pc.c[k];
                const uint2 cell = make_uint2(e[k], n);
                if (n >= 2u && n <= kThreadSortMax) A.cells_small[ks++] = cell;
                else if (n > kThreadSortMax && n <= kQuadSortMax) A.cells_quad[kq++] = cell;
                else if (n > kQuadSortMax && n <= kGroupSortMax) A.cells_mid[km++] = cell;
                else if (n > kWarpSortMax) A.big_cells[atomicAdd(&A.counters->big_cells, 1u)] = cell;
                else if (n > kGroupSortMax) A.cells_large[kl++] = cell;
            }
            if (!tight && lane < 4u) {
                const uint32_t w = lane < 2u ? sq : ml;
                room += lane & 1u ? w >> 16 : w & 0xFFFFu;
            }
            // append_active_fine_tile (:2207-2238): each of the page's 16 fine
            // tiles that lies on screen gets its non-empty cells, the tile's work
            // items of this page. Fine tile 8 p + k is register k of the lanes of
            // parity p.
            uint32_t work = 0u;
#pragma unroll
            for (uint32_t k = 0; k < 8u; ++k) {
                const uint32_t nonempty = __ballot_sync(0xFFFFFFFFu, pc.c[k] > 0u);
                if (k == (lane & 7u)) work = (uint32_t)__popc(nonempty & ((lane & 8u) ? 0xAAAAAAAAu : 0x55555555u));
            }
            if (lane < 16u) add_tile_work(P, A, page, m.x, lane, work);
            if (m.x >= P.camera_tile_end) shadow += refs;
        }
        if (lane == 0u && shadow) atomicAdd(&A.counters->shadow_refs, (unsigned long long)shadow);
    }
}

// ===========================================================================
// K13: ordered compaction of the active fine tiles (those with work items) into
// tile runs, and the base of each one's work items: two prefix sums over the same 1024 tiles a
// block, whose look-backs (active tiles, work items) run in two warps at once.
// ===========================================================================
__global__ void __launch_bounds__(kScanThreads) k_compact_active(const FrameParams* __restrict__ Pp, PrepassArgs A,
                                                                unsigned long long* lb_work) {
    stamp_start(A.stamps, kStampCompact);
    if (frame_failed(A.counters)) return;
    const FrameParams& P = *Pp;
    __shared__ uint32_t s_tile, s_base, s_work;
    __shared__ uint32_t s_warp[33];
    const uint32_t n = P.total_coarse_tiles * 16u;
    const uint32_t cam_end = P.camera_tile_end * 16u;
    const uint32_t per_tile = kScanThreads * kScanItems;
    const uint32_t n_tiles = ceil_div(n, per_tile);
    bool worked = blockIdx.x == 0u;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(A.tile_counter, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= n_tiles) break;
        worked = true;
        const uint32_t e0 = tile * per_tile + threadIdx.x * kScanItems;  // n is a multiple of 16
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (e0 < n) w = *reinterpret_cast<const uint4*>(A.tile_work + e0);
        const uint32_t work[kScanItems] = {w.x, w.y, w.z, w.w};
        uint32_t cnt = 0u, sum = 0u;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            cnt += work[j] ? 1u : 0u;
            sum += work[j];
        }
        uint32_t total, total_work;
        const uint32_t excl = block_exclusive_scan<kScanThreads>(cnt, s_warp, total);
        const uint32_t excl_work = block_exclusive_scan<kScanThreads>(sum, s_warp, total_work);
        // Tiles of cameras come first and whole blocks of four items share a
        // coarse tile's row, so a thread's four are all a camera's or none.
        uint32_t cam = e0 < cam_end ? cnt : 0u;
        for (int o = 16; o > 0; o >>= 1) cam += __shfl_xor_sync(0xFFFFFFFFu, cam, o);
        if ((threadIdx.x & 31) == 0 && cam) atomicAdd(&A.counters->camera_active, cam);
        if (threadIdx.x < 32u) {
            const uint32_t base = lb_exclusive_warp(A.lb_status, tile, P.epoch, total, &A.counters->error, lb_limit(P),
                                                    lb_withheld(P, kStageActive));
            if (threadIdx.x == 0) {
                s_base = base;
                if (tile == n_tiles - 1u) A.counters->active_tiles = base + total;
            }
        } else if (threadIdx.x < 64u) {
            const uint32_t base = lb_exclusive_warp(lb_work, tile, P.epoch, total_work, &A.counters->error, lb_limit(P),
                                                    lb_withheld(P, kStageEmit));
            if (threadIdx.x == 32u) {
                s_work = base;
                if (tile == n_tiles - 1u) A.counters->work_items = base + total_work;
            }
        }
        __syncthreads();
        uint32_t idx = s_base + excl, at = s_work + excl_work;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            if (work[j] == 0u) continue;
            const uint32_t e = e0 + j, ct = e / 16u, lt = e % 16u;
            const uint32_t f = frustum_for_tile(P, ct);
            const fiber_frustum_desc& d = P.frusta[f < P.F ? f : 0];
            const uint32_t lc = ct - d.coarse_depth_tile_base;
            const uint32_t fx = (lc % d.coarse_tiles_x) * kCoarseExtent + lt % kCoarseExtent;
            const uint32_t fy = (lc / d.coarse_tiles_x) * kCoarseExtent + lt / kCoarseExtent;
            const uint32_t screen_tile = fy * ceil_div(d.screen_width, d.froxel_size_x) + fx;
            A.active_list[idx] = e;
            A.tile_slot[e] = make_uint2(idx, at);
            // The tile's run; k_emit adds up its load.
            uint4* run = reinterpret_cast<uint4*>(A.runs + idx);
            run[0] = make_uint4(at, work[j], f, screen_tile);
            run[1] = make_uint4(0u, 0u, 0u, 0u);
            ++idx;
            at += work[j];
        }
        __syncthreads();
    }
    if (worked && threadIdx.x == 0u) stamp_end(A.stamps, kStampCompactEnd);
}

// ===========================================================================
// K14: emit raster work per active fine tile (256 depth slots = 16 coarse z x
// 16 fine z, near to far). The canonical order inside each cell (projected
// depth key descending, then instance, then segment) is made by k_sort_cells.
//
// Sixteen lanes per page, one per fine tile: the page's 256 cell counts and
// offsets are 16 rows (fine z) of 16 fine tiles, so every row is one coalesced
// 64 B read, and each lane writes its own items behind those of the nearer
// pages of its coarse tile (page_items) from the base the compaction gave it.
// Bound by the scattered 32 B item writes. One tile per warp with a look-back
// per tile, 4 B loads 64 B apart and items stored word by word took 0.27 ms on
// the medium frame (3.1 M items, 62,894 tiles) and 4.7 ms on the large one
// (22.5 M); sixteen lanes per coarse tile left the dense tiles' warps behind.
// ===========================================================================
__global__ void __launch_bounds__(256) k_emit(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    stamp_start(A.stamps, kStampEmit);
    if (frame_failed(A.counters)) return;
    const uint32_t lt = threadIdx.x & 15u, half = threadIdx.x & 16u;
    const uint32_t pages = *((volatile uint32_t*)&A.counters->pages);
    const uint32_t halves = gridDim.x * (blockDim.x >> 4);
    const uint32_t first_shadow = *((volatile uint32_t*)&A.counters->camera_active);
    const uint32_t limit = heavy_limit(A.counters, A.shadow_blocks);
    const uint32_t work_capacity = Pp->work_capacity;
    // Every lane of a warp takes every round.
    for (uint32_t p0 = 0; p0 < pages; p0 += halves) {
        const uint32_t page = p0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 4);
        fiber_fine_page_meta pm{};
        if (page < pages) pm = A.page_meta[page];
        const bool has = pm.seg_ref_count > 0u && pm.flags == 0u;
        const size_t slot_at = (size_t)pm.coarse_tile_id * 16u + lt;
        const uint32_t handle = has ? A.page_table[slot_at] : 0u;  // lane z: the page of coarse slice z
        const uint32_t n_work = has ? A.tile_work[slot_at] : 0u;
        const uint2 slot = n_work ? A.tile_slot[slot_at] : make_uint2(0u, 0u);
        uint32_t dst = slot.y;
#pragma unroll
        for (uint32_t z = 1; z < kDepthSlices; ++z) {
            const uint32_t h = __shfl_sync(0xFFFFFFFFu, handle, (int)(half + z));
            if (z > pm.coarse_z && h != 0u && h != kMarked) dst += A.page_items[(size_t)(h - 1u) * 16u + lt];
        }
        if (n_work == 0u) continue;
        const fiber_coarse_depth_lut_entry lut = A.lut[(size_t)pm.coarse_tile_id * kDepthSlices + pm.coarse_z];
        const uint4 run = *reinterpret_cast<const uint4*>(A.runs + slot.x);  // base, items, frustum, screen tile
        const uint32_t* cnt = A.counts + (size_t)page * kPageSize + lt;
        const uint32_t* off = A.offsets + (size_t)page * kPageSize + lt;
        uint32_t load = 0u;
#pragma unroll
        for (int h = 1; h >= 0; --h) {
            uint32_t c[8], o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                c[j] = cnt[(h * 8 + j) * 16];
                o[j] = off[(h * 8 + j) * 16];
            }
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                if (c[j] == 0u) continue;
                const uint32_t fz = (uint32_t)(h * 8 + j);
                const uint32_t dkey = lut.virtual_count_q == 0u
                                          ? fz
                                          : lut.virtual_start_q + (lut.virtual_count_q * fz) / kDepthSlices;
                if (dst < work_capacity) {
                    uint4* item = reinterpret_cast<uint4*>(A.work + dst);
                    item[0] = make_uint4(pm.seg_ref_base + o[j], c[j], run.z, run.w);
                    item[1] = make_uint4(dkey, c[j], page, fz * 16u + lt);
                } else {
                    atomicOr(&A.counters->overflow, 8u);
                }
                ++dst;
                load += c[j];
            }
        }
        if (load == 0u) continue;
        const uint32_t before = atomicAdd(&A.runs[slot.x].load_score, load);
        // The page that takes a shadow run over the limit lists it.
        if (slot.x >= first_shadow && before < limit && before + load >= limit)
            A.heavy_list[atomicAdd(&A.counters->heavy_runs, 1u)] = slot.x;
    }
    if ((blockIdx.x == 0u || blockIdx.x * (blockDim.x >> 4) < pages) && threadIdx.x == 0u)
        stamp_end(A.stamps, kStampEmitEnd);
}

// A cell's entries are binning task indices; the canonical order is by depth key
// descending, then instance, then segment. Tasks are in (frustum, instance,
// strand, segment) order, so where every instance's strands follow one another
// in its index slab (k_fine checks every strand against the one before it) the
// task index orders instance and segment, and an entry is one 64-bit word
// (0x1FFFF - depth key) << 32 | task that sorts alone (ByTask). Otherwise
// (strands in any order or sharing indices) the word is the full key of
// ref_sort_key and the task moves beside it (ByRecord). Depth keys repeat inside
// most cells (a fine cell spans some 100 to 500 of their steps), so the tie
// order has to be in the word.
struct ByTask {
    unsigned long long w;
    __device__ __forceinline__ void load(const PrepassArgs& A, uint32_t task) {
        w = ((unsigned long long)(0x1FFFFu - A.task_key[task]) << 32) | task;
    }
    __device__ __forceinline__ void pad() { w = ~0ull; }
    __device__ __forceinline__ uint32_t task() const { return (uint32_t)w; }
    __device__ __forceinline__ ByTask other(int mask) const { return ByTask{__shfl_xor_sync(0xFFFFFFFFu, w, mask)}; }
};
struct ByRecord {
    unsigned long long w;
    uint32_t t;
    __device__ __forceinline__ void load(const PrepassArgs& A, uint32_t task) {
        const uint4 r = reinterpret_cast<const uint4*>(A.task_rec)[(size_t)kTaskRec * task + 2u];
        w = ref_sort_key(A.task_key[task], r.x, r.y);
        t = task;
    }
    __device__ __forceinline__ void pad() { w = ~0ull; t = 0u; }
    __device__ __forceinline__ uint32_t task() const { return t; }
    __device__ __forceinline__ ByRecord other(int mask) const {
        return ByRecord{__shfl_xor_sync(0xFFFFFFFFu, w, mask), __shfl_xor_sync(0xFFFFFFFFu, t, mask)};
    }
};
// Compare and exchange by selects: as branches the exchanges diverged and most
// of the sort's time was branch resolution (291 M -> 105 M warp
// instructions, 0.42 -> 0.19 ms for the 23 M references of the medium frame).
__device__ __forceinline__ ByTask pick(bool p, ByTask a, ByTask b) { return ByTask{p ? a.w : b.w}; }
__device__ __forceinline__ ByRecord pick(bool p, ByRecord a, ByRecord b) {
    return ByRecord{p ? a.w : b.w, p ? a.t : b.t};
}
// Whether the lane that keeps the smaller (or the larger) of a pair takes the
// other lane's. Words of ByTask differ or are both padding; keys of ByRecord
// repeat where strands share segments, and then both lanes keep their own.
__device__ __forceinline__ bool takes_other(ByTask o, ByTask own, bool smaller) { return (o.w < own.w) == smaller; }
__device__ __forceinline__ bool takes_other(ByRecord o, ByRecord own, bool smaller) {
    return smaller ? o.w < own.w : o.w > own.w;
}
template <class E>
__device__ __forceinline__ void order(E& a, E& b, bool up) {
    const bool exchange = (a.w > b.w) == up;
    const E x = pick(exchange, b, a), y = pick(exchange, a, b);
    a = x;
    b = y;
}

// A group of G lanes (G-aligned inside the warp) sorts up to G x R entries in
// registers: element e = (lane % G) R + r, a bitonic network over G R words.
// Strides below R compare registers of one lane; larger strides exchange the
// same register with lane ^ (stride / R), inside the group. Every lane of the
// warp calls it.
template <class E, int G, int R>
__device__ __forceinline__ void group_sort(E* k, int gl) {
#pragma unroll
    for (int size = 2; size <= G * R; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= R) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int e = gl * R + r;
                    const E o = k[r].other(stride / R);
                    const bool up = (e & size) == 0;
                    const bool lower = (e & stride) == 0;
                    k[r] = pick(takes_other(o, k[r], lower == up), o, k[r]);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if ((r ^ stride) > r) order(k[r], k[r ^ stride], ((gl * R + r) & size) == 0);
            }
        }
    }
}
// Up to G R entries of a cell from `from` on (any order will do to begin with:
// the loads are coalesced).
template <class E, int G, int R>
__device__ __forceinline__ void group_load(E* k, const PrepassArgs& A, uint32_t from, uint32_t n, int gl) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t e = (uint32_t)(r * G + gl);
        k[r].pad();
        if (e < n) k[r].load(A, A.ref_task[from + e]);
    }
}
// One cell of up to G R references per group; padding sorts last, groups without
// a cell (n = 0) take part with padding.
template <class E, int G, int R>
__device__ __forceinline__ void group_sort_cell(const PrepassArgs& A, uint32_t base, uint32_t n, int lane) {
    const int gl = lane & (G - 1);
    E k[R];
    group_load<E, G, R>(k, A, base, n, gl);
    group_sort<E, G, R>(k, gl);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t e = (uint32_t)gl * R + r;
        if (e < n) A.ref_task[base + e] = k[r].task();
    }
}

template <class E>
__device__ __forceinline__ void warp_sort_any(const PrepassArgs& A, uint32_t base, uint32_t n, int lane) {
    if (n <= 32u) group_sort_cell<E, 32, 1>(A, base, n, lane);
    else if (n <= 64u) group_sort_cell<E, 32, 2>(A, base, n, lane);
    else if (n <= 128u) group_sort_cell<E, 32, 4>(A, base, n, lane);
    else group_sort_cell<E, 32, 8>(A, base, n, lane);
}

// Batcher's odd-even merge network for 8 entries in registers.
template <class E>
__device__ __forceinline__ void sort8(E* k) {
    auto cas = [&](int a, int b) { order(k[a], k[b], true); };
    cas(0, 1); cas(2, 3); cas(4, 5); cas(6, 7);
    cas(0, 2); cas(1, 3); cas(4, 6); cas(5, 7);
    cas(1, 2); cas(5, 6);
    cas(0, 4); cas(1, 5); cas(2, 6); cas(3, 7);
    cas(2, 4); cas(3, 5);
    cas(1, 2); cas(3, 4); cas(5, 6);
}

// One thread sorts a cell of at most 8 references in registers: Batcher's
// odd-even merge network for 8 inputs (19 comparators); padding sorts last.
template <class E>
__device__ __forceinline__ void thread_sort_cell(const PrepassArgs& A, uint32_t base, uint32_t n) {
    E k[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        k[e].pad();
        if ((uint32_t)e < n) k[e].load(A, A.ref_task[base + e]);
    }
    sort8(k);
#pragma unroll
    for (int e = 0; e < 8; ++e)
        if ((uint32_t)e < n) A.ref_task[base + e] = k[e].task();
}

// A cell longer than a warp sort is queued for k_sort_big_cells (page CSR).
__device__ __forceinline__ void queue_big_cell(const PrepassArgs& A, uint32_t b, uint32_t n, uint32_t lane) {
    if (lane == 0u) {
        const uint32_t slot = atomicAdd(&A.counters->big_cells, 1u);
        A.big_cells[slot] = make_uint2(b, n);
    }
}

// 32 consecutive small cells at once. k_prefix_pages lists a page's small
// cells together, in cell order, so their references usually form one span
// [lo, hi) of the reference array (holes: the page's other cells). When the
// span fits kSortSpan, each lane loads every 32nd entry of the span (8
// independent loads, then 8 independent key gathers) and parks the words in
// shared memory; each lane then sorts its own cell there with sort8 and the
// warp writes the span's own entries back coalesced. Otherwise each lane sorts
// its cell alone (as it does for entries that carry their task beside the word).
constexpr uint32_t kSortSpan = 256;
constexpr uint32_t kSortPerLane = kSortSpan / 32u;
struct SortSpanSmem {
    ByTask entry[kSortSpan];
    uint8_t own[kSortSpan];
};

__device__ __forceinline__ void warp_sort_small_cells(const PrepassArgs& A, uint32_t i0, uint32_t n_small,
                                                      uint32_t lane, SortSpanSmem* /*sm*/, ByRecord) {
    if (i0 + lane >= n_small) return;
    const uint2 e = A.cells_small[i0 + lane];
    thread_sort_cell<ByRecord>(A, e.x, e.y);
}
__device__ __forceinline__ void warp_sort_small_cells(const PrepassArgs& A, uint32_t i0, uint32_t n_small,
                                                      uint32_t lane, SortSpanSmem* smp, ByTask) {
    using E = ByTask;
    SortSpanSmem& sm = *smp;
    const uint32_t i = i0 + lane;
    const bool has = i < n_small;
    const uint2 e = has ? A.cells_small[i] : make_uint2(0u, 0u);
    uint32_t lo = has ? e.x : 0xFFFFFFFFu, hi = has ? e.x + e.y : 0u;
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if (hi <= lo || hi - lo > kSortSpan) {
        if (has) thread_sort_cell<E>(A, e.x, e.y);
        return;
    }
    const uint32_t span = hi - lo;
#pragma unroll
    for (uint32_t m = 0; m < kSortPerLane; ++m) sm.own[lane + 32u * m] = 0u;
    __syncwarp();
    if (has)
        for (uint32_t r = 0; r < e.y; ++r) sm.own[e.x - lo + r] = 1u;
    __syncwarp();
    uint32_t tk[kSortPerLane];
#pragma unroll
    for (uint32_t m = 0; m < kSortPerLane; ++m) {
        const uint32_t j = lane + 32u * m;
        tk[m] = (j < span && sm.own[j]) ? A.ref_task[lo + j] : kInvalid;
    }
    E en[kSortPerLane];
#pragma unroll
    for (uint32_t m = 0; m < kSortPerLane; ++m) {
        en[m].pad();
        if (tk[m] != kInvalid) en[m].load(A, tk[m]);
    }
#pragma unroll
    for (uint32_t m = 0; m < kSortPerLane; ++m) sm.entry[lane + 32u * m] = en[m];
    __syncwarp();
    if (has) {
        const uint32_t b = e.x - lo;
#pragma unroll
        for (uint32_t r = 0; r < 8u; ++r) {
            en[r].pad();
            if (r < e.y) en[r] = sm.entry[b + r];
        }
        sort8(en);
#pragma unroll
        for (uint32_t r = 0; r < 8u; ++r)
            if (r < e.y) sm.entry[b + r] = en[r];
    }
    __syncwarp();
#pragma unroll
    for (uint32_t m = 0; m < kSortPerLane; ++m) {
        const uint32_t j = lane + 32u * m;
        if (tk[m] != kInvalid) A.ref_task[lo + j] = sm.entry[j].task();
    }
    __syncwarp();
}

template <class E>
__device__ __forceinline__ void sort_cells(const PrepassArgs& A, SortSpanSmem* s_span) {
    const uint32_t lane = threadIdx.x & 31u;
    const volatile uint32_t* n_cells = A.counters->list_cells;
    const uint32_t n_small = n_cells[kListSmall], n_quad = n_cells[kListQuad];
    const uint32_t n_mid = n_cells[kListMid], n_large = n_cells[kListLarge];
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; i0 < n_small; i0 += stride)
        warp_sort_small_cells(A, i0, n_small, lane, s_span, E{});
    const uint32_t warps = stride >> 5;
    // Cells of 9..16 references: eight per warp, four lanes each.
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 8u < n_quad; w += warps) {
        const uint32_t ci = w * 8u + (lane >> 2);
        const uint2 e = ci < n_quad ? A.cells_quad[ci] : make_uint2(0u, 0u);
        group_sort_cell<E, 4, 4>(A, e.x, e.y, (int)lane);
    }
    // Cells of 17..32: four per warp, eight lanes each.
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 4u < n_mid; w += warps) {
        const uint32_t ci = w * 4u + (lane >> 3);
        const uint2 e = ci < n_mid ? A.cells_mid[ci] : make_uint2(0u, 0u);
        group_sort_cell<E, 8, 4>(A, e.x, e.y, (int)lane);
    }
    // Cells of more than 32: a warp per cell.
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n_large; w += warps) {
        const uint2 e = A.cells_large[w];
        warp_sort_any<E>(A, e.x, e.y, (int)lane);
    }
}

// Canonical order inside every cell, in place, after the fill, over the cell
// lists k_prefix_pages made: a warp per 32 cells of 2..8 references (a lane per
// cell), eight cells of 9..16 references per warp (four lanes each), four of
// 17..32 (eight lanes each), then a warp per larger cell of up to 256. Bound by the networks' 64-bit compares and selects (ALU pipe
// 71 % busy). An earlier form wrote 20 B of reference, key and task per entry and
// sorted a word beside its task by branches: 0.57 -> 0.19 ms for the medium frame,
// 11.0 -> 4.3 ms for the large frame's 349 M references. Frames with strands out
// of order (ByRecord: 16 B more gathered per entry, small cells one by one) take
// about 0.38 and 10.4 ms.
__global__ void __launch_bounds__(256, 5) k_sort_cells(PrepassArgs A) {
    stamp_start(A.stamps, kStampSort);
    if (frame_failed(A.counters)) return;
    __shared__ SortSpanSmem s_span[8];
    if (*((volatile uint32_t*)&A.counters->seg_unordered) == 0u) sort_cells<ByTask>(A, s_span + (threadIdx.x >> 5));
    else sort_cells<ByRecord>(A, s_span + (threadIdx.x >> 5));
}

// ===========================================================================
// Page-CSR backend (FineBinningBackend::PageCsr: prefix_page_candidates,
// scatter_page_candidates and build_fine_pages_csr, strand_prepass.wgsl:
// 1992-2049, 2387-2507). The reference lists each page's candidate tasks and
// traces every task again inside the page's workgroup; here the visit
// records of k_visit already hold every (page, cell, task) visit, so they are
// grouped by page (count, scan, scatter) and one block per page counts its
// cells in shared memory, takes the page's reference base in page order (as
// k_prefix_pages), fills the page's slots and sorts its cells while they are
// in L2. The results are the canonical ones of the default backend.
// ===========================================================================

// Visits per page; each visit keeps its rank inside its page. Lanes of a warp
// that hit the same page share one atomic.
__global__ void __launch_bounds__(256) k_page_count(PrepassArgs A) {
    stamp_start(A.stamps, kStampCount);
    if (frame_failed(A.counters)) return;
    if (visits_unused(A)) return;
    const uint32_t n = (uint32_t)*((volatile unsigned long long*)&A.counters->visits);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t r0 = blockIdx.x * blockDim.x; r0 < n; r0 += gridDim.x * blockDim.x) {
        const uint32_t r = r0 + threadIdx.x;
        uint32_t page = kInvalid, cell = 0u;
        if (r < n) {
            const uint32_t rec = A.visit_rec[r];
            const uint32_t h = A.page_table[rec >> 8];
            if (h != 0u && h != kMarked) {
                page = h - 1u;
                cell = rec & 0xFFu;
            }
        }
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, page);
        const uint32_t leader = (uint32_t)(__ffs(peers) - 1);
        uint32_t base = 0u;
        if (page != kInvalid && lane == leader) base = atomicAdd(A.page_nvis + page, (uint32_t)__popc(peers));
        base = __shfl_sync(0xFFFFFFFFu, base, (int)leader);
        if (r < n) {
            A.visit_rec[r] = page == kInvalid ? kInvalid : (page << 8) | cell;
            A.visit_rank[r] = base + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        }
    }
}

// Exclusive scan of the per-page visit counts (one block).
__global__ void __launch_bounds__(1024) k_page_scan(PrepassArgs A) {
    if (frame_failed(A.counters)) return;
    if (visits_unused(A)) return;
    __shared__ uint32_t s_warp[33];
    __shared__ uint32_t s_carry;
    const uint32_t pages = *((volatile uint32_t*)&A.counters->pages);
    if (threadIdx.x == 0) s_carry = 0u;
    __syncthreads();
    for (uint32_t b = 0; b < pages; b += 1024u) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < pages ? A.page_nvis[i] : 0u;
        uint32_t total;
        const uint32_t ex = block_exclusive_scan<1024>(v, s_warp, total);
        if (i < pages) A.page_vbase[i] = s_carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) s_carry += total;
        __syncthreads();
    }
}

// Visits into their page's bucket: (task, cell) at page base + rank.
__global__ void __launch_bounds__(256) k_page_scatter(PrepassArgs A) {
    if (frame_failed(A.counters)) return;
    if (visits_unused(A)) return;
    const uint32_t n = (uint32_t)*((volatile unsigned long long*)&A.counters->visits);
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const uint32_t rec = A.visit_rec[r];
        if (rec == kInvalid) continue;
        A.page_bucket[A.page_vbase[rec >> 8] + A.visit_rank[r]] = make_uint2(A.visit_task[r], rec & 0xFFu);
    }
}

// One block per page, in page order (the look-back of the page bases).
__global__ void __launch_bounds__(256, 3) k_build_pages(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    stamp_start(A.stamps, kStampFill);
    if (frame_failed(A.counters)) return;
    if (visits_unused(A)) return;
    const FrameParams& P = *Pp;
    __shared__ uint32_t s_tile, s_flags, s_pbase, s_nlarge;
    __shared__ uint32_t s_warp[33];
    __shared__ uint32_t s_counts[kPageSize], s_off[kPageSize], s_cur[kPageSize];
    __shared__ uint16_t s_large[kPageSize];
    const uint32_t pages = *((volatile uint32_t*)&A.counters->pages);
    const bool by_task = *((volatile uint32_t*)&A.counters->seg_unordered) == 0u;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (;;) {
        if (threadIdx.x == 0) {
            s_tile = atomicAdd(A.tile_counter, 1u);
            s_nlarge = 0u;
        }
        s_counts[threadIdx.x] = 0u;
        s_cur[threadIdx.x] = 0u;
        __syncthreads();
        const uint32_t page = s_tile;
        if (page >= pages) break;
        const uint32_t n = A.page_nvis[page], vb = A.page_vbase[page];
        for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) atomicAdd(&s_counts[A.page_bucket[vb + e].y], 1u);
        __syncthreads();
        const uint32_t c = s_counts[threadIdx.x];
        A.counts[(size_t)page * kPageSize + threadIdx.x] = c;
        const uint32_t excl = page_prefix(P, A, page, pages, c, s_warp, s_flags, s_pbase);
        s_off[threadIdx.x] = excl;
        if (s_flags == 0u) {
            __syncthreads();
            const uint32_t pbase = s_pbase;
            // Fill: the task index of every visit into its slot (the slots of
            // one page are a few KB, so these writes and the sort's reads stay
            // in L2); the order inside a cell is fixed by the sort below.
            for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) {
                const uint2 v = A.page_bucket[vb + e];
                A.ref_task[pbase + s_off[v.y] + atomicAdd(&s_cur[v.y], 1u)] = v.x;
            }
            __syncthreads();
            if (c >= 2u && c <= kThreadSortMax) {
                if (by_task) thread_sort_cell<ByTask>(A, pbase + excl, c);
                else thread_sort_cell<ByRecord>(A, pbase + excl, c);
            } else if (c > kThreadSortMax) s_large[atomicAdd(&s_nlarge, 1u)] = (uint16_t)threadIdx.x;
            __syncthreads();
            const uint32_t nl = s_nlarge;
            for (uint32_t i = warp; i < nl; i += blockDim.x >> 5) {
                const uint32_t cell = s_large[i], cb = pbase + s_off[cell], cn = s_counts[cell];
                if (cn > kWarpSortMax) queue_big_cell(A, cb, cn, lane);
                else if (by_task) warp_sort_any<ByTask>(A, cb, cn, (int)lane);
                else warp_sort_any<ByRecord>(A, cb, cn, (int)lane);
            }
            page_active_tiles(P, A, page, s_counts);
            if (threadIdx.x == 0 && A.page_meta[page].coarse_tile_id >= P.camera_tile_end)
                atomicAdd(&A.counters->shadow_refs, (unsigned long long)A.page_meta[page].seg_ref_count);
        } else if (threadIdx.x < 16u) {
            A.page_items[(size_t)page * 16u + threadIdx.x] = 0u;
        }
        __syncthreads();
    }
}

// Large cells: one block per cell. Bitonic sort in the ascending-only form
// (each stage starts with a "flip" compare i <-> i ^ (size - 1)), which never
// moves the virtual +inf padding below n, so the padding needs no storage.
// Up to kBigSmem entries sort in shared memory; longer cells sort in place in
// global memory with the same network.
constexpr uint32_t kBigSmem = 8192;
constexpr size_t kBigSmemBytes = kBigSmem * (sizeof(unsigned long long) + sizeof(uint32_t));

__device__ __forceinline__ void big_load(const PrepassArgs& A, uint32_t base, uint32_t n, uint32_t i,
                                         unsigned long long& k, uint32_t& m) {
    if (i < n) {
        ByRecord r;
        r.load(A, A.ref_task[base + i]);
        k = r.w;
        m = r.t;
    } else {
        k = ~0ull;
        m = 0u;
    }
}
// Pair t of a stage: (i, j) with i < j.
__device__ __forceinline__ void bitonic_pair(uint32_t t, uint32_t size, uint32_t stride, bool flip, uint32_t& i,
                                             uint32_t& j) {
    if (flip) {
        uint32_t half = size >> 1, blk = t / half, off = t % half;
        i = blk * size + off;
        j = blk * size + size - 1u - off;
    } else {
        i = (t / stride) * 2u * stride + (t % stride);
        j = i + stride;
    }
}

// A block of 256 threads sorts a cell of up to 256 S references: the warps sort
// chunks of 32 min(S, 8) in registers, then the sorted runs merge pairwise in
// shared memory, each thread S outputs of a level from the point where its first
// one splits the two runs (merge path: Odeh, Green, Mwassi, Shmueli, Birk 2012).
// A level's outputs stay in registers until every thread has read its inputs.
template <uint32_t S>
__device__ __forceinline__ void merge_sort_cell(const PrepassArgs& A, uint32_t base, uint32_t n, unsigned long long* s) {
    constexpr uint32_t R = S < 8u ? S : 8u, chunk = 32u * R;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t padded = ceil_div(n, chunk) * chunk;  // padding sorts last
    for (uint32_t c = (threadIdx.x >> 5) * chunk; c < padded; c += chunk * 8u) {
        ByTask k[R];
        group_load<ByTask, 32, R>(k, A, base + c, min(n - c, chunk), (int)lane);
        group_sort<ByTask, 32, R>(k, (int)lane);
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) s[c + lane * R + r] = k[r].w;
    }
    __syncthreads();
    const uint32_t at = threadIdx.x * S;
    for (uint32_t len = chunk; len < padded; len <<= 1) {
        unsigned long long out[S];
        if (at < padded) {
            const uint32_t a0 = at / (2u * len) * (2u * len), d = at - a0;
            const uint32_t a_n = min(len, padded - a0), b_n = min(len, padded - a0 - a_n);
            const unsigned long long *a = s + a0, *b = a + a_n;
            uint32_t lo = d > b_n ? d - b_n : 0u, hi = min(d, a_n);
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a[mid] <= b[d - 1u - mid]) lo = mid + 1u;
                else hi = mid;
            }
            uint32_t i = lo, j = d - lo;
#pragma unroll
            for (uint32_t o = 0; o < S; ++o) {
                // Past a run's end its word is the padding (the other run's are taken first).
                const unsigned long long x = i < a_n ? a[i] : ~0ull, y = j < b_n ? b[j] : ~0ull;
                const bool from_a = i < a_n && (x <= y || j >= b_n);
                out[o] = from_a ? x : y;
                i += from_a ? 1u : 0u;
                j += from_a ? 0u : 1u;
            }
        }
        __syncthreads();
        if (at < padded) {
#pragma unroll
            for (uint32_t o = 0; o < S; ++o) s[at + o] = out[o];
        }
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) A.ref_task[base + i] = (uint32_t)s[i];
    __syncthreads();
}

// Cells of more than 256 references, a block each. Up to kBigSmem references
// whose order is the task order (ByTask) take the merge sort: its levels read
// and write a word once where the bitonic network, which sorts the other cells,
// takes log2(n) steps with a barrier each. Cell sort of frames with 2,809 cells
// (1.3 M references), 2,894 (1.6 M) and 1,376 of up to 4,805 (1.1 M): 333, 403 and
// 493 -> 121, 126 and 145 us.
__global__ void __launch_bounds__(256) k_sort_big_cells(PrepassArgs A) {
    if (frame_failed(A.counters)) return;
    const bool by_task = *((volatile uint32_t*)&A.counters->seg_unordered) == 0u;
    extern __shared__ unsigned char s_raw[];
    unsigned long long* s_k = reinterpret_cast<unsigned long long*>(s_raw);
    uint32_t* s_m = reinterpret_cast<uint32_t*>(s_raw + kBigSmem * sizeof(unsigned long long));
    const uint32_t n_cells = *((volatile uint32_t*)&A.counters->big_cells);
    for (uint32_t c = blockIdx.x; c < n_cells; c += gridDim.x) {
        const uint2 bc = A.big_cells[c];
        const uint32_t base = bc.x, n = bc.y;
        if (by_task && n <= kBigSmem) {
            unsigned long long* words = reinterpret_cast<unsigned long long*>(s_raw);
            if (n <= 512u) merge_sort_cell<2>(A, base, n, words);
            else if (n <= 1024u) merge_sort_cell<4>(A, base, n, words);
            else if (n <= 2048u) merge_sort_cell<8>(A, base, n, words);
            else merge_sort_cell<32>(A, base, n, words);
            continue;
        }
        uint32_t np = 1;
        while (np < n) np <<= 1;
        const bool in_smem = np <= kBigSmem;
        if (in_smem) {
            for (uint32_t i = threadIdx.x; i < np; i += blockDim.x) big_load(A, base, n, i, s_k[i], s_m[i]);
            __syncthreads();
        }
        for (uint32_t size = 2; size <= np; size <<= 1) {
            for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
                const bool flip = stride == (size >> 1);
                for (uint32_t t = threadIdx.x; t < np / 2u; t += blockDim.x) {
                    uint32_t i, j;
                    bitonic_pair(t, size, stride, flip, i, j);
                    if (in_smem) {
                        unsigned long long ki = s_k[i], kj = s_k[j];
                        if (ki > kj) {
                            s_k[i] = kj; s_k[j] = ki;
                            uint32_t tm = s_m[i]; s_m[i] = s_m[j]; s_m[j] = tm;
                        }
                    } else if (j < n) {
                        unsigned long long ki, kj;
                        uint32_t mi, mj;
                        big_load(A, base, n, i, ki, mi);
                        big_load(A, base, n, j, kj, mj);
                        if (ki > kj) {
                            A.ref_task[base + i] = mj;
                            A.ref_task[base + j] = mi;
                        }
                    }
                }
                __syncthreads();
            }
        }
        if (in_smem) {
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) A.ref_task[base + i] = s_m[i];
            __syncthreads();
        }
    }
    if ((blockIdx.x == 0u || blockIdx.x < n_cells) && threadIdx.x == 0u) stamp_end(A.stamps, kStampSortEnd);
}

// finalize_telemetry (:2145-2188): totals, per-page candidate statistics and
// the per-frustum page, reference and raster-run sums, after the emit. The
// candidate count of a page is the number of tasks that marked its slot.
__global__ void __launch_bounds__(256) k_telemetry(const FrameParams* __restrict__ Pp, PrepassArgs A) {
    const FrameParams& P = *Pp;
    uint32_t* tel = A.tel;
    const uint32_t pages = min(*((volatile uint32_t*)&A.counters->pages), P.page_capacity);
    const uint32_t runs = *((volatile uint32_t*)&A.counters->active_tiles);
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (t0 == 0) {
        tel[0] = pages;
        tel[1] = *((volatile uint32_t*)&A.counters->tasks);
        tel[3] = *((volatile uint32_t*)&A.counters->refs);
        tel[6] = P.F;
        for (uint32_t f = 0; f < P.F && f < FIBER_TELEMETRY_MAX_FRUSTA; ++f) {
            const uint32_t a = A.counters->frustum_task_base[f], b = A.counters->frustum_task_base[f + 1];
            *tel_frustum(tel, f, kTelEmittedSegments) = b - a;
        }
    }
    for (uint32_t p = t0; p < pages; p += stride) {
        const fiber_fine_page_meta pm = A.page_meta[p];
        const uint32_t f = frustum_for_tile(P, pm.coarse_tile_id);
        if (f != kInvalid) atomicAdd(tel_frustum(tel, f, kTelAllocatedPages), 1u);
        const uint32_t cand = A.tel_slots[pm.coarse_tile_id * kDepthSlices + pm.coarse_z];
        if (cand == 0u) continue;
        atomicAdd(tel + 2, cand);
        atomicAdd(tel + 4, 1u);
        atomicMax(tel + 5, cand);
        atomicAdd(tel + kTelHistogram + min(31u - (uint32_t)__clz(cand), 31u), 1u);
        if (f != kInvalid) {
            atomicAdd(tel_frustum(tel, f, kTelPageCandidates), cand);
            atomicAdd(tel_frustum(tel, f, kTelFineRefs), pm.seg_ref_count);
            atomicMax(tel_frustum(tel, f, kTelMaxPageCandidates), cand);
        }
    }
    // FRUSTUM_TELEMETRY_RASTER_* (:2830-2832): every tile run with work.
    for (uint32_t r = t0; r < runs; r += stride) {
        const fiber_raster_tile_run run = A.runs[r];
        if (run.work_count == 0u || run.frustum_id >= P.F) continue;
        atomicAdd(tel_frustum(tel, run.frustum_id, kTelRasterRuns), 1u);
        atomicAdd(tel_frustum(tel, run.frustum_id, kTelRasterLoad), run.load_score);
        atomicMax(tel_frustum(tel, run.frustum_id, kTelMaxRasterLoad), run.load_score);
    }
}

// FineSegRef records of references [0, n), from their tasks' records. References
// of a page dropped by an overflow hold whatever an earlier frame left there.
__global__ void __launch_bounds__(256) k_expand_refs(const uint32_t* __restrict__ ref_task,
                                                     const float4* __restrict__ task_rec, uint32_t n_tasks, uint64_t n,
                                                     fiber_fine_seg_ref* __restrict__ out) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t task = ref_task[r];
        const uint4 w = task < n_tasks ? reinterpret_cast<const uint4*>(task_rec)[(size_t)kTaskRec * task + 2u]
                                       : make_uint4(0u, 0u, 0u, 0u);
        out[r] = fiber_fine_seg_ref{w.x, w.y, w.z};
    }
}

// ---------------------------------------------------------------------------
// Launch wrappers
// ---------------------------------------------------------------------------
void launch_opaque(const LaunchCtx& L, const PrepassArgs& A, const float* depth, uint32_t pitch, uint32_t samples,
                   uint32_t tiles, bool stamp) {
    unsigned blocks = ceil_div_host(tiles, 8);
    if (blocks > (unsigned)L.sm_count * 16u) blocks = (unsigned)L.sm_count * 16u;
    if (blocks == 0u) blocks = 1u;
    k_opaque_reduce<<<blocks, 256, 0, L.stream>>>(L.P, A, depth, pitch, samples, stamp);
}
void launch_broad(const LaunchCtx& L, const PrepassArgs& A, bool stamp) {
    k_broad<<<ceil_div_host(L.I, 4), 128, 0, L.stream>>>(L.P, L.inst, A, stamp);
}
void launch_lut(const LaunchCtx& L, const PrepassArgs& A) {
    if (L.total_coarse_tiles) k_lut<<<ceil_div_host(L.total_coarse_tiles, 128), 128, 0, L.stream>>>(L.P, A);
}
void launch_fine(const LaunchCtx& L, const PrepassArgs& A) {
    k_fine<<<L.sm_count * 6, kFineThreads, 0, L.stream>>>(L.P, L.inst, A);
}
cudaError_t configure_prepass() {
    const auto max_smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_visit<false, false>, max_smem, (int)kVisitSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_visit<false, true>, max_smem, (int)kVisitSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_visit<true, false>, max_smem, (int)kVisitSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_visit<true, true>, max_smem, (int)kVisitSmemBytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_sort_big_cells, max_smem, (int)kBigSmemBytes);
    return e;
}
template <bool kOpaque, bool kTel>
static void launch_visit_as(const LaunchCtx& L, const PrepassArgs& A) {
    // The resident blocks (3 per SM), each looping over warps of tasks.
    k_visit<kOpaque, kTel><<<L.sm_count * 3, kVisitThreads, kVisitSmemBytes, L.stream>>>(L.P, A);
}
void launch_visit(const LaunchCtx& L, const PrepassArgs& A) {
    if (L.telemetry) {
        if (L.opaque) launch_visit_as<true, true>(L, A);
        else launch_visit_as<false, true>(L, A);
    } else {
        if (L.opaque) launch_visit_as<true, false>(L, A);
        else launch_visit_as<false, false>(L, A);
    }
}
void launch_alloc(const LaunchCtx& L, const PrepassArgs& A) {
    k_alloc_pages<<<L.sm_count * 4, kScanThreads, 0, L.stream>>>(L.P, A);
}
void launch_zero_pages(const LaunchCtx& L, const PrepassArgs& A) {
    k_zero_pages<<<L.sm_count * 4, 256, 0, L.stream>>>(A);
}
void launch_count(const LaunchCtx& L, const PrepassArgs& A) {
    k_count_visits<<<L.sm_count * 8, 256, 0, L.stream>>>(A);
}
void launch_count_walk(const LaunchCtx& L, const PrepassArgs& A) {
    if (L.opaque) k_traverse<kCount, true><<<L.sm_count * 8, 256, 0, L.stream>>>(L.P, A);
    else k_traverse<kCount, false><<<L.sm_count * 8, 256, 0, L.stream>>>(L.P, A);
}
void launch_prefix(const LaunchCtx& L, const PrepassArgs& A, bool csr) {
    k_prefix_pages<<<L.sm_count * 3, 256, 0, L.stream>>>(L.P, A, csr);
}
void launch_page_csr_count(const LaunchCtx& L, const PrepassArgs& A) {
    k_page_count<<<L.sm_count * 8, 256, 0, L.stream>>>(A);
    k_page_scan<<<1, 1024, 0, L.stream>>>(A);
    k_page_scatter<<<L.sm_count * 8, 256, 0, L.stream>>>(A);
}
void launch_build_pages(const LaunchCtx& L, const PrepassArgs& A) {
    k_build_pages<<<L.sm_count * 6, 256, 0, L.stream>>>(L.P, A);
}
void launch_fill_walk(const LaunchCtx& L, const PrepassArgs& A) {
    if (L.opaque) k_traverse<kFill, true><<<L.sm_count * 8, 256, 0, L.stream>>>(L.P, A);
    else k_traverse<kFill, false><<<L.sm_count * 8, 256, 0, L.stream>>>(L.P, A);
}
void launch_fill(const LaunchCtx& L, const PrepassArgs& A) {
    k_fill_visits<<<L.sm_count * 8, 256, 0, L.stream>>>(A);
}
void launch_compact_active(const LaunchCtx& L, const PrepassArgs& A, unsigned long long* lb_work) {
    k_compact_active<<<L.sm_count * 4, kScanThreads, 0, L.stream>>>(L.P, A, lb_work);
}
void launch_emit(const LaunchCtx& L, const PrepassArgs& A) {
    k_emit<<<L.sm_count * 4, 256, 0, L.stream>>>(L.P, A);
}
void launch_sort_cells(const LaunchCtx& L, const PrepassArgs& A) {
    k_sort_cells<<<L.sm_count * 5, 256, 0, L.stream>>>(A);  // the resident blocks (5 per SM)
}
void launch_telemetry(const LaunchCtx& L, const PrepassArgs& A) {
    k_telemetry<<<L.sm_count * 2, 256, 0, L.stream>>>(L.P, A);
}
void launch_expand_refs(cudaStream_t s, const uint32_t* ref_task, const float4* task_rec, uint32_t n_tasks, uint64_t n,
                        fiber_fine_seg_ref* out) {
    if (n) k_expand_refs<<<std::min(ceil_div_host(n, 256), 4096u), 256, 0, s>>>(ref_task, task_rec, n_tasks, n, out);
}
void launch_sort_big(const LaunchCtx& L, const PrepassArgs& A) {
    k_sort_big_cells<<<L.sm_count * 2, 256, kBigSmemBytes, L.stream>>>(A);
}

}  // namespace fiber
