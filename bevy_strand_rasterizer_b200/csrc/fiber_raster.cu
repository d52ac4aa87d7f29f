// fiber_raster.cu — the deep-opacity shadow raster (with the shadow-map
// stampback fused into its epilogue) and the camera colour raster:
// strand_rasterizer.wgsl:391-711 (SHADOWS) and :855-1044 (LINEAR),
// shadow_dom_stampback.wgsl:74-123.
//
// One 64-thread block per tile run, one thread per pixel slot (the reference's
// 64 slots; its 4 depth workers per pixel become the order in which one
// thread applies the same operations). Blocks claim runs from a counter. The
// run's references, its work items laid end to end, are taken in rounds of
// 128: each warp reads 32 references' task records at a time, keeps their
// end points, radii and shading in shared memory and turns them into one
// coverage-candidate bit per (pixel, entry) by a conservative band test; then
// each pixel walks its candidates, two at a time. Block barriers happen only
// between rounds. Shadow runs that would outlast the rest of the frame
// (heavy_limit) take 256-thread blocks, a thread per pixel and depth worker. The
// blend order is the reference's: work items near to far, references in groups of
// 4 from each item's start, (w0 over w1) over (w2 over w3), early out after each
// item once alpha > 0.98.
//
// Both rasters are bound by the walk's instructions: on the benchmark's medium
// frame 71 and 72 % of the issue slots are taken, by 24 and 18 of 32 lanes, and
// what is left are fixed-latency waits, staging loads and barriers at 24 warps
// per SM. So the walk is written for few instructions, with the results of the
// plain binary32 formulas bit for bit: packed pairs (.f32x2) for what comes in pairs, and quotients and square roots
// by a reciprocal estimate and fused corrections (fiber_device.cuh) instead of
// the general-range division and square root.
#include "fiber_kernels.cuh"

namespace fiber {

constexpr uint32_t kMaxRunItems = 256;  // 16 coarse z x 16 fine z cells per fine tile

// A block of kSplit threads per pixel slot, and its round of staged references.
template <uint32_t kSplit>
struct Tile {
    static constexpr uint32_t threads = kPixelSlots * kSplit, warps = threads / 32;
    static constexpr uint32_t round = kSplit == 1 ? 128 : 256, words = round / 32;
    static constexpr uint32_t groups = words / warps;  // of 32 references, per warp
    static_assert(groups * warps == words, "a round is whole groups of 32 per warp");
};

// ---------------------------------------------------------------------------
// Packed binary32 pairs. The assembler contracts a packed product and a packed
// sum of it into one fused operation whatever the rounding modifiers and flags
// say, also when the product is written as a fused multiply-add onto a constant
// -0. So a product is a fused multiply-add onto a -0 that comes as a kernel
// argument (RenderArgs::neg_zero2): it rounds the product alone (x + -0 = x for
// every x) and cannot be told from a real addend.
// ---------------------------------------------------------------------------
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(F2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 dup2(float x) { return pack2(x, x); }
struct Mul2 {
    F2 nz;  // (-0, -0)
    __device__ __forceinline__ F2 operator()(F2 a, F2 b) const { return fma2(a, b, nz); }
};
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, dup2(-1.0f), a); }
__device__ __forceinline__ float sum2(F2 v) {
    float x, y;
    unpack2(v, x, y);
    return __fadd_rn(x, y);
}

// Two square roots and two quotients at once (see Exact in fiber_device.cuh).
__device__ __forceinline__ F2 sqrt2_exact(Mul2 mul2, float x0, float x1) {
    const F2 x = pack2(x0, x1), y = pack2(rsqrt_estimate(x0), rsqrt_estimate(x1));
    const F2 s = mul2(x, y);
    return fma2(fma2(mul2(s, dup2(-1.0f)), s, x), mul2(y, dup2(0.5f)), s);
}
__device__ __forceinline__ F2 div2_exact(Mul2 mul2, F2 a, float b0, float b1) {
    const F2 nb = pack2(-b0, -b1), y0 = pack2(rcp_estimate(b0), rcp_estimate(b1));
    const F2 y = fma2(fma2(nb, y0, dup2(1.0f)), y0, y0);
    const F2 q = mul2(a, y);
    return fma2(fma2(nb, q, a), y, q);
}

// ---------------------------------------------------------------------------
// A run's references: its valid work items' first references and their starts
// in the run's order (items laid end to end).
// ---------------------------------------------------------------------------
struct RunItems {
    uint32_t base[kMaxRunItems];
    uint32_t start[kMaxRunItems + 1];
    uint32_t warp_refs[8], warp_items[8];
};

// Loads the run's work items (kChecked: those of the run's frustum and tile);
// items without references are left out. Returns their count; `total` the
// references. All threads; ends with a block barrier.
template <bool kChecked, uint32_t kWarps>
__device__ __forceinline__ uint32_t load_run_items(RunItems& s, const fiber_raster_work_item* __restrict__ work,
                                                   const fiber_raster_tile_run& run, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t n = min(run.work_count, kMaxRunItems);
    uint32_t items = 0u, refs = 0u;
    for (uint32_t c = 0; c < n; c += kWarps * 32u) {
        const uint32_t i = c + threadIdx.x;
        uint4 w = make_uint4(0u, 0u, 0u, 0u);  // seg_ref_base, seg_ref_count, frustum_id, screen_tile_id
        if (i < n) w = __ldg(reinterpret_cast<const uint4*>(work + run.work_base + i));
        if (kChecked && (w.z != run.frustum_id || w.w != run.screen_tile_id)) w.y = 0u;
        const uint32_t kept = __ballot_sync(0xFFFFFFFFu, w.y != 0u);
        uint32_t x = w.y;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31u) {
            s.warp_refs[warp] = x;
            s.warp_items[warp] = (uint32_t)__popc(kept);
        }
        __syncthreads();
        uint32_t items_before = items, refs_before = refs;
#pragma unroll
        for (uint32_t v = 0; v < kWarps; ++v) {
            if (v < warp) {
                items_before += s.warp_items[v];
                refs_before += s.warp_refs[v];
            }
            items += s.warp_items[v];
            refs += s.warp_refs[v];
        }
        const uint32_t at = items_before + (uint32_t)__popc(kept & ((1u << lane) - 1u));
        if (w.y != 0u) {
            s.base[at] = w.x;
            s.start[at] = refs_before + x - w.y;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) s.start[items] = refs;
    __syncthreads();
    total = refs;
    return items;
}

// The item that holds reference e0 + lane of the run, for the 32 lanes of a
// warp (meaningful where e0 + lane < total; e0 < total): the item of e0 by two
// ballots over the starts, then one bit per item that starts inside the 32.
__device__ __forceinline__ uint32_t item_of(const RunItems& s, uint32_t n_items, uint32_t e0, uint32_t lane) {
    const uint32_t k8 = lane * 8u;
    const unsigned b8 = __ballot_sync(0xFFFFFFFFu, k8 < n_items && s.start[k8] <= e0);
    const uint32_t first8 = ((uint32_t)__popc(b8) - 1u) * 8u;
    const unsigned b1 = __ballot_sync(0xFFFFFFFFu, lane < 8u && first8 + lane < n_items && s.start[min(first8 + lane, kMaxRunItems)] <= e0);
    const uint32_t i0 = first8 + (uint32_t)__popc(b1) - 1u;
    const uint32_t nx = i0 + 1u + lane;
    const uint32_t d = nx < n_items ? s.start[nx] - e0 : 32u;
    const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, d < 32u ? 1u << d : 0u);
    return i0 + (uint32_t)__popc(starts & (0xFFFFFFFFu >> (31u - lane)));
}

// The tasks of a warp's references of one round, a lane per reference, and their
// places: run item << 2 | worker. Read before the walk of the round before, so
// that staging a round waits for its records alone.
template <class T>
struct RoundTasks {
    uint32_t task[T::groups], place[T::groups];
    __device__ __forceinline__ RoundTasks(const RunItems& s, uint32_t n_items, const uint32_t* __restrict__ ref_task,
                                          uint32_t e0, uint32_t total, uint32_t lane, uint32_t warp) {
#pragma unroll
        for (uint32_t u = 0; u < T::groups; ++u) {
            const uint32_t ef = e0 + (warp + u * T::warps) * 32u;
            task[u] = place[u] = 0u;
            if (ef < total) {
                const uint32_t item = item_of(s, n_items, ef, lane);
                if (ef + lane < total) {
                    const uint32_t j = ef + lane - s.start[item];
                    task[u] = __ldg(ref_task + s.base[item] + j);
                    place[u] = (item << 2) | (j & 3u);
                }
            }
        }
    }
};
// The records of those tasks (lanes without one read task 0's).
template <class T>
struct RoundRecords {
    float4 a[T::groups], b[T::groups];
    uint4 w[T::groups];  // instance, segment, material
    __device__ __forceinline__ RoundRecords(const float4* __restrict__ task_rec, const RoundTasks<T>& t) {
#pragma unroll
        for (uint32_t u = 0; u < T::groups; ++u) {
            const float4* rec = task_rec + (size_t)kTaskRec * t.task[u];
            a[u] = __ldg(rec);
            b[u] = __ldg(rec + 1);
            w[u] = __ldg(reinterpret_cast<const uint4*>(rec) + 2);
        }
    }
};

// ---------------------------------------------------------------------------
// Coverage candidates. The exact test covers pixel p (cov > 0) only if p lies
// within the radius bound rb = rmin + (rmax - rmin) clamp(max z) of the
// segment's line and between the normals through its end points (t in [0, 1]).
// The band is widened by 1e-4 rb + 1e-6 rmax + 0.01 px + 1e-5 of the largest
// coordinate magnitude, over a hundred float ulps beyond the rounding of the
// exact test and of this one (a few ulps of the coordinates), so every pixel
// the band rejects is one the exact test leaves uncovered. A segment that is
// not `regular` or is shorter than 1e-6 px is a candidate of every pixel.
//
// regular: coordinates up to 2^24 px, each component of the end points'
// difference zero or at least 2^-20 px, radii up to 2^60. Then every
// intermediate of the corrected operations above stays normal: the projection
// numerator is zero or at least 2^-69 (pixel centres are half integers, so
// p - a is zero or at least 2^-25, the products at least 2^-45 and their
// cancelled sum at least 2^-69), its correction at least 2^-116. NaN fails it.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool regular_segment(float4 ab, float rmax) {
    const float X = fmaxf(fmaxf(fabsf(ab.x), fabsf(ab.y)), fmaxf(fabsf(ab.z), fabsf(ab.w)));
    const float dx = fabsf(ab.z - ab.x), dy = fabsf(ab.w - ab.y);
    const float tiny = 9.5367431640625e-7f;  // 2^-20
    return X <= 16777216.0f && (dx >= tiny || dx == 0.0f) && (dy >= tiny || dy == 0.0f) && rmax <= 1.152921504606847e18f;
}

// Shifts whose amounts clamp at 32 (0xFF moved out altogether).
__device__ __forceinline__ uint32_t shl_clamp(uint32_t x, uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}
__device__ __forceinline__ uint32_t shr_clamp(uint32_t x, uint32_t n) {
    uint32_t r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}

// Columns [il, ih] and rows [jl, jh] a candidate may lie in (the colour
// raster's bounding-box test, which is exact).
struct CellBox {
    int il, ih, jl, jh;
};

// Candidate bits of a segment (a.xy, b.xy in ab) against the tile's pixel slots
// p = j fsx + i (p < 64), pixel centres (x0 + i, y0 + j). On row j the band
// |n . (p - a)| <= thr is the columns [L + G j, H + G j], and so is the range
// of the distance along the segment; their intersection sets the row's bits.
// A slope below 1e-20 is taken as 1e-20, which puts a row of a line parallel
// to it wholly in or out by the sign. Interval ends are widened by 1e-3
// column; estimates of the reciprocals move them by a few ulps of
// (|f00| + thr) / |g|, far inside the band's slack divided by |g|. Both sides
// of the dispatch give the same bits: 8 x 8 tiles (every configuration's
// default) take rows as bytes without a loop bound or 64-bit shifts.
__device__ __forceinline__ unsigned long long candidate_bits(float4 ab, float z0, float z1, float rmin, float rmax,
                                                             float tile_max, float x0, float y0, uint32_t fsx,
                                                             uint32_t fsy, CellBox box) {
    const float X = fmaxf(fmaxf(fmaxf(fabsf(ab.x), fabsf(ab.y)), fmaxf(fabsf(ab.z), fabsf(ab.w))), tile_max);
    const float rb = rmin + (rmax - rmin) * __saturatef(fmaxf(z0, z1));
    const float slack = 0.01f + 1e-5f * X;
    const float thr = rb * 1.0001f + 1e-6f * rmax + slack;
    const float abx = ab.z - ab.x, aby = ab.w - ab.y;
    const float l2 = __fmaf_rn(abx, abx, aby * aby);
    if (!(l2 > 1e-12f)) return ~0ull;
    const float il = rsqrt_estimate(l2);
    const float ux = abx * il, uy = aby * il, len = l2 * il;
    const float px = x0 - ab.x, py = y0 - ab.y;
    const float d00 = __fmaf_rn(ux, py, -(uy * px)), s00 = __fmaf_rn(ux, px, uy * py);
    const float gx = copysignf(fmaxf(fabsf(ux), 1e-20f), ux), gy = copysignf(fmaxf(fabsf(uy), 1e-20f), uy);
    const float ix = rcp_estimate(gx), iy = rcp_estimate(gy);
    // n = (-uy, ux): d = d00 - uy i + ux j; s = s00 + ux i + uy j.
    const float dm = d00 * iy, dh = fabsf(thr * iy) + 1e-3f, Gd = ux * iy;
    const float sh = 0.5f * len + slack, sm = (0.5f * len - s00) * ix, shx = fabsf(sh * ix) + 1e-3f, Gs = -uy * ix;
    const float Ld = dm - dh, Hd = dm + dh, Ls = sm - shx, Hs = sm + shx;
    if (fsx == 8u && fsy == 8u) {
        uint32_t w[2] = {0u, 0u};
        box.ih = min(box.ih, 7);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float jf = (float)j;
            const float lo = fmaxf(__fmaf_rn(Gd, jf, Ld), __fmaf_rn(Gs, jf, Ls));
            const float hi = fminf(__fmaf_rn(Gd, jf, Hd), __fmaf_rn(Gs, jf, Hs));
            const int l = max(__float2int_ru(lo), box.il), h = min(__float2int_rd(hi), box.ih);
            uint32_t m = shl_clamp(0xFFu, (uint32_t)l) & shr_clamp(0xFFu, (uint32_t)(7 - h));
            if (j < box.jl || j > box.jh) m = 0u;
            w[j >> 2] |= m << ((j & 3) * 8);
        }
        return ((unsigned long long)w[1] << 32) | w[0];
    }
    const int cols = (int)min(fsx, 64u), rows = (int)min(fsy, (64u + fsx - 1u) / fsx);
    unsigned long long bits = 0ull;
    for (int j = max(0, box.jl); j < rows && j <= box.jh; ++j) {
        const float jf = (float)j;
        const float lo = fmaxf(__fmaf_rn(Gd, jf, Ld), __fmaf_rn(Gs, jf, Ls));
        const float hi = fminf(__fmaf_rn(Gd, jf, Hd), __fmaf_rn(Gs, jf, Hs));
        const int l = max(__float2int_ru(lo), box.il), h = min(min(__float2int_rd(hi), box.ih), cols - 1);
        if (l <= h) bits |= (((2ull << h) - 1ull) & ~((1ull << l) - 1ull)) << (j * (int)fsx);
    }
    return bits;
}

// 32 x 32 bit transpose across the warp: lane i holds row i on entry, lane p
// holds column p on return (bit i = bit p of lane i's row). Each stage swaps
// one bit of the lane index with the same bit of the bit position.
template <uint32_t J, uint32_t M>
__device__ __forceinline__ uint32_t transpose_stage(uint32_t x, uint32_t lane) {
    const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, J);
    return (lane & J) ? ((x & ~M) | ((y >> J) & M)) : ((x & M) | ((y & M) << J));
}
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, uint32_t lane) {
    x = transpose_stage<16u, 0x0000FFFFu>(x, lane);
    x = transpose_stage<8u, 0x00FF00FFu>(x, lane);
    x = transpose_stage<4u, 0x0F0F0F0Fu>(x, lane);
    x = transpose_stage<2u, 0x33333333u>(x, lane);
    return transpose_stage<1u, 0x55555555u>(x, lane);
}
// The entries' bits as per-pixel words: [word][pixel slot].
__device__ __forceinline__ void store_candidates(uint32_t* s_pmask, uint32_t word, unsigned long long bits, uint32_t lane) {
    s_pmask[word * kPixelSlots + lane] = warp_transpose32((uint32_t)bits, lane);
    s_pmask[word * kPixelSlots + 32u + lane] = warp_transpose32((uint32_t)(bits >> 32), lane);
}

// A pixel's walk over its candidates of a round, in entry order; with kMasked
// over those of one worker (`own`: the worker's entries of each word).
template <bool kMasked>
struct Walk {
    const uint32_t* mask;  // this pixel's column of the candidate words
    const uint32_t* own;
    uint32_t words, q, m;
    __device__ __forceinline__ Walk(const uint32_t* s_pmask, uint32_t slot, uint32_t n, const uint32_t* own_ = nullptr)
        : mask(s_pmask + slot), own(own_), words((n + 31u) >> 5), q(0u), m(0u) {}
    __device__ __forceinline__ uint32_t next() {
        while (m == 0u && q < words) {
            m = mask[q * kPixelSlots];
            if (kMasked) m &= own[q];
            ++q;
        }
        if (m == 0u) return kInvalid;
        const uint32_t bit = (uint32_t)(__ffs(m) - 1);
        m &= m - 1u;
        return (q - 1u) * 32u + bit;
    }
};

// ===========================================================================
// K16 deep-opacity shadow raster + K17 stampback.
//
// One 64-thread block per shadow tile run, one thread per pixel. The pixel's
// thread walks its coverage candidates in entry order: pass 1 finds the
// nearest covered depth, pass 2 accumulates the opacity of every covered
// entry into the partial of the reference's depth worker that owns the entry
// (worker w takes entries w, w+4, ... from each item's start), so each
// worker's partial sees its entries in the reference's order; the four
// partials combine in worker order as the reference does.
//
// The benchmark's medium frame (21,988 runs): 1.145 G -> 0.715 G warp
// instructions, 1.31 -> 0.99 ms of the light runs' launch; large (226,793 runs,
// 2.97 G covered pairs): 29.2 -> 17.5 ms. About a third of it is staging (364 warp instructions per 32
// references), the rest the walk. Rounds of 64, 192 and 256 references were
// slower (1.20, 1.17, 1.26 ms against 1.14), 14 and 16 blocks per SM too (shared
// memory holds 12 at 8 slices).
// ===========================================================================
constexpr int kMaxDomSlices = 16;
constexpr uint32_t kShadowEntry = 3;  // float4 words of a staged entry

template <uint32_t kSplit>
size_t shadow_smem_bytes(uint32_t K) {
    return (size_t)Tile<kSplit>::round * kShadowEntry * sizeof(float4) + (size_t)kPixelSlots * 4u * K * sizeof(float);
}

// Coverage of one staged entry at pixel centre (x, y) by the plain operators (0
// when the pixel's projection falls outside the segment), and the depth there.
__device__ __forceinline__ float shadow_coverage(const float4* e, float x, float y, float& qz) {
    const float4 ab = e[0], zl = e[1], c = e[2];
    const float t = line_t(x, y, ab.x, ab.y, ab.z, ab.w);
    const float qx = wmix(ab.x, ab.z, t), qy = wmix(ab.y, ab.w, t);
    qz = wmix(zl.x, zl.y, t);
    const float rr = wmix(c.x, c.y, wclamp(qz, 0.0f, 1.0f));
    const float dx = x - qx, dy = y - qy;
    const float cov = wclamp(1.0f - sqrtf(dx * dx + dy * dy) / rr, 0.0f, 1.0f);
    return (t < 0.0f || t > 1.0f) ? 0.0f : cov;
}

// The same of two regular entries side by side: t = num / l2 by the entry's
// reciprocal, then the distance over the radius for both at once. A squared
// distance below 2^-100 is raised to it: the quotient stays below 2^-36 (radii
// are at least 1e-4), which leaves 1 - quotient = 1 as a distance of 0 does.
__device__ __forceinline__ void shadow_point(Mul2 mul2, const float4* e, F2 p, float& t, float& qz, float& d2, float& rr) {
    const float4 ab = e[0], zl = e[1];
    const float2 c = *reinterpret_cast<const float2*>(e + 2);
    const F2 a = pack2(ab.x, ab.y), b = pack2(ab.z, ab.w);
    const float num = sum2(mul2(sub2(p, a), sub2(b, a)));
    t = div_by_rcp(num, zl.z, zl.w);
    const F2 tt = dup2(t), om = sub2(dup2(1.0f), tt);
    const F2 q = add2(mul2(a, om), mul2(b, tt));
    float om0, om1;
    unpack2(om, om0, om1);
    qz = __fadd_rn(__fmul_rn(zl.x, om0), __fmul_rn(zl.y, t));
    rr = wmix(c.x, c.y, __saturatef(qz));
    const F2 d = sub2(p, q);
    d2 = fmaxf(sum2(mul2(d, d)), 7.888609052210118e-31f);
}
__device__ __forceinline__ void shadow_coverage2(Mul2 mul2, const float4* e0, const float4* e1, F2 p, float& cov0, float& qz0,
                                                 float& cov1, float& qz1) {
    float t0, t1, d0, d1, r0, r1, c0, c1;
    shadow_point(mul2, e0, p, t0, qz0, d0, r0);
    shadow_point(mul2, e1, p, t1, qz1, d1, r1);
    unpack2(div2_exact(mul2, sqrt2_exact(mul2, d0, d1), r0, r1), c0, c1);
    cov0 = (t0 < 0.0f || t0 > 1.0f) ? 0.0f : __saturatef(__fsub_rn(1.0f, c0));
    cov1 = (t1 < 0.0f || t1 > 1.0f) ? 0.0f : __saturatef(__fsub_rn(1.0f, c1));
}

// kSplit: threads per pixel. With 1 a pixel's thread takes the four workers'
// entries in turn; with 4 each thread takes one worker's entries (its partials
// are its own), and the pixel's nearest item is the least of its four. The
// first renders the light runs, the second the heavy ones (k_emit lists them), side
// by side.
template <uint32_t kSplit>
__global__ void __launch_bounds__(Tile<kSplit>::threads, kSplit == 1 ? 12 : 3)
    k_shadow(const FrameParams* __restrict__ Pp, const InstanceView* __restrict__ inst, RenderArgs R) {
    using T = Tile<kSplit>;
    if (kSplit != 1u) stamp_start(R.stamps, kStampShadow);  // the heavy runs take the SMs first
    if (frame_failed(R.counters)) return;
    const FrameParams& P = *Pp;
    // Per staged entry: (ax, ay, bx, by), (z0, z1, |ab|^2, its reciprocal),
    // (rmin, rmax, opacity, run item << 16 | worker's partial offset).
    extern __shared__ float4 s_entry[];
    // [worker][K][pixel]: a warp's 32 pixels hit 32 banks whatever the slice.
    float* s_partial = reinterpret_cast<float*>(s_entry + T::round * kShadowEntry);
    __shared__ RunItems s_items;
    __shared__ uint32_t s_pmask[T::words * kPixelSlots];  // [word][pixel] candidate bits
    __shared__ uint32_t s_own[kSplit == 1 ? 1 : 4 * T::words];  // [worker][word] the worker's entries
    __shared__ uint32_t s_best[kSplit == 1 ? 1 : T::threads];   // [worker][pixel] nearest item so far
    __shared__ float s_best_z[kSplit == 1 ? 1 : T::threads];
    __shared__ uint32_t s_run;

    const uint32_t K = P.K, D = P.dom_size, S = P.shadow_map_size;
    const uint32_t slot = threadIdx.x % kPixelSlots, worker = threadIdx.x / kPixelSlots;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float* partial = s_partial + slot;  // partial[(w K + i) kPixelSlots]
    const uint32_t* own = kSplit == 1 ? nullptr : s_own + worker * T::words;
    const float Kf = u2f(K);
    const Mul2 mul2{R.neg_zero2};

    // Blocks claim runs from a counter, so long runs do not pile up on one
    // block; the next claim is in flight while a run is rendered.
    const uint32_t first = *((volatile uint32_t*)&R.counters->camera_active);
    const uint32_t n_runs = kSplit == 1 ? *((volatile uint32_t*)&R.counters->active_tiles) - first
                                        : *((volatile uint32_t*)&R.counters->heavy_runs);
    const uint32_t limit = heavy_limit(R.counters, R.shadow_blocks);
    uint32_t* counter = &R.counters->tile_counter[kSplit == 1 ? kShadowRunCounter : kHeavyRunCounter];
    uint32_t claim = 0u;
    if (threadIdx.x == 0) claim = atomicAdd(counter, 1u);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_run = claim;
        __syncthreads();
        const uint32_t r = s_run;
        if (r >= n_runs) break;
        if (threadIdx.x == 0) claim = atomicAdd(counter, 1u);
        const fiber_raster_tile_run run = R.runs[kSplit == 1 ? first + r : R.heavy_list[r]];
        if (kSplit == 1u && run.load_score >= limit) continue;  // the other kernel's
        const uint32_t f = run.frustum_id;
        const uint32_t layer = light_layer(P, f);
        if (run.work_count == 0u || layer == kInvalid) continue;
        const fiber_frustum_desc& d = P.frusta[f];
        const uint32_t fsx = d.froxel_size_x, fsy = d.froxel_size_y;
        const uint32_t ftx = ceil_div(d.screen_width, fsx);
        const uint32_t tx = run.screen_tile_id % ftx, ty = run.screen_tile_id / ftx;
        const uint32_t px = tx * fsx + slot % fsx;
        const uint32_t py = ty * fsy + slot / fsx;
        const bool active = slot < fsx * fsy && px < d.screen_width && py < d.screen_height;
        const float pfx = u2f(px) + 0.5f, pfy = u2f(py) + 0.5f;
        const F2 pf = pack2(pfx, pfy);
        uint32_t total;
        const uint32_t n_items = load_run_items<true, T::warps>(s_items, R.work, run, total);

        // Stages references [e0, e0 + n) of the run, whose tasks are in `next`,
        // and fetches the following round's tasks: each warp takes 32 at a
        // time, a lane per reference (its record as k_fine wrote it for this
        // frustum, then its material), stores the entry and its candidate bits.
        // Returns whether every entry is regular and of finite opacity; has a block
        // barrier.
        RoundTasks<T> next(s_items, n_items, R.ref_task, 0u, total, lane, warp);
        auto stage = [&](uint32_t e0, uint32_t n) -> bool {
            const float x0 = u2f(tx * fsx) + 0.5f, y0 = u2f(ty * fsy) + 0.5f;
            const float tile_max = fmaxf(u2f((tx + 1u) * fsx), u2f((ty + 1u) * fsy)) + 1.0f;
            bool plain = false;
            const RoundRecords<T> rr(R.task_rec, next);
#pragma unroll
            for (uint32_t u = 0; u < T::groups; ++u) {
                const uint32_t q = warp + u * T::warps, s = q * 32u + lane;
                if (q * 32u >= n) break;
                unsigned long long bits = 0ull;
                if (s < n) {
                    const float4 a = rr.a[u], b = rr.b[u];
                    const fiber_strand_material& m = inst[rr.w[u].x].materials[rr.w[u].z];
                    const float rmin = wmax(m.min_radius_pixels, 1e-4f), rmax = wmax(m.max_radius_pixels, rmin);
                    const float4 ab = make_float4(a.x, a.y, b.x, b.y);
                    const float z0 = normalize_depth01(a.z), z1 = normalize_depth01(b.z);
                    const float abx = b.x - a.x, aby = b.y - a.y, l2 = abx * abx + aby * aby;
                    // l2 = 0: t = 0 as line_t gives it.
                    s_entry[s * kShadowEntry] = ab;
                    s_entry[s * kShadowEntry + 1u] = make_float4(z0, z1, l2, l2 > 0.0f ? 1.0f / l2 : 0.0f);
                    const uint32_t tag = (next.place[u] >> 2 << 16) | ((next.place[u] & 3u) * K * kPixelSlots);
                    s_entry[s * kShadowEntry + 2u] = make_float4(rmin, rmax, m.absorption_color[3], __uint_as_float(tag));
                    if (regular_segment(ab, rmax)) {
                        bits = candidate_bits(ab, z0, z1, rmin, rmax, tile_max, x0, y0, fsx, fsy, CellBox{0, 63, 0, 63});
                    } else {
                        bits = ~0ull;
                        plain = true;
                    }
                    // The regular walk deposits entries of coverage 0 too: 0 x an
                    // infinite or NaN opacity would not leave the partials alone.
                    plain = plain || !(fabsf(m.absorption_color[3]) <= 3.402823466e38f);
                }
                __syncwarp();
                store_candidates(s_pmask, q, bits, lane);
                if (kSplit != 1u) {
#pragma unroll
                    for (uint32_t w = 0; w < 4u; ++w) {
                        const uint32_t of_w = __ballot_sync(0xFFFFFFFFu, s < n && (next.place[u] & 3u) == w);
                        if (lane == 0u) s_own[w * T::words + q] = of_w;
                    }
                }
            }
            next = RoundTasks<T>(s_items, n_items, R.ref_task, e0 + T::round, total, lane, warp);
            return !__syncthreads_or(plain);
        };

        // ---- Pass 1: nearest covered depth = max depth of the covered entries
        // of the first run item holding one; the walk stops once the next
        // candidate lies past that item.
        uint32_t best = kInvalid;  // first item with a covered entry
        float z0 = -1.0f;          // its max covered depth
        bool complete = !active;   // the best item is fully processed
        bool regular = true;       // of the round that is staged
        uint32_t e0 = 0u, staged = kInvalid;
        for (; e0 < total; e0 += T::round) {
            const uint32_t n = min(T::round, total - e0);
            regular = stage(e0, n);
            staged = e0;
            if (!complete) {
                Walk<kSplit != 1u> walk(s_pmask, slot, n, own);
                for (;;) {
                    const uint32_t bi = walk.next();
                    if (bi == kInvalid) break;
                    const float4* e = s_entry + bi * kShadowEntry;
                    const uint32_t item = __float_as_uint(e[2].w) >> 16;
                    if (best != kInvalid && item > best) break;
                    float qz;
                    if (shadow_coverage(e, pfx, pfy, qz) > 0.0f) {
                        best = item;
                        z0 = wmax(z0, qz);
                    }
                }
            }
            uint32_t nearest = best;
            if (kSplit != 1u) {
                s_best[threadIdx.x] = best;
                __syncthreads();
#pragma unroll
                for (uint32_t w = 0; w < kSplit; ++w) nearest = min(nearest, s_best[w * kPixelSlots + slot]);
            }
            complete = !active || (nearest != kInvalid && s_items.start[nearest + 1u] <= e0 + n);
            if (__syncthreads_and(complete)) break;
        }
        if (kSplit != 1u) {
            // The pixel's: the nearest of its workers' items, and the depth of
            // those that found it.
            s_best[threadIdx.x] = best;
            s_best_z[threadIdx.x] = z0;
            __syncthreads();
#pragma unroll
            for (uint32_t w = 0; w < kSplit; ++w) {
                const uint32_t b = s_best[w * kPixelSlots + slot];
                const float z = s_best_z[w * kPixelSlots + slot];
                if (b < best) {
                    best = b;
                    z0 = z;
                } else if (b == best) {
                    z0 = wmax(z0, z);
                }
            }
        }
        const bool found = active && best != kInvalid;

        // ---- Pass 2: opacity partials, each covered entry into its worker's.
        if (kSplit == 1u) {
            for (uint32_t i = 0; i < 4u * K; ++i) partial[i * kPixelSlots] = 0.0f;
        } else {
            for (uint32_t i = 0; i < K; ++i) partial[(worker * K + i) * kPixelSlots] = 0.0f;
        }
        const float alpha_z0 = found ? z0 : 1.0f;
        const float inv_span = 1.0f / wmax(1e-6f, alpha_z0);
        if (__syncthreads_or(found)) {
            // Pass 1 that stopped after the first round left it staged.
            if (staged != 0u) next = RoundTasks<T>(s_items, n_items, R.ref_task, 0u, total, lane, warp);
            for (e0 = 0u; e0 < total; e0 += T::round) {
                const uint32_t n = min(T::round, total - e0);
                if (e0 != 0u || staged != 0u) regular = stage(e0, n);
                if (found) {
                    // The entry's slice and weight, then its deposits: the
                    // slice of u = clamp((z0 - qz) / z0) K (pow(u, DOM_GAMMA = 1)
                    // is u) and, with its fraction, the next one. u K < 2^23, so
                    // adding 2^23 rounding down leaves its floor in the low bits.
                    auto deposit = [&](const float4* e, float cov, float qz) {
                        const float2 c = *(reinterpret_cast<const float2*>(e + 2) + 1);  // opacity, tag
                        const float tl = __fmul_rn(__saturatef(__fmul_rn(__fsub_rn(alpha_z0, qz), inv_span)), Kf);
                        const float fl = __fadd_rd(tl, 8388608.0f);
                        const float wf = __fsub_rn(tl, __fsub_rn(fl, 8388608.0f));
                        const uint32_t si = min(__float_as_uint(fl) & 31u, K - 1u);
                        const float al = __fmul_rn(__fmul_rn(cov, c.x), 0.5f);
                        float* pw = partial + ((__float_as_uint(c.y) & 0xFFFFu) + si * kPixelSlots);
                        const float a0 = pw[0];
                        pw[0] = __saturatef(a0 + (1.0f - a0) * (1.0f - wf) * al);
                        if (si + 1u < K) {
                            const float a1 = pw[kPixelSlots];
                            pw[kPixelSlots] = __saturatef(a1 + (1.0f - a1) * wf * al);
                        }
                    };
                    Walk<kSplit != 1u> walk(s_pmask, slot, n, own);
                    if (regular) {
                        // Candidates two at a time: both coverages side by side,
                        // the deposits in entry order.
                        for (;;) {
                            const uint32_t b0 = walk.next();
                            if (b0 == kInvalid) break;
                            const uint32_t b1 = walk.next();
                            const float4* ea = s_entry + b0 * kShadowEntry;
                            const float4* eb = b1 != kInvalid ? s_entry + b1 * kShadowEntry : ea;
                            float cov0, cov1, qz0, qz1;
                            shadow_coverage2(mul2, ea, eb, pf, cov0, qz0, cov1, qz1);
                            // A coverage of 0 leaves the partials as they are
                            // (a + (1 - a) w 0 = a, the opacity being finite),
                            // and few are: no branch.
                            deposit(ea, cov0, qz0);
                            if (b1 == kInvalid) break;
                            deposit(eb, cov1, qz1);
                        }
                    } else {
                        for (uint32_t bi = walk.next(); bi != kInvalid; bi = walk.next()) {
                            const float4* e = s_entry + bi * kShadowEntry;
                            float qz;
                            const float cov = shadow_coverage(e, pfx, pfy, qz);
                            if (cov > 0.0f) deposit(e, cov, qz);
                        }
                    }
                }
                __syncthreads();
            }
        }
        // ---- Combine the 4 workers per slice, write the DOM, stamp the shadow map.
        if (active && worker == 0u) {
            // A texel of a page the sparse pool could not hold is not stored
            // (counted as a DOM pool overflow); the stampback still runs.
            // Dense layers index the texel directly; the sparse pool goes
            // through the page table (dom_texel).
            const bool dense = P.dom_pool_pages == 0u;
            float* dz = nullptr;
            float* dop = nullptr;
            size_t ds = 0;
            const size_t dom_px = (size_t)py * D + px;
            const bool stored = dense || dom_texel(P, R, layer, px, py, dz, dop, ds);
            if (!found) {
                if (dense) {
                    R.dom_depth[(size_t)layer * D * D + dom_px] = 0.0f;
                    for (uint32_t i = 0; i < K; ++i) R.dom_opacity[((size_t)layer * K + i) * D * D + dom_px] = 0.0f;
                } else if (stored) {
                    *dz = 0.0f;
                    for (uint32_t i = 0; i < K; ++i) dop[i * ds] = 0.0f;
                }
            } else {
                if (dense) R.dom_depth[(size_t)layer * D * D + dom_px] = z0;
                else if (stored) *dz = z0;
                float acc = 0.0f;
                for (uint32_t i = 0; i < K; ++i) {
                    float a = 0.0f;
                    for (uint32_t wk = 0; wk < 4u; ++wk) a = a + (1.0f - a) * partial[(wk * K + i) * kPixelSlots];
                    acc = acc + (1.0f - acc) * a;  // opaque_terminal_slice = K without an opaque depth
                    if (dense) R.dom_opacity[((size_t)layer * K + i) * D * D + dom_px] = acc;
                    else if (stored) dop[i * ds] = acc;
                }
                // Fused stampback: every target texel whose DOM footprint holds
                // this texel takes the max depth (the target starts cleared).
                if (z0 > 0.0f) {
                    uint32_t x_lo = (uint32_t)(((uint64_t)px * S) / D), y_lo = (uint32_t)(((uint64_t)py * S) / D);
                    x_lo = x_lo > 0u ? x_lo - 1u : 0u;
                    y_lo = y_lo > 0u ? y_lo - 1u : 0u;
                    for (uint32_t ty2 = y_lo; ty2 < S && ty2 <= y_lo + 2u + S / D; ++ty2) {
                        uint32_t mny = min((ty2 * D) / S, D - 1u), mxy = min(((ty2 + 1u) * D + S - 1u) / S, D);
                        if (py < mny || py >= mxy) continue;
                        for (uint32_t tx2 = x_lo; tx2 < S && tx2 <= x_lo + 2u + S / D; ++tx2) {
                            uint32_t mnx = min((tx2 * D) / S, D - 1u), mxx = min(((tx2 + 1u) * D + S - 1u) / S, D);
                            if (px < mnx || px >= mxx) continue;
                            atomicMax(reinterpret_cast<int*>(R.shadow_map + (size_t)layer * S * S + (size_t)ty2 * S + tx2),
                                      __float_as_int(z0));
                        }
                    }
                }
            }
        }
    }
}

// ===========================================================================
// Sparse DOM residency (the reference's bevy_vsms demand paging, replaced by
// a per-frame page pool). Every shadow tile run with work requests the DOM
// pages under its tile and their neighbours (request_shadow_dom_pages,
// strand_prepass.wgsl:2540-2579, DOM_PREFETCH_PAGE_BORDER = 1); requested
// pages take pool pages in page-table order (layer, row, column), as many as
// the pool holds; their depth planes are cleared (a texel without depth is
// empty whatever its opacity words hold).
// ===========================================================================
constexpr uint32_t kDomBorder = 1;

__global__ void __launch_bounds__(256) k_dom_request(const FrameParams* __restrict__ Pp, RenderArgs R) {
    if (frame_failed(R.counters)) return;
    const FrameParams& P = *Pp;
    const uint32_t first = *((volatile uint32_t*)&R.counters->camera_active);
    const uint32_t last = *((volatile uint32_t*)&R.counters->active_tiles);
    const uint32_t ppx = P.dom_pages_x;
    for (uint32_t r = first + blockIdx.x * blockDim.x + threadIdx.x; r < last; r += gridDim.x * blockDim.x) {
        const fiber_raster_tile_run run = R.runs[r];
        const uint32_t layer = light_layer(P, run.frustum_id);
        if (run.work_count == 0u || layer == kInvalid) continue;
        const fiber_frustum_desc& d = P.frusta[run.frustum_id];
        const uint32_t ftx = ceil_div(d.screen_width, d.froxel_size_x);
        const uint32_t x0 = (run.screen_tile_id % ftx) * d.froxel_size_x, y0 = (run.screen_tile_id / ftx) * d.froxel_size_y;
        const uint32_t x1 = min(x0 + d.froxel_size_x - 1u, d.screen_width - 1u);
        const uint32_t y1 = min(y0 + d.froxel_size_y - 1u, d.screen_height - 1u);
        const uint32_t pmx0 = x0 / kDomPage, pmy0 = y0 / kDomPage;
        const uint32_t px0 = pmx0 - min(pmx0, kDomBorder), py0 = pmy0 - min(pmy0, kDomBorder);
        const uint32_t px1 = min(x1 / kDomPage + kDomBorder, ppx - 1u), py1 = min(y1 / kDomPage + kDomBorder, ppx - 1u);
        for (uint32_t py = py0; py <= py1; ++py)
            for (uint32_t px = px0; px <= px1; ++px) R.dom_page_table[((size_t)layer * ppx + py) * ppx + px] = kMarked;
    }
}

// One block: requested entries, in table order, get pool page index + 1.
__global__ void __launch_bounds__(1024) k_dom_alloc(const FrameParams* __restrict__ Pp, RenderArgs R, uint32_t entries) {
    if (frame_failed(R.counters)) return;
    const FrameParams& P = *Pp;
    __shared__ uint32_t s_warp[33];
    __shared__ uint32_t s_carry;
    if (threadIdx.x == 0) s_carry = 0u;
    __syncthreads();
    for (uint32_t b = 0; b < entries; b += 1024u) {
        const uint32_t i = b + threadIdx.x;
        const bool req = i < entries && R.dom_page_table[i] == kMarked;
        uint32_t total;
        const uint32_t ex = block_exclusive_scan<1024>(req ? 1u : 0u, s_warp, total);
        if (req) {
            const uint32_t idx = s_carry + ex;
            R.dom_page_table[i] = idx < P.dom_pool_pages ? idx + 1u : 0u;
        }
        __syncthreads();
        if (threadIdx.x == 0) s_carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        R.counters->dom_pages = s_carry;
        if (s_carry > P.dom_pool_pages) atomicOr(&R.counters->overflow, 16u);
    }
}

__global__ void __launch_bounds__(256) k_dom_clear(const FrameParams* __restrict__ Pp, RenderArgs R) {
    const FrameParams& P = *Pp;
    const uint32_t pages = min(*((volatile uint32_t*)&R.counters->dom_pages), P.dom_pool_pages);
    const size_t per_page = kDomPageTexels / 4u, n = (size_t)pages * per_page;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        float* page = R.dom_pool + (k / per_page) * kDomPageTexels * (P.K + 1u);
        reinterpret_cast<float4*>(page)[k % per_page] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

void launch_dom_paging(const LaunchCtx& L, const RenderArgs& R, uint32_t table_entries) {
    k_dom_request<<<L.sm_count * 2, 256, 0, L.stream>>>(L.P, R);
    k_dom_alloc<<<1, 1024, 0, L.stream>>>(L.P, R, table_entries);
    k_dom_clear<<<L.sm_count * 4, 256, 0, L.stream>>>(L.P, R);
}

// ===========================================================================
// K19 camera colour raster.
//
// One 64-thread block per camera tile run, one thread per pixel. Each pixel
// walks its candidate entries in order (two per step: both entries' coverage
// and shading side by side, then they land in entry order). An entry belongs to
// worker w of its group of 4 (an item's entries 4g .. 4g+3 from the item start),
// and a group blends as the reference's four workers do: (w0 over w1) over (w2
// over w3), then final over group. A worker without a covered entry contributes
// transparent black and depth 0, and x over 0 = 0 over x = x exactly, so the
// group is held as at most two halves and most groups, which hold one covered
// entry, are that entry. Group and item state carry over from round to round.
//
// The benchmark's medium frame (25,918 runs): 620 M -> 382 M warp instructions,
// 0.68 -> 0.49 ms; large: 3.50 -> 1.84 ms.
// ===========================================================================
constexpr uint32_t kCamEntry = 5;  // float4 words of a staged entry

// A premultiplied colour as two pairs: (r, g), (b, a).
struct Rgba {
    F2 rg, ba;
    __device__ __forceinline__ float alpha() const {
        float b, a;
        unpack2(ba, b, a);
        return a;
    }
};
// blend_over_premult (strand_rasterizer.wgsl:156-162)
__device__ __forceinline__ Rgba over(Mul2 mul2, const Rgba& fg, const Rgba& bg) {
    const F2 oma = dup2(__fsub_rn(1.0f, fg.alpha()));
    return Rgba{add2(fg.rg, mul2(bg.rg, oma)), add2(fg.ba, mul2(bg.ba, oma))};
}

// Coverage, depth and shaded premultiplied colour of one staged entry at pixel
// centre (x, y) by the plain operators.
__device__ __forceinline__ bool cam_eval(const float4* e, float x, float y, Rgba& v, float& pz) {
    const float4 ab = e[0], zw = e[1], c = e[2], c0 = e[3], c1 = e[4];
    const float rmax = c.y;
    const bool in_box = !((x < wmin(ab.x, ab.z) - rmax || y < wmin(ab.y, ab.w) - rmax) ||
                          (x > wmax(ab.x, ab.z) + rmax || y > wmax(ab.y, ab.w) + rmax));
    const float abx = ab.z - ab.x, aby = ab.w - ab.y;
    const float t = ((x - ab.x) * abx + (y - ab.y) * aby) * c.z;
    const float fx = ab.x + abx * t, fy = ab.y + aby * t;
    pz = wmix(zw.x, zw.y, t);
    const float rr = wmix(c.x, rmax, wclamp(normalize_depth01(pz), 0.0f, 1.0f));
    const float dx = x - fx, dy = y - fy;
    const float d2 = dx * dx + dy * dy;
    const float cov = wclamp(1.0f - sqrtf(d2) / rr, 0.0f, 1.0f);
    const float tw = (t * zw.z) / ((1.0f - t) * zw.w + t * zw.z);  // perspective_correct_line_t (:149-154)
    const float alpha = wmix(c0.w, c1.w, tw) * cov;
    v.rg = pack2(wmix(c0.x, c1.x, tw) * c.w * alpha, wmix(c0.y, c1.y, tw) * c.w * alpha);
    v.ba = pack2(wmix(c0.z, c1.z, tw) * c.w * alpha, alpha);
    return in_box && t >= 0.0f && t <= 1.0f && d2 < rr * rr;
}

// The same for two regular entries side by side, whose candidate bits already
// hold the box test and whose depths lie in [0, 1] (so the depth at a covered
// pixel does too, up to an ulp above 1, and its normalised value is its clamp).
struct CamPoint {
    float t, pz, d2, rr, num, den;  // tw = num / den
};
__device__ __forceinline__ CamPoint cam_point(Mul2 mul2, const float4* e, F2 p) {
    const float4 ab = e[0], zw = e[1];
    const float4 c = e[2];
    CamPoint r;
    const F2 a = pack2(ab.x, ab.y), b = pack2(ab.z, ab.w), ba = sub2(b, a);
    r.t = __fmul_rn(sum2(mul2(sub2(p, a), ba)), c.z);
    const F2 d = sub2(p, add2(a, mul2(ba, dup2(r.t))));
    r.d2 = sum2(mul2(d, d));
    const float om = __fsub_rn(1.0f, r.t);
    r.pz = __fadd_rn(__fmul_rn(zw.x, om), __fmul_rn(zw.y, r.t));
    r.rr = wmix(c.x, c.y, __saturatef(r.pz));
    r.num = __fmul_rn(r.t, zw.z);
    r.den = __fadd_rn(__fmul_rn(om, zw.w), r.num);
    return r;
}
__device__ __forceinline__ Rgba cam_colour(Mul2 mul2, const float4* e, float cov, float tw) {
    const float4 c0 = e[3], c1 = e[4];
    const float vis = e[2].w;
    const F2 tt = dup2(tw), om = sub2(dup2(1.0f), tt);
    const F2 rg = add2(mul2(pack2(c0.x, c0.y), om), mul2(pack2(c1.x, c1.y), tt));
    const F2 ba = add2(mul2(pack2(c0.z, c0.w), om), mul2(pack2(c1.z, c1.w), tt));
    const F2 vba = mul2(ba, pack2(vis, cov));  // (blue * visibility, alpha)
    float bl, alpha;
    unpack2(vba, bl, alpha);
    return Rgba{mul2(mul2(rg, dup2(vis)), dup2(alpha)), pack2(__fmul_rn(bl, alpha), alpha)};
}
__device__ __forceinline__ bool cam_covered(const CamPoint& p) {
    return p.t >= 0.0f && p.t <= 1.0f && p.d2 < __fmul_rn(p.rr, p.rr);
}

__global__ void __launch_bounds__(Tile<1>::threads, 12) k_raster(const FrameParams* __restrict__ Pp,
                                                            const InstanceView* __restrict__ inst, RenderArgs R) {
    using T = Tile<1>;
    stamp_start(R.stamps, kStampRaster);
    if (frame_failed(R.counters)) return;
    const FrameParams& P = *Pp;
    // Per staged entry: (ax, ay, bx, by), (depths, then |w| of both end points,
    // at least 1e-6), (rmin, rmax, 1 / |ab|^2, visibility), the shading texels
    // of both end points; s_tag: run item << 2 | worker.
    __shared__ float4 s_entry[T::round * kCamEntry];
    __shared__ uint16_t s_tag[T::round];
    __shared__ uint32_t s_pmask[T::words * kPixelSlots];  // [word][pixel] candidate bits
    __shared__ RunItems s_items;
    __shared__ uint32_t s_run;

    const uint32_t n_runs = *((volatile uint32_t*)&R.counters->camera_active);
    const uint32_t slot = threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t cap = P.atlas_cap;
    const __half* hist = R.history[(P.hist_in & 1u) ^ 1u];
    const Mul2 mul2{R.neg_zero2};
    // Blocks claim runs from a counter, so long runs do not pile up on one
    // block; the next claim is in flight while a run is rendered.
    uint32_t claim = 0u;
    if (threadIdx.x == 0) claim = atomicAdd(&R.counters->tile_counter[kCameraRunCounter], 1u);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_run = claim;
        __syncthreads();
        const uint32_t r = s_run;
        if (r >= n_runs) break;
        if (threadIdx.x == 0) claim = atomicAdd(&R.counters->tile_counter[kCameraRunCounter], 1u);
        const fiber_raster_tile_run run = R.runs[r];
        const uint32_t f = run.frustum_id;
        if (run.work_count == 0u || f >= P.camera_frustum_end) continue;
        const fiber_frustum_desc& d = P.frusta[f];
        const uint32_t fsx = d.froxel_size_x, fsy = d.froxel_size_y;
        const uint32_t ftx = ceil_div(d.screen_width, fsx);
        const uint32_t tx = run.screen_tile_id % ftx, ty = run.screen_tile_id / ftx;
        const uint32_t px = tx * fsx + slot % fsx;
        const uint32_t py = ty * fsy + slot / fsx;
        const bool active = slot < fsx * fsy && px < d.screen_width && py < d.screen_height;
        const float pcx = u2f(px) + 0.5f, pcy = u2f(py) + 0.5f;
        const F2 pc = pack2(pcx, pcy);
        uint32_t total;
        const uint32_t n_items = load_run_items<false, T::warps>(s_items, R.work, run, total);

        Rgba fin{0ull, 0ull}, cur{0ull, 0ull}, half{0ull, 0ull};
        float gdepth = 0.0f;
        bool done = !active;
        uint32_t frags = 0;
        // The group being gathered: its run position (kInvalid: none), the half
        // that `cur` belongs to, whether `half` holds the first one, its item.
        uint32_t lead = kInvalid, side = 0u, item = 0u;
        bool two_halves = false;
        auto blend_group = [&]() {
            if (lead == kInvalid) return;
            fin = over(mul2, fin, two_halves ? over(mul2, half, cur) : cur);
            lead = kInvalid;
            two_halves = false;
        };
        // Early out (alpha > 0.98) at the end of an item.
        auto end_item = [&]() {
            const float w = fin.alpha();
            if (w > 0.98f) {
                float x, y, z, w_;
                unpack2(fin.rg, x, y);
                unpack2(fin.ba, z, w_);
                fin.rg = pack2(x / w, y / w);
                fin.ba = pack2(z / w, 1.0f);
                done = true;
            }
        };
        // A covered entry (run position e, tag item << 2 | worker).
        auto land = [&](uint32_t e, uint32_t tag, const Rgba& v, float pz) {
            const uint32_t w = tag & 3u, at = e - w, sd = w >> 1;
            if (at == lead) {
                if (sd == side) {
                    cur = over(mul2, cur, v);
                } else {
                    half = cur;
                    two_halves = true;
                    cur = v;
                    side = sd;
                }
            } else {
                const bool had = lead != kInvalid;
                blend_group();
                if (had && (tag >> 2) > item) {
                    end_item();
                    if (done) return;
                }
                lead = at;
                item = tag >> 2;
                cur = v;
                side = sd;
            }
            gdepth = wmax(gdepth, pz);
            ++frags;
        };
        RoundTasks<T> next(s_items, n_items, R.ref_task, 0u, total, lane, warp);
        for (uint32_t e0 = 0u; e0 < total; e0 += T::round) {
            const uint32_t n = min(T::round, total - e0);
            // Stage the round, whose tasks are in `next`, and fetch the
            // following one's: each warp takes 32 references at a time, a lane
            // per reference (its record as k_fine wrote it for this frustum,
            // then its material, shading and history texels).
            const float x0 = u2f(tx * fsx) + 0.5f, y0 = u2f(ty * fsy) + 0.5f;
            const float tile_max = fmaxf(u2f((tx + 1u) * fsx), u2f((ty + 1u) * fsy)) + 1.0f;
            bool plain = false;
            const RoundRecords<T> rr(R.task_rec, next);
#pragma unroll
            for (uint32_t u = 0; u < T::groups; ++u) {
                const uint32_t q = warp + u * T::warps, s = q * 32u + lane;
                if (q * 32u >= n) break;
                unsigned long long bits = 0ull;
                if (s < n) {
                    const float4 a = rr.a[u], b = rr.b[u];
                    const uint4 w = rr.w[u];
                    s_tag[s] = (uint16_t)next.place[u];
                    if (!(a.x < 0.0f && b.x < 0.0f)) {  // else behind the camera: never a candidate
                        const fiber_strand_material& m = inst[w.x].materials[w.z];
                        const uint32_t i0 = min(w.y, cap - 1u), i1 = min(i0 + 1u, cap - 1u);
                        const size_t t0 = (size_t)w.x * cap + i0, t1 = (size_t)w.x * cap + i1;
                        // min_radius = max(rmin, 1e-4) and max(rmax, min_radius) are
                        // idempotent on these values, so they are applied once here.
                        const float rmin = wmax(m.min_radius_pixels, 1e-4f), rmax = wmax(m.max_radius_pixels, rmin);
                        const float4 ab = make_float4(a.x, a.y, b.x, b.y);
                        const float abx = b.x - a.x, aby = b.y - a.y;
                        float4* e = s_entry + s * kCamEntry;
                        e[0] = ab;
                        e[1] = make_float4(a.z, b.z, wmax(fabsf(a.w), 1e-6f), wmax(fabsf(b.w), 1e-6f));
                        e[2] = make_float4(rmin, rmax, 1.0f / (abx * abx + aby * aby), __half2float(hist[t0 * 2]));
                        e[3] = load_half4(R.atlas + t0 * 4);
                        e[4] = load_half4(R.atlas + t1 * 4);
                        const bool depths = a.z >= 0.0f && a.z <= 1.0f && b.z >= 0.0f && b.z <= 1.0f;
                        const float wmx = fmaxf(fabsf(a.w), fabsf(b.w));
                        if (depths && wmx <= 1.152921504606847e18f && regular_segment(ab, rmax)) {
                            // The box test: pixel x is inside where x + 0.5 >= lo and
                            // x + 0.5 <= hi. lo - 0.5 and hi - 0.5 are exact where they
                            // come near a pixel index (0 or more), so rounding them to
                            // integers decides as the comparisons do.
                            const float lx = wmin(a.x, b.x) - rmax, ly = wmin(a.y, b.y) - rmax;
                            const float hx = wmax(a.x, b.x) + rmax, hy = wmax(a.y, b.y) + rmax;
                            const int bx = (int)(tx * fsx), by = (int)(ty * fsy);
                            const CellBox box{max(__float2int_ru(lx - 0.5f), 0) - bx, __float2int_rd(hx - 0.5f) - bx,
                                              max(__float2int_ru(ly - 0.5f), 0) - by, __float2int_rd(hy - 0.5f) - by};
                            bits = candidate_bits(ab, a.z, b.z, rmin, rmax, tile_max, x0, y0, fsx, fsy,
                                                  CellBox{max(box.il, 0), box.ih, max(box.jl, 0), box.jh});
                        } else {
                            bits = ~0ull;
                            plain = true;
                        }
                    }
                }
                __syncwarp();
                store_candidates(s_pmask, q, bits, lane);
            }
            next = RoundTasks<T>(s_items, n_items, R.ref_task, e0 + T::round, total, lane, warp);
            const bool regular = !__syncthreads_or(plain);
            if (!done) {
                Walk<false> walk(s_pmask, slot, n);
                if (regular) {
                    for (;;) {
                        const uint32_t b0 = walk.next();
                        if (b0 == kInvalid) break;
                        const uint32_t b1 = walk.next();
                        const bool two = b1 != kInvalid;
                        const uint32_t c1 = two ? b1 : b0;
                        const float4* ea = s_entry + b0 * kCamEntry;
                        const float4* eb = s_entry + c1 * kCamEntry;
                        const CamPoint p0 = cam_point(mul2, ea, pc), p1 = cam_point(mul2, eb, pc);
                        const float lim = 7.888609052210118e-31f;  // as in shadow_point
                        float q0, q1, w0, w1;
                        unpack2(div2_exact(mul2, sqrt2_exact(mul2, fmaxf(p0.d2, lim), fmaxf(p1.d2, lim)), p0.rr, p1.rr), q0, q1);
                        unpack2(div2_exact(mul2, pack2(p0.num, p1.num), p0.den, p1.den), w0, w1);
                        const Rgba v0 = cam_colour(mul2, ea, __saturatef(__fsub_rn(1.0f, q0)), w0);
                        const Rgba v1 = cam_colour(mul2, eb, __saturatef(__fsub_rn(1.0f, q1)), w1);
                        if (cam_covered(p0)) {
                            land(e0 + b0, s_tag[b0], v0, p0.pz);
                            if (done) break;
                        }
                        if (!two) break;
                        if (cam_covered(p1)) {
                            land(e0 + b1, s_tag[b1], v1, p1.pz);
                            if (done) break;
                        }
                    }
                } else {
                    for (uint32_t bi = walk.next(); bi != kInvalid && !done; bi = walk.next()) {
                        Rgba v;
                        float pz;
                        if (cam_eval(s_entry + bi * kCamEntry, pcx, pcy, v, pz)) land(e0 + bi, s_tag[bi], v, pz);
                    }
                }
                // The item last blended into ends with this round.
                if (!done && lead != kInvalid && s_items.start[item + 1u] <= e0 + n) {
                    blend_group();
                    end_item();
                }
            }
            if (!__syncthreads_or(!done)) break;
        }
        if (active) {
            const size_t pi = (size_t)P.out_base[f] + (size_t)py * d.screen_width + px;  // this pixel's output
            float x, y, z, w;
            unpack2(fin.rg, x, y);
            unpack2(fin.ba, z, w);
            if (w > 1e-6f && w < 1.0f) {
                x /= w;
                y /= w;
                z /= w;
            }
            reinterpret_cast<uint2*>(R.color)[pi] = pack_half4(x, y, z, w);
            R.depth[pi] = gdepth;
            if (P.fragment_counts) R.fragments[pi] = frags;
        }
    }
    if (threadIdx.x == 0) stamp_end(R.stamps, kStampEnd);
}

cudaError_t configure_raster() {
    const auto max_smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_shadow<1>, max_smem, (int)shadow_smem_bytes<1>(kMaxDomSlices));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_shadow<4>, max_smem, (int)shadow_smem_bytes<4>(kMaxDomSlices));
    return e;
}

uint32_t shadow_blocks_per_sm(uint32_t K) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_shadow<1>, (int)Tile<1>::threads, shadow_smem_bytes<1>(K)) !=
        cudaSuccess)
        cudaGetLastError();
    return n > 0 ? (uint32_t)n : 1u;
}

template <uint32_t kSplit>
static void launch_shadow_split(const LaunchCtx& L, const RenderArgs& R, uint32_t K) {
    k_shadow<kSplit><<<L.sm_count * (kSplit == 1 ? 16 : 3), Tile<kSplit>::threads, shadow_smem_bytes<kSplit>(K), L.stream>>>(
        L.P, L.inst, R);
}

void launch_shadow(const LaunchCtx& L, const RenderArgs& R, uint32_t K) { launch_shadow_split<1>(L, R, K); }
void launch_shadow_heavy(const LaunchCtx& L, const RenderArgs& R, uint32_t K) { launch_shadow_split<4>(L, R, K); }

void launch_raster(const LaunchCtx& L, const RenderArgs& R) {
    k_raster<<<L.sm_count * 16, Tile<1>::threads, 0, L.stream>>>(L.P, L.inst, R);
}

}  // namespace fiber
