// pf_kernels.cu - the stages of the GPU-driven fill pipeline for sm_103a.
//
// Stage map (reference -> here):
//   SegmentsD3D11::add_path / SegmentsIter   -> k_contour_segments (count + emit)
//   BuiltPath / round_rect_out_to_tile_bounds -> k_paths
//   dice.comp (here: the d3d9 recursive bisection, tiler.cpp:284-315)
//                                              -> k_flatten_pool<learned|count|write>; k_flatten
//                                                 where segments are shallow
//   bin.comp (here: the d3d9 tile walk + add_fill, tiler.cpp:131-279,
//             object_builder.cpp:19-114),
//   bound.comp (tile records), propagate.comp / Tiler::prepare_tiles
//                                              -> k_bin_fused (one CTA per path: counts, backdrops,
//                                                 offsets, fills grouped by tile; no linked lists);
//                                                 k_bin_small (a warp) for small rects, k_bin_cluster
//                                                 and k_bin_large* for rects too big for a CTA
//   sort.comp (z-culled per-framebuffer-tile lists)
//                                              -> k_rows (per framebuffer row: the spanning paths in
//                                                 path order) + the front-to-back walk of k_composite,
//                                                 which stops at the first occluder; k_list_dump
//                                                 writes the lists out for the canonical read-back
//   fill.comp + tile.comp                      -> k_composite (coverage never leaves the SM)
//   (learned frame) per-path budgets            -> pf_sizer.cu: k_features, k_mlp, k_budgets;
//                                                 here k_flatten_pool and the spill-pool lists
//
// Integer outputs follow the reference's d3d9 CPU tiler bit for bit, so every float
// operation on that path is written with __f*_rn intrinsics (no FMA contraction), in the
// same order as the reference's SSE lanes (pathfinder/common/f32x4.h).
#include <algorithm>
#include <atomic>

#include "pf_internal.h"

namespace pfc {

namespace {

constexpr int kThreads = 256;
// Shared words of the binning's CTA classes (see "Binning by path").
__host__ __device__ constexpr uint32_t class_words(int c) { return c == 0 ? 1088u : c == 1 ? 4352u : 16896u; }
constexpr uint32_t kSmallWords = 128;  // of the class binned by a warp
constexpr int kSmallClass = kRectSmall, kClusterClass = kRectCluster;
// The class binned by a cluster of CTAs, each with the tiles of a band of rows and a word per column
// for two purposes.
constexpr uint32_t kClusterCtas = 4, kClusterTiles = 16384, kClusterCols = 512;
__device__ __forceinline__ uint32_t cluster_rows(uint32_t rh) { return (rh + kClusterCtas - 1) / kClusterCtas; }
__device__ __forceinline__ bool fits_cluster(uint32_t rw, uint32_t rh) {
    return rw <= kClusterCols && (uint64_t)cluster_rows(rh) * rw <= kClusterTiles;
}
// The class that holds a rect; 3: none (global passes).
__device__ __forceinline__ int rect_class(uint32_t rw, uint32_t rh) {
    const uint64_t words = (uint64_t)rw * ((uint64_t)rh + 1);
    return words <= kSmallWords ? kSmallClass
           : words <= class_words(0) ? 0 : words <= class_words(1) ? 1 : words <= class_words(2) ? 2
           : fits_cluster(rw, rh) ? kClusterClass : 3;
}

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// first index i in [0, n) with a[i] > v (a non-decreasing), n if none
__device__ __forceinline__ uint32_t upper_bound(const uint32_t *a, uint32_t n, uint32_t v) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] <= v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t global_tid() { return blockIdx.x * blockDim.x + threadIdx.x; }

inline unsigned grid_for(uint64_t n, int threads = kThreads) {
    return static_cast<unsigned>((n + threads - 1) / threads);
}

// ---------------------------------------------------------------------------
// Per path, one warp: its contours and points in frame-wide numbering (the scenes' offsets are their
// own), its flags, and its bounds and tile rect.
// Outline::bounds (pathfinder/core/data/path.cpp), RectF::intersection and
// round_rect_out_to_tile_bounds (pathfinder/core/data/data.h:131-133), Tiler::Tiler
// (pathfinder/core/d3d9/tiler.cpp:317-335).

// A path of many points is read by its block: a dashed path can have 100,000, and one warp on it
// outlasted the other 19,000 paths (set-up of a stroked batch 0.42 -> 0.19 ms).
constexpr uint32_t kWarpPoints = 4096;
constexpr int kPathThreads = 128;

struct PointBox {
    float l = INFINITY, t = INFINITY, r = -INFINITY, b = -INFINITY;
    uint32_t bad = 0;
    __device__ __forceinline__ void add(const float2 *points, uint32_t i, uint32_t e, uint32_t step) {
#pragma unroll 4
        for (; i < e; i += step) {
            const float2 q = points[i];
            bad |= !(isfinite(q.x) && isfinite(q.y));
            l = fminf(l, q.x);
            t = fminf(t, q.y);
            r = fmaxf(r, q.x);
            b = fmaxf(b, q.y);
        }
    }
    __device__ __forceinline__ void reduce() {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            l = fminf(l, __shfl_xor_sync(0xffffffffu, l, d));
            t = fminf(t, __shfl_xor_sync(0xffffffffu, t, d));
            r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, d));
            b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, d));
        }
        bad = __any_sync(0xffffffffu, bad);
    }
};

__global__ void __launch_bounds__(kPathThreads) k_paths(Batch b, uint2 *path_contours) {
    __shared__ uint2 s_long[kPathThreads / 32];
    __shared__ PointBox s_box[kPathThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t p = blockIdx.x * (kPathThreads / 32) + warp;
    const uint32_t pg = b.path_base + p;
    uint32_t s = 0, c0 = 0, c1 = 0, a = 0, e = 0;
    if (p < b.n_paths) {
        s = upper_bound(b.scene_path_first + b.scene_base, b.n_scenes + 1, pg) - 1 + b.scene_base;
        const SceneDev &S = b.scenes[s];
        const uint32_t local = pg - S.path_first;
        const uint32_t k0 = b.path_start_cat[S.pstart_base + local], k1 = b.path_start_cat[S.pstart_base + local + 1];
        c0 = S.contour_first + k0 - b.contour_base;
        c1 = S.contour_first + k1 - b.contour_base;
        for (uint32_t c = c0 + lane; c < c1; c += 32) b.contour_path[c] = p;
        a = S.point_first + b.contour_start_cat[S.cstart_base + k0];
        e = S.point_first + b.contour_start_cat[S.cstart_base + k1];
    }
    PointBox box;
    const bool many = e > a && e - a > kWarpPoints;
    if (!many) box.add(b.points, a + lane, e, 32);
    if (__syncthreads_or(many)) {
        if (lane == 0) s_long[warp] = many ? make_uint2(a, e) : make_uint2(0u, 0u);
        __syncthreads();
        for (int k = 0; k < kPathThreads / 32; k++) {
            const uint2 range = s_long[k];
            if (range.x == range.y) continue;
            PointBox part;
            part.add(b.points, range.x + threadIdx.x, range.y, kPathThreads);
            part.reduce();
            if (lane == 0) s_box[warp] = part;
            __syncthreads();
            if (k == warp && lane < kPathThreads / 32) box = s_box[lane];
            __syncthreads();
        }
    }
    box.reduce();
    if (p >= b.n_paths) return;
    const SceneDev &S = b.scenes[s];
    float l = box.l, t = box.t, r = box.r, bt = box.b;
    const bool bad = box.bad;
    if (lane != 0) return;
    if (bad) atomicOr(&b.status[kStErr], kErrNonFinite);
    path_contours[p] = make_uint2(c0, c1);
    PathDev P{};
    P.scene = s;
    // occludes: an opaque paint (PaintMetadata::is_opaque): an opaque colour, or a gradient
    // whose stops are all opaque
    bool opaque = (b.color[pg] >> 24) == 0xffu;
    if (b.path_grad && b.path_grad[pg] != kNone) opaque = __float_as_uint(b.grad_meta[4 * b.path_grad[pg] + 3].z) != 0;
    P.flags = (b.fill_rule[pg] ? 1u : 0u) | (opaque ? 2u : 0u);
    if (b.path_clip_cat) {
        // clip paths are tiled like the others but never drawn; a clipped path's clip is in its
        // scene, addressed here within the frame
        if (b.path_is_clip_cat[pg]) P.flags |= kPathIsClip;
        const uint32_t lc = b.path_clip_cat[pg];
        b.path_clip_rel[p] = lc == kNone ? kNone : S.path_first - b.path_base + lc;
    }
    float il, it, ir, ib;
    if (e == a) {  // no points: the default (invalid) RectF {1, 1, 0, 0}
        l = 1.0f;
        t = 1.0f;
        r = 0.0f;
        bt = 0.0f;
    }
    // RectF::intersection with the view box (common/math/rect.h:160-172)
    if (l > S.vb_right || r < S.vb_left || t > S.vb_bottom || bt < S.vb_top) {
        il = 1.0f;
        it = 1.0f;
        ir = 0.0f;
        ib = 0.0f;
    } else {
        il = l < S.vb_left ? S.vb_left : l;
        it = t < S.vb_top ? S.vb_top : t;
        ir = S.vb_right < r ? S.vb_right : r;
        ib = S.vb_bottom < bt ? S.vb_bottom : bt;
    }
    b.path_bounds[p] = make_float4(l, t, r, bt);
    const float inv = 1.0f / kTile;
    P.rx0 = (int32_t)floorf(fmul(il, inv));
    P.ry0 = (int32_t)floorf(fmul(it, inv));
    P.rx1 = (int32_t)ceilf(fmul(ir, inv));
    P.ry1 = (int32_t)ceilf(fmul(ib, inv));
    const int32_t w = max(P.rx1 - P.rx0, 0), h = max(P.ry1 - P.ry0, 0);
    b.paths[p] = P;
    b.path_tiles[p] = (uint32_t)(w * h);
    b.path_cols[p] = (uint32_t)w;
}

// ---------------------------------------------------------------------------
// Segments of a contour, as SegmentsIter::get_next(force_closed = true) yields them
// (pathfinder/core/data/contour.cpp:110-175): stop at the first malformed point pattern;
// at the end, an implicit closing line unless first ~= last within 1e-4.
//
// One warp per contour, a point per lane; or eight lanes, where contours are short on average (up to
// 40 points: a round over the contour's points waits for memory anyway, and four contours' rounds
// wait together).  Every segment ends on the on-curve point the next one
// starts from, so up to the first malformed pattern the segments are the on-curve points but the
// last, each with a kind read off the three flags after it, and their order is a ballot's.  (A
// thread walking its contour point by point: 101 + 16 us for 300,000 glyph contours, 270 + 126 us
// for the 420,000 of a stroked batch, 22 + 11 us where 240 contours are all there is.)
//
// The count pass also looks at the segments of every sample-th contour (about 2048 of them): how
// many would bisect into more than kDeepLines lines, by the flatness value at the root, which a
// bisection shrinks about 16-fold.  launch_flatten picks its kernel by that.
constexpr float kDeepFlatness = 4096.0f;  // 8^4: more than 8 lines

__device__ __forceinline__ bool deep_segment(const float2 *p, uint32_t kind) {
    float m = 0.0f;
    if (kind == kSegQuad) {
        const float dx = p[1].x - 0.5f * (p[0].x + p[2].x), dy = p[1].y - 0.5f * (p[0].y + p[2].y);
        m = 4.0f * (dx * dx + dy * dy);
    } else if (kind == kSegCubic) {
        const float ux = 3.0f * p[1].x - 2.0f * p[0].x - p[3].x, uy = 3.0f * p[1].y - 2.0f * p[0].y - p[3].y;
        const float vx = 3.0f * p[2].x - 2.0f * p[3].x - p[0].x, vy = 3.0f * p[2].y - 2.0f * p[3].y - p[0].y;
        m = fmaxf(ux * ux, vx * vx) + fmaxf(uy * uy, vy * vy);
    }
    return m > kDeepFlatness;
}

template <bool kWrite, int kGroup>
__global__ void __launch_bounds__(kThreads) k_contour_segments(Batch b, uint32_t sample) {
    const int lane = threadIdx.x & 31, shift = lane & ~(kGroup - 1), l = lane & (kGroup - 1);
    const unsigned group = kGroup == 32 ? 0xffffffffu : (1u << (kGroup & 31)) - 1u;
    const uint32_t c = blockIdx.x * (kThreads / kGroup) + threadIdx.x / kGroup;
    uint32_t a = 0, n = 0, out = 0, path = 0;
    if (c < b.n_contours) {
        path = b.contour_path[c];
        if (!kWrite) {
            // the contour's points in frame-wide numbering, kept for the kernels that follow
            const SceneDev &S = b.scenes[b.paths[path].scene];
            const uint32_t *start = b.contour_start_cat + S.cstart_base + (b.contour_base + c - S.contour_first);
            a = S.point_first + start[0];
            n = start[1] - start[0];
            if (l == 0) b.contour_point_first[c] = a;
            if (l == 0 && c == b.n_contours - 1) b.contour_point_first[b.n_contours] = a + n;
        } else {
            a = b.contour_point_first[c];
            n = b.contour_point_first[c + 1] - a;
            out = b.contour_segs[c];
            if (l == 0 && b.path_contours[path].x == c) b.path_seg_first[path] = out;
            if (out > b.seg_cap) n = 0;
        }
    }
    const uint8_t *fl = b.flags + a;
    auto emit = [&](uint32_t k, const SegDev &s) {
        if (k < b.seg_cap) b.segs[k] = s;
        else atomicOr(&b.status[kStErr], kErrOverflowSeg);
    };
    uint32_t count = 0, deep = 0;
    bool ends = n != 0 && fl[0] == 0;  // no malformed pattern so far
    for (uint32_t base = 0; __any_sync(0xffffffffu, ends && base < n); base += kGroup) {
        const uint32_t i = base + (uint32_t)l;
        uint32_t kind = kSegClose;  // none
        bool bad = false;
        if (ends && i < n && fl[i] == 0 && i + 1 < n) {
            const uint8_t f1 = fl[i + 1], f2 = i + 2 < n ? fl[i + 2] : 3, f3 = i + 3 < n ? fl[i + 3] : 3;
            if (f1 == 0) kind = kSegLine;
            else if (f1 == 1 && f2 == 0) kind = kSegQuad;
            else if (f1 == 1 && f2 == 2 && f3 == 0) kind = kSegCubic;
            else bad = true;
        }
        const unsigned bads = __ballot_sync(0xffffffffu, bad) >> shift & group;
        const unsigned before = bads ? (bads & (0u - bads)) - 1u : group;  // lanes before the first one
        const unsigned heads = __ballot_sync(0xffffffffu, kind != kSegClose) >> shift & before;
        const bool head = (heads >> l & 1u) != 0;
        if (kWrite && head) emit(out + count + __popc(heads & ((1u << l) - 1u)), SegDev{a + i, 0, kind, path});
        if (!kWrite) {
            const bool d = head && c % sample == 0 && deep_segment(b.points + a + i, kind);
            deep += __popc(__ballot_sync(0xffffffffu, d) >> shift & group);
        }
        count += __popc(heads);
        ends = ends && bads == 0;
    }
    if (ends && n > 1) {
        const float2 f = b.points[a], z = b.points[a + n - 1];
        const float dx = fsub(f.x, z.x), dy = fsub(f.y, z.y);
        const float len = __fsqrt_rn(fadd(fmul(dx, dx), fmul(dy, dy)));
        if (!(len <= 0.0001f)) {
            if (kWrite && l == 0) emit(out + count, SegDev{a + n - 1, a, kSegClose, path});
            count++;
        }
    }
    if (!kWrite && l == 0 && c < b.n_contours) {
        b.contour_segs[c] = count;
        if (c % sample == 0) {
            atomicAdd(&b.status[kStSampled], count);
            if (deep) atomicAdd(&b.status[kStSampledDeep], deep);
        }
    }
}

// ---------------------------------------------------------------------------
// Flattening: the d3d9 recursive bisection (process_segment, tiler.cpp:284-315) run
// depth first with an explicit stack, so leaves come out in the reference's order.
// Segment::is_flat_cubic (segment.cpp:12-20), is_flat_quadratic (:22-36), split_cubic
// at t = 0.5 (:42-100) and split_quadratic (:102-126), with the same operation order.

__device__ __forceinline__ bool flat_cubic(const float bb[4], const float cc[4]) {
    const float bz[4] = {bb[2], bb[3], bb[0], bb[1]};
    float uv[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float t = fmul(3.0f, cc[k]);
        t = fsub(t, bb[k]);
        t = fsub(t, bb[k]);
        t = fsub(t, bz[k]);
        uv[k] = fmul(t, t);
    }
    const float m0 = uv[0] > uv[2] ? uv[0] : uv[2];
    const float m1 = uv[1] > uv[3] ? uv[1] : uv[3];
    return fadd(m0, m1) <= 1.0f;
}

__device__ __forceinline__ bool flat_quad(const float bb[4], const float cc[2]) {
    const float mx = fmul(fadd(bb[0], bb[2]), 0.5f), my = fmul(fadd(bb[1], bb[3]), 0.5f);
    const float dx = fsub(cc[0], mx), dy = fsub(cc[1], my);
    return fadd(fmul(dx, dx), fmul(dy, dy)) <= 0.25f;
}

__device__ __forceinline__ float half_lerp(float a, float b) { return fadd(a, fmul(0.5f, fsub(b, a))); }

// The stack of pending second halves is kept small, as it lives in local memory: an entry
// holds a half's start point and control points only.  A half ends where the half pushed
// before it (the entry below) begins, or at the segment's end for the bottom entry, because
// each split pushes the second half of the current piece, whose end is the current piece's.
// Depths need no slot either: the path from the root has at most one pending half per depth,
// so a bit mask of pending depths gives the top entry's depth (its highest bit).

template <class Emit>
__device__ void flatten_cubic(float b0, float b1, float b2, float b3, float c0, float c1, float c2, float c3,
                              Emit &&emit, uint32_t *status, int depth0 = 0) {
    float4 sa[kMaxDepth];  // start x, y, first control x, y
    float2 sb[kMaxDepth];  // second control x, y
    uint32_t pending = 0;
    int sp = 0;
    float bb[4] = {b0, b1, b2, b3}, cc[4] = {c0, c1, c2, c3};
    int depth = depth0;
    for (;;) {
        if (depth >= kMaxDepth - 1 || flat_cubic(bb, cc)) {
            if (depth >= kMaxDepth - 1) atomicOr(status, kErrDepth);
            emit(bb[0], bb[1], bb[2], bb[3]);
            if (sp == 0) return;
            sp--;
            const float4 a = sa[sp];
            const float2 c = sb[sp];
            bb[0] = a.x;
            bb[1] = a.y;
            cc[0] = a.z;
            cc[1] = a.w;
            cc[2] = c.x;
            cc[3] = c.y;
            if (sp > 0) {
                const float4 below = sa[sp - 1];
                bb[2] = below.x;
                bb[3] = below.y;
            } else {
                bb[2] = b2;
                bb[3] = b3;
            }
            depth = 31 - __clz(pending);
            pending &= ~(1u << depth);
            continue;
        }
        float p01[2], p12[2], p23[2], p012[2], p123[2], p0123[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            p01[k] = half_lerp(bb[k], cc[k]);
            p12[k] = half_lerp(cc[k], cc[2 + k]);
            p23[k] = half_lerp(cc[2 + k], bb[2 + k]);
            p012[k] = half_lerp(p01[k], p12[k]);
            p123[k] = half_lerp(p12[k], p23[k]);
            p0123[k] = half_lerp(p012[k], p123[k]);
        }
        // push the second half, continue with the first
        sa[sp] = make_float4(p0123[0], p0123[1], p123[0], p123[1]);
        sb[sp] = make_float2(p23[0], p23[1]);
        sp++;
        depth++;
        pending |= 1u << depth;
        bb[2] = p0123[0];
        bb[3] = p0123[1];
        cc[0] = p01[0];
        cc[1] = p01[1];
        cc[2] = p012[0];
        cc[3] = p012[1];
    }
}

template <class Emit>
__device__ void flatten_quad(float b0, float b1, float b2, float b3, float c0, float c1, Emit &&emit,
                             uint32_t *status, int depth0 = 0) {
    float4 sa[kMaxDepth];  // start x, y, control x, y
    uint32_t pending = 0;
    int sp = 0;
    float bb[4] = {b0, b1, b2, b3}, cc[2] = {c0, c1};
    int depth = depth0;
    for (;;) {
        if (depth >= kMaxDepth - 1 || flat_quad(bb, cc)) {
            if (depth >= kMaxDepth - 1) atomicOr(status, kErrDepth);
            emit(bb[0], bb[1], bb[2], bb[3]);
            if (sp == 0) return;
            sp--;
            const float4 a = sa[sp];
            bb[0] = a.x;
            bb[1] = a.y;
            cc[0] = a.z;
            cc[1] = a.w;
            if (sp > 0) {
                const float4 below = sa[sp - 1];
                bb[2] = below.x;
                bb[3] = below.y;
            } else {
                bb[2] = b2;
                bb[3] = b3;
            }
            depth = 31 - __clz(pending);
            pending &= ~(1u << depth);
            continue;
        }
        float a[2], q[2], m[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            a[k] = fadd(bb[k], fmul(fsub(cc[k], bb[k]), 0.5f));
            q[k] = fadd(cc[k], fmul(fsub(bb[2 + k], cc[k]), 0.5f));
            m[k] = fadd(a[k], fmul(fsub(q[k], a[k]), 0.5f));
        }
        sa[sp] = make_float4(m[0], m[1], q[0], q[1]);
        sp++;
        depth++;
        pending |= 1u << depth;
        bb[2] = m[0];
        bb[3] = m[1];
        cc[0] = a[0];
        cc[1] = a[1];
    }
}

template <bool kWrite>
__global__ void __launch_bounds__(kThreads) k_flatten(Batch b, uint32_t n_segs) {
    const uint32_t i = global_tid();
    if (i >= n_segs || i >= b.status[kStSegs]) return;
    if (kWrite && b.status[kStLeaves] > b.leaf_cap) {
        if (i == 0) atomicOr(&b.status[kStErr], kErrOverflowLeaf);
        return;
    }
    const SegDev sg = b.segs[i];
    uint32_t out = kWrite ? b.seg_leaves[i] : 0u;
    uint32_t count = 0;
    auto emit = [&](float x0, float y0, float x1, float y1) {
        if (kWrite) b.leaves[out + count] = make_float4(x0, y0, x1, y1);
        count++;
    };
    const float2 p0 = b.points[sg.a];
    switch (sg.kind) {
        case kSegLine: {
            const float2 p1 = b.points[sg.a + 1];
            emit(p0.x, p0.y, p1.x, p1.y);
        } break;
        case kSegClose: {
            const float2 p1 = b.points[sg.b];
            emit(p0.x, p0.y, p1.x, p1.y);
        } break;
        case kSegQuad: {
            const float2 c = b.points[sg.a + 1], p2 = b.points[sg.a + 2];
            flatten_quad(p0.x, p0.y, p2.x, p2.y, c.x, c.y, emit, &b.status[kStErr]);
        } break;
        default: {
            const float2 c0 = b.points[sg.a + 1], c1 = b.points[sg.a + 2], p3 = b.points[sg.a + 3];
            flatten_cubic(p0.x, p0.y, p3.x, p3.y, c0.x, c0.y, c1.x, c1.y, emit, &b.status[kStErr]);
        } break;
    }
    if (!kWrite) b.seg_leaves[i] = count;
}

// ---------------------------------------------------------------------------
// Binning: the d3d9 tile walk of one leaf line (process_line_segment, tiler.cpp:131-279),
// with clip_line_segment_to_rect (:46-125, clip box top = -inf), ObjectBuilder::add_fill
// (object_builder.cpp:19-64: cull outside the tile rect, x256 local coordinates, clamp to
// [0, 4095], round half to even, cull vertical) and adjust_alpha_tile_backdrop (:96-114).

struct WalkCtx {
    int32_t rx0, ry0, rx1, ry1, rw, rh;
    float vb_left, vb_right, vb_bottom;  // the clip box: the view box with its top at -infinity
};

__device__ __forceinline__ int outcode(const WalkCtx &w, float x, float y) {
    int o = 0;
    if (x < w.vb_left) o |= 1;
    else if (x > w.vb_right) o |= 2;
    if (y > w.vb_bottom) o |= 8;
    return o;
}

__device__ __forceinline__ float lerp_clamped(float a, float b, float t) {
    t = t < 0.0f ? 0.0f : (t > 1.0f ? 1.0f : t);
    return fadd(a, fmul(fsub(b, a), t));
}

__device__ __forceinline__ int clip_line(const WalkCtx &w, float &x0, float &y0, float &x1, float &y1,
                                         uint32_t *status) {
    int of = outcode(w, x0, y0), ot = outcode(w, x1, y1);
    for (int iter = 0; iter < 64; iter++) {
        if (of == 0 && ot == 0) return 1;
        if ((of & ot) != 0) return 0;
        const bool clip_from = of > ot;
        const int oc = clip_from ? of : ot;
        float px = clip_from ? x0 : x1, py = clip_from ? y0 : y1;
        if (oc & 1) {
            px = w.vb_left;
            py = lerp_clamped(y0, y1, fdiv(fsub(w.vb_left, x0), fsub(x1, x0)));
        } else if (oc & 2) {
            px = w.vb_right;
            py = lerp_clamped(y0, y1, fdiv(fsub(w.vb_right, x0), fsub(x1, x0)));
        } else if (oc & 8) {
            px = lerp_clamped(x0, x1, fdiv(fsub(w.vb_bottom, y0), fsub(y1, y0)));
            py = w.vb_bottom;
        }
        if (clip_from) {
            x0 = px;
            y0 = py;
            of = outcode(w, px, py);
        } else {
            x1 = px;
            y1 = py;
            ot = outcode(w, px, py);
        }
    }
    atomicOr(status, kErrClip);
    return 0;
}

// Quantise a piece of line in tile (tx, ty); returns false when add_fill culls it.
__device__ __forceinline__ bool quantise(const WalkCtx &w, float x0, float y0, float x1, float y1, int32_t tx,
                                         int32_t ty, uint2 &packed) {
    if (!(w.rx0 <= tx && tx <= w.rx1 - 1 && w.ry0 <= ty && ty <= w.ry1 - 1)) return false;
    const float ox = fmul((float)tx, 16.0f), oy = fmul((float)ty, 16.0f);
    float v[4] = {fmul(fsub(x0, ox), 256.0f), fmul(fsub(y0, oy), 256.0f), fmul(fsub(x1, ox), 256.0f),
                  fmul(fsub(y1, oy), 256.0f)};
    uint32_t q[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        float c = v[k] > 0.0f ? v[k] : 0.0f;
        c = c < 4095.0f ? c : 4095.0f;
        q[k] = (uint32_t)rintf(c);
    }
    if (q[0] == q[2]) return false;
    packed = make_uint2(q[0] | (q[1] << 16), q[2] | (q[3] << 16));
    return true;
}

// Walk of one line, split into a set-up and steps.  A step has a decision - which tile
// boundary the line crosses next and at which parameter (crossing parameters accumulate, so
// decisions are sequential) - and an emission: the fill(s) and backdrop delta of the tile,
// which depend only on that step's decision and the one before.  on_fill(local_tile, packed)
// for every fill kept; on_delta(local_tile or -1 - column, delta) for every backdrop change
// that lands in the rect or above it.
struct WalkState {
    float x0, y0, vx, vy, tmx, tmy, tdx, tdy, curx, cury;
    int32_t tcx, tcy, ex, ey, sx, sy;
    int last;  // 0 none, 1 x, 2 y
    uint32_t it;
};

struct WalkStep {
    float curx, cury, nt;
    int32_t tcx, tcy;
    int last, next;
};

// False when nothing is left to step: a non-finite or clipped-away line, or a line inside one
// tile, whose single fill is emitted here.
template <class OnFill>
__device__ __forceinline__ bool walk_begin(const WalkCtx &w, float x0, float y0, float x1, float y1, WalkState &s,
                                           OnFill &&on_fill, uint32_t *status) {
    if (!(isfinite(x0) && isfinite(y0) && isfinite(x1) && isfinite(y1))) return false;
    if (!clip_line(w, x0, y0, x1, y1, status)) return false;
    const float inv = 1.0f / kTile;
    const int32_t fx = (int32_t)floorf(fmul(x0, inv)), fy = (int32_t)floorf(fmul(y0, inv));
    const int32_t ex = (int32_t)floorf(fmul(x1, inv)), ey = (int32_t)floorf(fmul(y1, inv));
    const float vx = fsub(x1, x0), vy = fsub(y1, y0);
    if (fx == ex && fy == ey) {
        // A line inside one tile: the walk would stop at its first step with t = 1 (the next
        // tile boundary in each direction lies beyond the end point, so both crossing
        // parameters are >= 1 or infinite), add the one fill from (x0, y0) to
        // (x0 + vx * 1, y0 + vy * 1), and neither an extra fill nor a backdrop delta.
        uint2 q;
        if (quantise(w, x0, y0, fadd(x0, vx), fadd(y0, vy), fx, fy, q))
            on_fill((fy - w.ry0) * w.rw + (fx - w.rx0), q);
        return false;
    }
    s.x0 = x0;
    s.y0 = y0;
    s.vx = vx;
    s.vy = vy;
    s.sx = vx < 0.0f ? -1 : 1;
    s.sy = vy < 0.0f ? -1 : 1;
    const float cx = fmul(fadd((float)fx, vx >= 0.0f ? 1.0f : 0.0f), 16.0f);
    const float cy = fmul(fadd((float)fy, vy >= 0.0f ? 1.0f : 0.0f), 16.0f);
    s.tmx = fdiv(fsub(cx, x0), vx);
    s.tmy = fdiv(fsub(cy, y0), vy);
    s.tdx = fabsf(fdiv(16.0f, vx));
    s.tdy = fabsf(fdiv(16.0f, vy));
    s.curx = x0;
    s.cury = y0;
    s.tcx = fx;
    s.tcy = fy;
    s.ex = ex;
    s.ey = ey;
    s.last = 0;
    s.it = 0;
    return true;
}

// The decision of the next step, which it records, and the walk state advanced past it;
// false once the line is done (or the step bound is hit).
__device__ __forceinline__ bool walk_decide(WalkState &s, WalkStep &r, uint32_t *status) {
    if (s.it >= kMaxWalk) {
        atomicOr(status, kErrWalk);
        r.next = -1;  // nothing to emit
        return false;
    }
    s.it++;
    int next;
    if (s.tmx < s.tmy) next = 1;
    else if (s.tmx > s.tmy) next = 2;
    else next = s.sx > 0 ? 1 : 2;
    float nt = next == 1 ? s.tmx : s.tmy;
    nt = (1.0f < nt) ? 1.0f : nt;
    if (s.tcx == s.ex && s.tcy == s.ey) next = 0;
    r.curx = s.curx;
    r.cury = s.cury;
    r.nt = nt;
    r.tcx = s.tcx;
    r.tcy = s.tcy;
    r.last = s.last;
    r.next = next;
    if (next == 1) {
        s.tmx = fadd(s.tmx, s.tdx);
        s.tcx += s.sx;
    } else if (next == 2) {
        s.tmy = fadd(s.tmy, s.tdy);
        s.tcy += s.sy;
    } else {
        return false;
    }
    s.curx = fadd(s.x0, fmul(s.vx, nt));
    s.cury = fadd(s.y0, fmul(s.vy, nt));
    s.last = next;
    return true;
}

// The fills and backdrop delta of one decided step.
template <class OnFill, class OnDelta>
__device__ __forceinline__ void walk_emit(const WalkCtx &w, const WalkState &s, const WalkStep &r, OnFill &&on_fill,
                                          OnDelta &&on_delta) {
    const float npx = fadd(s.x0, fmul(s.vx, r.nt)), npy = fadd(s.y0, fmul(s.vy, r.nt));
    const int32_t lx = r.tcx - w.rx0, ly = r.tcy - w.ry0;
    uint2 q;
    if (quantise(w, r.curx, r.cury, npx, npy, r.tcx, r.tcy, q)) on_fill(ly * w.rw + lx, q);
    if (s.sy < 0 && r.next == 2) {
        if (quantise(w, npx, npy, fmul((float)r.tcx, 16.0f), fmul((float)r.tcy, 16.0f), r.tcx, r.tcy, q))
            on_fill(ly * w.rw + lx, q);
    } else if (s.sy > 0 && r.last == 2) {
        if (quantise(w, fmul((float)r.tcx, 16.0f), fmul((float)r.tcy, 16.0f), r.curx, r.cury, r.tcx, r.tcy, q))
            on_fill(ly * w.rw + lx, q);
    }
    int delta = 0;
    if (s.sx < 0 && r.last == 1) delta = 1;
    else if (s.sx > 0 && r.next == 1) delta = -1;
    if (delta != 0 && lx >= 0 && lx < w.rw && ly < w.rh) {
        if (ly < 0) on_delta(-1 - lx, delta);
        else on_delta(ly * w.rw + lx, delta);
    }
}

// One lane walks one line.
template <class OnFill, class OnDelta>
__device__ void walk_line(const WalkCtx &w, float x0, float y0, float x1, float y1, OnFill &&on_fill,
                          OnDelta &&on_delta, uint32_t *status) {
    WalkState s;
    if (!walk_begin(w, x0, y0, x1, y1, s, on_fill, status)) return;
    for (;;) {
        WalkStep r;
        const bool more = walk_decide(s, r, status);
        if (r.next >= 0) walk_emit(w, s, r, on_fill, on_delta);
        if (!more) return;
    }
}

// The whole warp walks one (long) line: every lane runs the same sequence of decisions, lane
// j % 32 keeps step j, and the lanes emit their steps together, 32 steps per round.  The
// decisions are a few instructions each, the emissions (clip, quantise, fills) the bulk.
template <class OnFill, class OnDelta>
__device__ void walk_line_warp(const WalkCtx &w, float4 f, OnFill &&on_fill, OnDelta &&on_delta, uint32_t *status) {
    const int lane = threadIdx.x & 31;
    WalkState s;
    if (!walk_begin(w, f.x, f.y, f.z, f.w, s,
                    [&](int32_t local, uint2 q) {
                        if (lane == 0) on_fill(local, q);
                    },
                    status))
        return;
    bool more = true;
    while (more) {
        WalkStep mine;
        mine.next = -1;
#pragma unroll 1
        for (int j = 0; j < 32 && more; j++) {
            WalkStep r;
            more = walk_decide(s, r, status);
            if (j == lane) mine = r;
        }
        if (mine.next >= 0) walk_emit(w, s, mine, on_fill, on_delta);
        __syncwarp();
    }
}

// The same walk for 32 lines at once, one per lane, with the lanes in step: the walk the binning
// kernels spend their time in.  It is bound by instructions, so it does the reference's float
// operations in the form that takes fewest:
//
// * Coordinates are kept in tiles (x / 16), which changes no rounding: scaling by a power of two
//   is exact, so boundaries, parameters and positions are the same values over 16.  (It is not
//   exact below 2^-122; a line with such a coordinate takes walk_line.)
// * add_fill's quantisation of a coordinate v (times 256, rounded half to even, clamped to
//   [0, 4095]) is a subtract of the tile and one fused multiply-add to 1.5 * 2^23, whose low
//   mantissa bits are then the rounded integer (the product is exact, so the addition rounds
//   once, as rint does), and one clamp of both coordinates as packed 16-bit integers.
// * A crossing point is quantised once, in the tile it leaves; the tile it enters differs by one
//   in the crossed coordinate, which is 4096 in quantised units.  (Both subtractions of the tile
//   are exact, or - around the axes, where a coordinate has finer bits than the difference - the
//   point is so close to the boundary that both forms give 0 and 4095.)
// * The extra fill of a vertical crossing runs between the crossing point and the tile's corner,
//   which quantises to (0, 0): it reuses the quantised crossing point.
// * A tile visit's fills and backdrop delta are added to the tile's counter with one atomic.
// * One reciprocal per direction gives the boundary spacing: |1 / vx| is |16 / vx| over 16.
// * A line takes one step per tile boundary between its end points' tiles, so the loop is counted.
//   A walk that rounding sends past one of those boundaries never comes to the end tile (steps
//   only go on from it): it reports the walk error after its last step instead of at the step bound.
// With the tile visits staged as they are walked (12 bytes for up to two fills, their slots from a
// ballot instead of a counter in shared memory) binning takes, against one walk_line per lane:
// 10.00 -> 7.86 ms on 256 scenes (162M lines, 485M fills), 1.05 -> 0.81 ms on 20,000 paths.  A round
// of 32 steps is about 90 instructions, the set-up of 32 lines about 150.
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
constexpr uint32_t kFillMax = 0x0fff0fffu;
constexpr int32_t kMaxLaneSpan = 255;  // tiles; longer lines are always walked by the whole warp

// a tile-unit point in tile (tx, ty), rounded to 1/256 px but not clamped: x | y << 16, signed
__device__ __forceinline__ uint32_t round_point(float x, float y, float tx, float ty) {
    const float qx = __fmaf_rn(fsub(x, tx), 4096.0f, kMagic), qy = __fmaf_rn(fsub(y, ty), 4096.0f, kMagic);
    return __byte_perm(__float_as_uint(qx), __float_as_uint(qy), 0x5410);
}

// One line of a lane.
struct LaneLine {
    float x0, y0, vx, vy, tmx, tmy, tdx, tdy, ftx, fty, fex;
    uint32_t pa;     // the tile's first point, quantised
    int32_t lx, ly;  // the first tile, in the path's rect
    int32_t steps;   // tile boundaries to cross; -1: no line
    bool right, down;
};

// The steps of up to 32 lines.  visit(live, m, e, pa, pb, down, local, inc) is called by all lanes
// once per step: live, the lane's line is still being walked; m, the tile's fill (pa, pb) is kept;
// e, the vertical crossing's extra fill - (0, pa) going down, (pb, 0) going up - is kept; inc, the
// number of both plus the backdrop delta << 24.  The values are meaningless unless live.
// kChecked: tiles may lie outside the path's rect, and on_above(column, delta) gets the deltas above it.
template <bool kChecked, class Visit, class OnAbove>
__device__ __forceinline__ void lane_steps(const WalkCtx &w, const LaneLine &s, int32_t steps, Visit &&visit,
                                           OnAbove &&on_above, uint32_t *status) {
    float tmx = s.tmx, tmy = s.tmy, ftx = s.ftx, fty = s.fty;
    int32_t lx = s.lx, ly = s.ly;
    uint32_t local = (uint32_t)(s.ly * w.rw + s.lx);
    uint32_t pa = s.pa;
    uint32_t last = 0;  // the boundary the tile was entered through: 0 none, 1 vertical, 2 horizontal
    const int32_t sx = s.right ? 1 : -1, sy = s.down ? 1 : -1, srow = s.down ? w.rw : -w.rw;
    const float sxf = s.right ? 1.0f : -1.0f, syf = s.down ? 1.0f : -1.0f;
    const uint32_t shx = s.right ? 0xf000u : 0x1000u, shy = s.down ? 0xf0000000u : 0x10000000u;
    const uint32_t dval = s.right ? 0xff000000u : 0x01000000u, top = (uint32_t)(w.rw * w.rh) - 1u;
    const int32_t rounds = __reduce_max_sync(0xffffffffu, steps);
    bool lost = false;
#pragma unroll 1
    for (int32_t it = 0; it <= rounds; it++) {
        const bool live = it <= steps, done = it == steps;
        const bool stepx = tmx < tmy || (s.right && tmx <= tmy);
        const uint32_t next = done ? 0u : stepx ? 1u : 2u;
        const float nt = fminf(fminf(tmx, tmy), 1.0f);
        const uint32_t pu = round_point(fadd(s.x0, fmul(s.vx, nt)), fadd(s.y0, fmul(s.vy, nt)), ftx, fty);
        const uint32_t pb = __vimin_s16x2_relu(pu, kFillMax);
        bool m = ((pa ^ pb) & 0xffffu) != 0;
        bool e = (s.down ? last : next) == 2u && ((s.down ? pa : pb) & 0xffffu) != 0;
        const bool cross = (s.right ? next : last) == 1u;
        uint32_t d = cross ? dval : 0u;
        if (kChecked) {
            const bool col = (uint32_t)lx < (uint32_t)w.rw, in = col && (uint32_t)ly < (uint32_t)w.rh;
            if (live && col && ly < 0 && cross) on_above(lx, s.right ? -1 : 1);
            m = m && in;
            e = e && in;
            d = in ? d : 0u;
            local = (uint32_t)(ly * w.rw + lx);
        } else {
            local = min(local, top);  // a lost line's tiles stay inside the counters
        }
        visit(live, m, e, pa, pb, s.down, local, (uint32_t)m + (uint32_t)e + d);
        lost = lost || (done && ftx != s.fex);
        pa = __viaddmin_s16x2_relu(pu, stepx ? shx : shy, kFillMax);
        tmx = fadd(tmx, stepx ? s.tdx : 0.0f);
        tmy = fadd(tmy, stepx ? 0.0f : s.tdy);
        ftx += stepx ? sxf : 0.0f;
        fty += stepx ? 0.0f : syf;
        if (kChecked) {
            lx += stepx ? sx : 0;
            ly += stepx ? 0 : sy;
        } else {
            local += (uint32_t)(stepx ? sx : srow);
        }
        last = next;
    }
    if (lost) atomicOr(status, kErrWalk);
}

// Walks 32 lines (have: this lane has one).  Lines spanning more than long_line tiles are walked by
// the whole warp, one after the other - unless they are so many that 32 lanes in step are done sooner: a
// step in lockstep costs what some four of a warp's do, so where the long lines' steps add up to more than
// four times the longest's, they stay with their lanes.  (A hatching of 1,000 paths with 400 lines of
// about 100 tiles: binning 4.80 -> 2.02 ms; of 40 tiles 0.97 -> 0.32; 256 scenes the same.)  The few
// outside the fast form's range (coordinates beyond 2^20, or tiny) are walked by their lane alone, both
// with on_fill / on_delta after begin_single() and before end_single().
template <class Visit, class OnAbove, class OnFill, class OnDelta, class Begin, class End>
__device__ __forceinline__ void walk_lines(const WalkCtx &w, float4 f, bool have, float long_line, Visit &&visit,
                                           OnAbove &&on_above, OnFill &&on_fill, OnDelta &&on_delta,
                                           Begin &&begin_single, End &&end_single, uint32_t *status) {
    const float inv = 1.0f / kTile, low = -1048576.0f;
    LaneLine s;
    s.x0 = s.y0 = s.vx = s.vy = s.ftx = s.fty = 0.0f;
    s.tmx = s.tmy = s.tdx = s.tdy = INFINITY;
    s.fex = 0.0f;
    s.pa = 0;
    s.lx = s.ly = 0;
    s.steps = -1;
    s.right = s.down = true;
    bool alone = false, along = false, safe = true;
    if (have) {
        float ax = f.x, ay = f.y, bx = f.z, by = f.w;
        const bool inside = ax >= w.vb_left && ax <= w.vb_right && ay <= w.vb_bottom && bx >= w.vb_left &&
                            bx <= w.vb_right && by <= w.vb_bottom;
        bool keep = true;
        if (!inside) {
            keep = isfinite(ax) && isfinite(ay) && isfinite(bx) && isfinite(by);
            if (keep) keep = clip_line(w, ax, ay, bx, by, status);
        }
        if (keep) {
            alone = !(ay >= low && by >= low);
            s.x0 = fmul(ax, inv);
            s.y0 = fmul(ay, inv);
            const float x1 = fmul(bx, inv), y1 = fmul(by, inv);
            s.vx = fsub(x1, s.x0);
            s.vy = fsub(y1, s.y0);
            s.ftx = floorf(s.x0);
            s.fty = floorf(s.y0);
            const int32_t lx = (int32_t)s.ftx - w.rx0, ly = (int32_t)s.fty - w.ry0;
            s.fex = floorf(x1);
            const int32_t ex = (int32_t)s.fex - w.rx0, ey = (int32_t)floorf(y1) - w.ry0;
            s.lx = lx;
            s.ly = ly;
            s.right = s.vx >= 0.0f;
            s.down = s.vy >= 0.0f;
            s.pa = __vimin_s16x2_relu(round_point(s.x0, s.y0, s.ftx, s.fty), kFillMax);
            safe = max((uint32_t)lx, (uint32_t)ex) < (uint32_t)w.rw && max((uint32_t)ly, (uint32_t)ey) < (uint32_t)w.rh;
            const int32_t nx = abs(ex - lx), ny = abs(ey - ly);
            s.steps = nx + ny;
            // a line inside one tile goes to its end at once (t = 1)
            if (s.steps != 0 && !alone) {
                // 2 |bits| - 1 is below 2^-122's for tiny values only (zero wraps to the largest)
                const uint32_t tiny = min(min(2u * __float_as_uint(ax) - 1u, 2u * __float_as_uint(ay) - 1u),
                                          min(2u * __float_as_uint(bx) - 1u, 2u * __float_as_uint(by) - 1u));
                alone = tiny < 2u * 0x02800000u - 1u;
                along = !alone && ((float)(s.steps + 1) > long_line || s.steps > kMaxLaneSpan);
                s.tmx = fdiv(fsub(s.right ? s.ftx + 1.0f : s.ftx, s.x0), s.vx);
                s.tmy = fdiv(fsub(s.down ? s.fty + 1.0f : s.fty, s.y0), s.vy);
                s.tdx = fabsf(__frcp_rn(s.vx));
                s.tdy = fabsf(__frcp_rn(s.vy));
            }
            if (alone) s.steps = -1;
        }
    }
    unsigned k = __ballot_sync(0xffffffffu, along);
    if (k) {
        const int32_t steps = along ? s.steps : 0;
        if (__reduce_add_sync(0xffffffffu, steps) > 4 * __reduce_max_sync(0xffffffffu, steps)) {
            along = along && steps > kMaxLaneSpan;
            k = __ballot_sync(0xffffffffu, along);
        }
        if (along) s.steps = -1;
    }
    lane_steps<false>(w, s, safe ? s.steps : -1, visit, on_above, status);
    if (!__all_sync(0xffffffffu, safe)) lane_steps<true>(w, s, safe ? -1 : s.steps, visit, on_above, status);
    if (k || __any_sync(0xffffffffu, alone)) {
        begin_single();
        if (alone) walk_line(w, f.x, f.y, f.z, f.w, on_fill, on_delta, status);
        for (; k; k &= k - 1) {
            const int l = __ffs(k) - 1;
            const float4 g = make_float4(__shfl_sync(0xffffffffu, f.x, l), __shfl_sync(0xffffffffu, f.y, l),
                                         __shfl_sync(0xffffffffu, f.z, l), __shfl_sync(0xffffffffu, f.w, l));
            walk_line_warp(w, g, on_fill, on_delta, status);
        }
        end_single();
    }
}

// Flattening shared by the lanes of a warp, for both frames:
// * learned frame: each path's leaf lines go to the path's region, laid out from
//   the sizer's budget; lines past the budget spill into the shared pool, and an exhausted pool
//   sets the overflow bit (the frame is then redone by the exact two-pass method);
// * exact frame's write pass: each segment's lines go to its range of the leaf
//   buffer, counted by the count pass;
// * exact frame's count pass: only the number of each segment's lines is kept.
//
// The bisection is shared by the 32 lanes of a warp.  With one segment per lane (as k_flatten does where
// segments are shallow) a warp runs the split branch and the emit branch of every step one after
// the other, with only the lanes on one side doing work in each (13 of 32 lanes active on the
// 512-scene batch; flattening took 5.93 ms of the learned frame that way, and 4.54 when this form came
// in).  Here the lanes share the work of the warp's segments instead:
//
// * a split round: each lane takes a pending (not flat) piece from the warp's pool in shared
//   memory, splits it at t = 0.5, and tests both halves: a flat half (or one at the depth bound)
//   joins the warp's leaf queue (count pass: adds to its segment's count), the other goes back on
//   the pool;
// * an emit round: each lane takes a queued leaf line and stores it.  Learned frame: the
//   segment's first leaf (its leftmost piece) at the segment's own slot in its path's region, the
//   others at slots reserved with one atomic per path among the round's lines (lanes grouped by
//   path) and stored one round later, so that the atomic's round trip overlaps the next split
//   round; lines past the budget go to the spill pool.  Exact frame: at the next slots of the
//   segment's range, from a counter in the warp's segment table (no global atomics).
//
// Every piece is split with the same operations as in the depth-first walk, so the leaf lines
// are the same lines bit for bit; only their order within a path's region differs, which no
// output depends on (fills are counted and placed per tile, coverage sums are integers).  The
// pool is a stack, so it stays near 32 pieces per level of the warp's deepest segments; a half
// that finds it full is flattened depth first by its lane alone.  The pool and the segment table are
// what limits the warps per SM, so they are as small as that stays rare: 256 scenes by the learned
// frame, 2.00 ms with 224 pieces and 128 segments, 1.89 with 192 and 64 (11 blocks per SM instead of
// 9), 1.95 with 176; taking fewer pieces when the pool is nearly full, so that none is left alone,
// 1.96.  The exact passes keep 128 segments (stroked batch 0.565 ms with 224 pieces, 0.548 with 192,
// 0.576 with 64 segments).  Warps take their segments a group at a time from
// a frame-wide ticket: 32, or fewer (a power of two) when that would leave a resident warp under 8
// groups, so the last groups end together and small frames use every SM.  A group's slots in the
// segment table are reused once no pending piece or queued line refers to them.
//
// Segments are taken as they lie.  Sorting them by depth first (four kernels, 33 us with 700,000
// segments) had kept the last groups small and, when a lane flattened its segment alone, a warp's
// lanes alike; with shared lanes and small groups it no longer pays (flattening and binning, sorted
// against not: 256 scenes by the learned frame 10.06 / 10.00 ms, 20,000 paths 1.26 / 1.28 ms, 24
// clipped scenes 0.72 / 0.70 ms, 240 paths 0.20 / 0.18 ms).
constexpr int kPoolWarps = 2;     // warps per block
constexpr int kPoolCap = 192;     // pending pieces per warp
constexpr int kPoolLeafCap = 96;  // queued leaf lines per warp: < 32 before a round, + 2 per lane
enum : int { kPoolLearned = 0, kPoolCount = 1, kPoolWrite = 2 };
// segments in flight per warp (at most 32 groups)
__host__ __device__ constexpr int pool_entries(int mode) { return mode == kPoolLearned ? 64 : 128; }
// piece and line tags: bits 0-6 the segment's table entry (group * 32 + lane), bit 7 the
// segment's leftmost piece, bit 8 a cubic (else a quadratic), bits 9-13 the depth
constexpr uint32_t kTagEntry = 127u, kTagLeft = 1u << 7, kTagCubic = 1u << 8;
constexpr int kTagDepthShift = 9;

template <int kMode>
struct FlattenPool {
    float4 pend_ends[kPoolCap];   // x0, y0, x1, y1
    float4 pend_ctrl[kPoolCap];   // first control x, y, second control x, y (quadratic: first only)
    uint32_t pend_tag[kPoolCap];
    float4 leaf[kMode == kPoolCount ? 1 : kPoolLeafCap];  // x0, y0, x1, y1
    uint32_t leaf_tag[kMode == kPoolCount ? 1 : kPoolLeafCap];
    // learned frame: path, region, budget, own slot; write pass: the segment's first leaf slot and
    // its lines stored so far; count pass: the segment (kNone: none) and its lines so far
    uint4 seg[kMode == kPoolLearned ? pool_entries(kMode) : 1];
    uint2 seg2[kMode == kPoolLearned ? 1 : pool_entries(kMode)];
};

// Where a lane stores leaf lines by itself.
struct LeafSink {
    float4 *leaves;
    uint32_t *cursor, *status, *pool_path;
    uint32_t pool_first, pool_cap;
};

// A half that found the pool full: flattened depth first from its depth, its lines stored one
// slot at a time.  Returns the lines it produced.
__device__ __noinline__ uint32_t flatten_piece_alone(LeafSink out, uint4 sg, float4 ends, float4 ctrl, uint32_t tag) {
    bool left = (tag & kTagLeft) != 0;
    uint32_t produced = 0;
    auto emit = [&](float x0, float y0, float x1, float y1) {
        const float4 v = make_float4(x0, y0, x1, y1);
        produced++;
        if (left) {
            out.leaves[sg.w] = v;
            left = false;
            return;
        }
        const uint32_t slot = atomicAdd(&out.cursor[sg.x], 1u);
        if (slot < sg.z) {
            out.leaves[sg.y + slot] = v;
            return;
        }
        if (slot == sg.z) atomicAdd(&out.status[kStPathsOver], 1u);
        const uint32_t j = atomicAdd(&out.status[kStPoolUsed], 1u);
        if (j < out.pool_cap) {
            out.leaves[out.pool_first + j] = v;
            out.pool_path[j] = sg.x;
        } else {
            atomicOr(&out.status[kStErr], kErrOverflowLeaf);
        }
    };
    const int depth = (int)(tag >> kTagDepthShift) & 31;
    if (tag & kTagCubic)
        flatten_cubic(ends.x, ends.y, ends.z, ends.w, ctrl.x, ctrl.y, ctrl.z, ctrl.w, emit, &out.status[kStErr],
                      depth);
    else
        flatten_quad(ends.x, ends.y, ends.z, ends.w, ctrl.x, ctrl.y, emit, &out.status[kStErr], depth);
    return produced;
}

// The same for the exact frame: the segment's lines go to its range of the leaf buffer (from the
// count pass), the next slot taken from the segment's counter in the warp's table.
__device__ __noinline__ void flatten_piece_alone_exact(float4 *leaves, uint32_t leaf_cap, uint32_t *status,
                                                       uint32_t *stored, uint32_t first, float4 ends, float4 ctrl,
                                                       uint32_t tag) {
    auto emit = [&](float x0, float y0, float x1, float y1) {
        const uint32_t idx = first + atomicAdd(stored, 1u);
        if (idx < leaf_cap) leaves[idx] = make_float4(x0, y0, x1, y1);
        else atomicOr(&status[kStErr], kErrOverflowLeaf);
    };
    const int depth = (int)(tag >> kTagDepthShift) & 31;
    if (tag & kTagCubic)
        flatten_cubic(ends.x, ends.y, ends.z, ends.w, ctrl.x, ctrl.y, ctrl.z, ctrl.w, emit, &status[kStErr], depth);
    else
        flatten_quad(ends.x, ends.y, ends.z, ends.w, ctrl.x, ctrl.y, emit, &status[kStErr], depth);
}

// And for the count pass: the number of the piece's lines.
__device__ __noinline__ uint32_t count_piece_alone(uint32_t *status, float4 ends, float4 ctrl, uint32_t tag) {
    uint32_t n = 0;
    auto emit = [&](float, float, float, float) { n++; };
    const int depth = (int)(tag >> kTagDepthShift) & 31;
    if (tag & kTagCubic)
        flatten_cubic(ends.x, ends.y, ends.z, ends.w, ctrl.x, ctrl.y, ctrl.z, ctrl.w, emit, &status[kStErr], depth);
    else
        flatten_quad(ends.x, ends.y, ends.z, ends.w, ctrl.x, ctrl.y, emit, &status[kStErr], depth);
    return n;
}

__device__ __forceinline__ bool piece_flat(bool cubic, float4 e, float4 c) {
    const float bb[4] = {e.x, e.y, e.z, e.w}, cc[4] = {c.x, c.y, c.z, c.w};
    return cubic ? flat_cubic(bb, cc) : flat_quad(bb, cc);
}

template <int kMode>
__global__ void __launch_bounds__(kPoolWarps * 32) k_flatten_pool(Batch b, uint32_t n_segs, int group_shift) {
    __shared__ FlattenPool<kMode> pools[kPoolWarps];
    FlattenPool<kMode> &W = pools[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    uint32_t *const err = &b.status[kStErr];
    if (kMode == kPoolWrite && b.status[kStLeaves] > b.leaf_cap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, kErrOverflowLeaf);
        return;
    }
    n_segs = min(n_segs, b.status[kStSegs]);
    constexpr int kTicket = kMode == kPoolWrite ? kStFlatTicket2 : kStFlatTicket;
    const uint32_t group = 1u << group_shift, n_groups = (n_segs + group - 1u) >> group_shift;
    const uint32_t n_sets = min(32u, (uint32_t)pool_entries(kMode) >> group_shift);
    const uint32_t all_sets = n_sets == 32u ? ~0u : (1u << n_sets) - 1u;
    // a group of segments: lane 0 takes the ticket, and the lanes read it when they need it, so the
    // atomic's round trip overlaps the work in between
    uint32_t ticket = lane == 0 ? atomicAdd(&b.status[kTicket], 1u) : 0u;
    auto current_group = [&]() { return __shfl_sync(~0u, ticket, 0); };
    uint32_t open = 0;  // count pass: the table's groups whose counts are not stored yet
    auto store_counts = [&](uint32_t set) {
        if ((uint32_t)lane < group) {
            const uint2 c = W.seg2[(set << group_shift) + lane];
            if (c.x != kNone) b.seg_leaves[c.x] = c.y;
        }
    };
    int top = 0, nleaf = 0;  // pool and queue sizes (the same in every lane)
    uint32_t produced = 0;

    // An emit round reserves its lines' slots and stores them one round later: the reservation's
    // round trip overlaps the split rounds in between.  The lines waiting for their slots:
    bool held = false;                                   // this lane holds one
    float4 held_line = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    uint32_t held_path = 0, held_region = 0, held_budget = 0;
    uint32_t held_first = 0;                             // the reservation's first slot (its leader lane)
    uint32_t held_count = 0, held_rank = 0;
    int held_leader = 0;
    auto store_held = [&]() {
        const unsigned held_mask = __ballot_sync(~0u, held);
        if (!held_mask) return;
        bool spill = false;
        if (held) {
            const uint32_t slot = __shfl_sync(held_mask, held_first, held_leader) + held_rank;
            if (lane == held_leader && held_first <= held_budget && held_first + held_count > held_budget)
                atomicAdd(&b.status[kStPathsOver], 1u);
            spill = slot >= held_budget;
            if (!spill) b.leaves[held_region + slot] = held_line;
        }
        const unsigned spill_mask = __ballot_sync(~0u, spill);
        if (spill_mask) {
            const int first = __ffs(spill_mask) - 1;
            uint32_t q = 0;
            if (lane == first) q = atomicAdd(&b.status[kStPoolUsed], (uint32_t)__popc(spill_mask));
            q = __shfl_sync(~0u, q, first);
            if (spill) {
                const uint32_t j = q + __popc(spill_mask & below);
                if (j < b.leaf_pool_cap) {
                    b.leaves[b.leaf_pool_first + j] = held_line;
                    b.pool_path[j] = held_path;
                } else {
                    atomicOr(err, kErrOverflowLeaf);
                }
            }
        }
        held = false;
    };

    // n (1..32) queued lines from the top of the queue, one per lane: a segment's leftmost line
    // goes to the segment's own slot, the others reserve slots (one atomic per path)
    auto emit_round = [&](int n) {
        if constexpr (kMode == kPoolWrite) {
            // exact frame: each segment's lines fill its counted range, slots taken from the
            // segment's counter by one lane per segment among the round's lines
            const bool act = lane < n;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            uint32_t entry = 0;
            if (act) {
                const int k = nleaf - 1 - lane;
                v = W.leaf[k];
                entry = W.leaf_tag[k] & kTagEntry;
            }
            nleaf -= n;
            const unsigned act_mask = __ballot_sync(~0u, act);
            if (act) {
                const unsigned same = __match_any_sync(act_mask, entry);
                const int leader = __ffs(same) - 1;
                uint32_t stored = 0;
                if (lane == leader) {
                    stored = W.seg2[entry].y;
                    W.seg2[entry].y = stored + __popc(same);
                }
                stored = __shfl_sync(act_mask, stored, leader);
                const uint32_t idx = W.seg2[entry].x + stored + __popc(same & below);
                if (idx < b.leaf_cap) b.leaves[idx] = v;
                else atomicOr(err, kErrOverflowLeaf);
            }
            __syncwarp();
            return;
        }
        store_held();
        const bool act = lane < n;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint32_t tag = 0;
        uint4 sg = make_uint4(0u, 0u, 0u, 0u);
        if (act) {
            const int k = nleaf - 1 - lane;
            v = W.leaf[k];
            tag = W.leaf_tag[k];
            sg = W.seg[tag & kTagEntry];
        }
        nleaf -= n;
        produced += act ? 1u : 0u;
        const bool left = act && (tag & kTagLeft);
        if (left) b.leaves[sg.w] = v;
        held = act && !left;
        const unsigned held_mask = __ballot_sync(~0u, held);
        if (held) {
            const unsigned same = __match_any_sync(held_mask, sg.x);
            held_leader = __ffs(same) - 1;
            held_count = __popc(same);
            held_rank = __popc(same & below);
            if (lane == held_leader) held_first = atomicAdd(&b.path_leaf_cursor[sg.x], held_count);
            held_line = v;
            held_path = sg.x;
            held_region = sg.y;
            held_budget = sg.z;
        }
        __syncwarp();
    };
    auto drain = [&]() {
        while (nleaf >= 32) emit_round(32);
    };

    for (;;) {
        drain();
        if (top < 32 && current_group() < n_groups) {
            // a table group that no pending piece or queued line refers to
            uint32_t used = 0;
            for (int k = lane; k < top; k += 32) used |= 1u << ((W.pend_tag[k] & kTagEntry) >> group_shift);
            for (int k = lane; k < nleaf; k += 32) used |= 1u << ((W.leaf_tag[k] & kTagEntry) >> group_shift);
            used = __reduce_or_sync(~0u, used);
            if (used != all_sets) {
                const uint32_t set = __ffs(~used) - 1;
                const uint32_t i = (current_group() << group_shift) + (uint32_t)lane;
                const bool slot = (uint32_t)lane < group, valid = slot && i < n_segs;
                const uint32_t entry = (set << group_shift) + (uint32_t)lane;
                if (kMode == kPoolCount) {
                    if (open >> set & 1u) store_counts(set);
                    open |= 1u << set;
                }
                bool is_leaf = false, is_piece = false;
                float4 ends = make_float4(0.0f, 0.0f, 0.0f, 0.0f), ctrl = ends;
                uint32_t tag = (entry & kTagEntry) | kTagLeft;
                if (valid) {
                    const SegDev sg = b.segs[i];
                    if constexpr (kMode == kPoolLearned) {
                        const uint32_t region = b.path_leaf_first[sg.path];
                        W.seg[entry] = make_uint4(sg.path, region, b.path_leaf_budget[sg.path],
                                                  region + (i - b.path_seg_first[sg.path]));
                    }
                    if constexpr (kMode == kPoolWrite) W.seg2[entry] = make_uint2(b.seg_leaves[i], 0u);
                    const float2 p0 = b.points[sg.a], p1 = b.points[sg.kind == kSegClose ? sg.b : sg.a + 1];
                    ends = make_float4(p0.x, p0.y, p1.x, p1.y);
                    if (sg.kind == kSegQuad) {
                        const float2 p2 = b.points[sg.a + 2];
                        ends = make_float4(p0.x, p0.y, p2.x, p2.y);
                        ctrl = make_float4(p1.x, p1.y, 0.0f, 0.0f);
                    } else if (sg.kind == kSegCubic) {
                        const float2 p2 = b.points[sg.a + 2], p3 = b.points[sg.a + 3];
                        ends = make_float4(p0.x, p0.y, p3.x, p3.y);
                        ctrl = make_float4(p1.x, p1.y, p2.x, p2.y);
                        tag |= kTagCubic;
                    }
                    is_leaf = sg.kind == kSegLine || sg.kind == kSegClose || piece_flat(tag & kTagCubic, ends, ctrl);
                    is_piece = !is_leaf;
                }
                if constexpr (kMode == kPoolCount) {
                    if (slot) W.seg2[entry] = make_uint2(valid ? i : kNone, is_leaf ? 1u : 0u);
                    is_leaf = false;
                }
                const unsigned leaf_mask = __ballot_sync(~0u, is_leaf), piece_mask = __ballot_sync(~0u, is_piece);
                // nleaf < 32 and top < 32 here: the group fits (checked all the same)
                if (is_leaf) {
                    const int k = nleaf + __popc(leaf_mask & below);
                    if (k < kPoolLeafCap) {
                        W.leaf[k] = ends;
                        W.leaf_tag[k] = tag;
                    } else {
                        atomicOr(err, kErrOverflowLeaf);
                    }
                }
                if (is_piece) {
                    const int k = top + __popc(piece_mask & below);
                    if (k < kPoolCap) {
                        W.pend_ends[k] = ends;
                        W.pend_ctrl[k] = ctrl;
                        W.pend_tag[k] = tag;
                    } else {
                        atomicOr(err, kErrOverflowLeaf);
                    }
                }
                nleaf = min(nleaf + __popc(leaf_mask), kPoolLeafCap);
                top = min(top + __popc(piece_mask), kPoolCap);
                __syncwarp();
                if (lane == 0) ticket = atomicAdd(&b.status[kTicket], 1u);
                drain();
            }
        }
        if (top == 0) {
            if (nleaf > 0) emit_round(nleaf);
            if (current_group() >= n_groups) break;
            continue;
        }

        // split round: up to 32 pieces from the top of the pool
        const int n = min(top, 32);
        const bool act = lane < n;
        float4 ends = make_float4(0.0f, 0.0f, 0.0f, 0.0f), ctrl = ends;
        uint32_t tag = 0;
        if (act) {
            const int k = top - 1 - lane;
            ends = W.pend_ends[k];
            ctrl = W.pend_ctrl[k];
            tag = W.pend_tag[k];
        }
        top -= n;
        __syncwarp();
        const bool cubic = (tag & kTagCubic) != 0;
        float4 e0 = ends, c0 = ctrl, e1 = ends, c1 = ctrl;  // first and second halves
        if (cubic) {
            const float p01x = half_lerp(ends.x, ctrl.x), p01y = half_lerp(ends.y, ctrl.y);
            const float p12x = half_lerp(ctrl.x, ctrl.z), p12y = half_lerp(ctrl.y, ctrl.w);
            const float p23x = half_lerp(ctrl.z, ends.z), p23y = half_lerp(ctrl.w, ends.w);
            const float p012x = half_lerp(p01x, p12x), p012y = half_lerp(p01y, p12y);
            const float p123x = half_lerp(p12x, p23x), p123y = half_lerp(p12y, p23y);
            const float mx = half_lerp(p012x, p123x), my = half_lerp(p012y, p123y);
            e0 = make_float4(ends.x, ends.y, mx, my);
            c0 = make_float4(p01x, p01y, p012x, p012y);
            e1 = make_float4(mx, my, ends.z, ends.w);
            c1 = make_float4(p123x, p123y, p23x, p23y);
        } else {
            const float ax = fadd(ends.x, fmul(fsub(ctrl.x, ends.x), 0.5f));
            const float ay = fadd(ends.y, fmul(fsub(ctrl.y, ends.y), 0.5f));
            const float qx = fadd(ctrl.x, fmul(fsub(ends.z, ctrl.x), 0.5f));
            const float qy = fadd(ctrl.y, fmul(fsub(ends.w, ctrl.y), 0.5f));
            const float mx = fadd(ax, fmul(fsub(qx, ax), 0.5f)), my = fadd(ay, fmul(fsub(qy, ay), 0.5f));
            e0 = make_float4(ends.x, ends.y, mx, my);
            c0 = make_float4(ax, ay, 0.0f, 0.0f);
            e1 = make_float4(mx, my, ends.z, ends.w);
            c1 = make_float4(qx, qy, 0.0f, 0.0f);
        }
        const uint32_t depth = ((tag >> kTagDepthShift) & 31u) + 1u;
        const bool deep = depth >= (uint32_t)(kMaxDepth - 1);
        if (act && deep) atomicOr(err, kErrDepth);
        const uint32_t tag0 = (tag & ~(31u << kTagDepthShift)) | depth << kTagDepthShift;
        const uint32_t tag1 = tag0 & ~kTagLeft;
        const bool leaf0 = act && (deep || piece_flat(cubic, e0, c0));
        const bool leaf1 = act && (deep || piece_flat(cubic, e1, c1));
        const unsigned l0 = __ballot_sync(~0u, leaf0), l1 = __ballot_sync(~0u, leaf1);
        if constexpr (kMode == kPoolCount) {
            const uint32_t lines = (leaf0 ? 1u : 0u) + (leaf1 ? 1u : 0u);
            if (lines) atomicAdd(&W.seg2[tag & kTagEntry].y, lines);
        } else {
        // nleaf < 32 before the round, so at most 31 + 64 lines are queued after it (the
        // bounds checks below never fail; a failure would send the frame to the exact redo)
        if (leaf0) {
            const int k = nleaf + __popc(l0 & below);
            if (k < kPoolLeafCap) {
                W.leaf[k] = e0;
                W.leaf_tag[k] = tag0;
            } else {
                atomicOr(err, kErrOverflowLeaf);
            }
        }
        if (leaf1) {
            const int k = nleaf + __popc(l0) + __popc(l1 & below);
            if (k < kPoolLeafCap) {
                W.leaf[k] = e1;
                W.leaf_tag[k] = tag1;
            } else {
                atomicOr(err, kErrOverflowLeaf);
            }
        }
        nleaf = min(nleaf + __popc(l0) + __popc(l1), kPoolLeafCap);
        }
        // halves that are not flat go back on the pool, the second below the first
        const bool keep0 = act && !leaf0, keep1 = act && !leaf1;
        const unsigned m0 = __ballot_sync(~0u, keep0), m1 = __ballot_sync(~0u, keep1);
        const int k1 = top + __popc(m1 & below), k0 = top + __popc(m1) + __popc(m0 & below);
        if (keep1) {
            if (k1 < kPoolCap) {
                W.pend_ends[k1] = e1;
                W.pend_ctrl[k1] = c1;
                W.pend_tag[k1] = tag1;
            }
        }
        if (keep0) {
            if (k0 < kPoolCap) {
                W.pend_ends[k0] = e0;
                W.pend_ctrl[k0] = c0;
                W.pend_tag[k0] = tag0;
            }
        }
        top = min(top + __popc(m0) + __popc(m1), kPoolCap);
        if ((keep1 && k1 >= kPoolCap) || (keep0 && k0 >= kPoolCap)) {
            if constexpr (kMode == kPoolCount) {
                if (keep1 && k1 >= kPoolCap)
                    atomicAdd(&W.seg2[tag1 & kTagEntry].y, count_piece_alone(b.status, e1, c1, tag1));
                if (keep0 && k0 >= kPoolCap)
                    atomicAdd(&W.seg2[tag0 & kTagEntry].y, count_piece_alone(b.status, e0, c0, tag0));
            } else if constexpr (kMode == kPoolWrite) {
                if (keep1 && k1 >= kPoolCap) {
                    uint2 &sg = W.seg2[tag1 & kTagEntry];
                    flatten_piece_alone_exact(b.leaves, b.leaf_cap, b.status, &sg.y, sg.x, e1, c1, tag1);
                }
                if (keep0 && k0 >= kPoolCap) {
                    uint2 &sg = W.seg2[tag0 & kTagEntry];
                    flatten_piece_alone_exact(b.leaves, b.leaf_cap, b.status, &sg.y, sg.x, e0, c0, tag0);
                }
            } else {
                const LeafSink out{b.leaves, b.path_leaf_cursor, b.status, b.pool_path, b.leaf_pool_first,
                                   b.leaf_pool_cap};
                if (keep1 && k1 >= kPoolCap)
                    produced += flatten_piece_alone(out, W.seg[tag1 & kTagEntry], e1, c1, tag1);
                if (keep0 && k0 >= kPoolCap)
                    produced += flatten_piece_alone(out, W.seg[tag0 & kTagEntry], e0, c0, tag0);
            }
        }
        __syncwarp();
    }
    if constexpr (kMode == kPoolCount) {
        for (uint32_t set = 0; set < n_sets; set++)
            if (open >> set & 1u) store_counts(set);
    }
    if constexpr (kMode == kPoolLearned) {
        store_held();
        const uint32_t total = __reduce_add_sync(~0u, produced);
        if (lane == 0) atomicAdd(&b.status[kStLeafCount], total);
    }
}

// ---------------------------------------------------------------------------
// Binning by path (the d3d9 Tiler::process_line_segment walk and Tiler::prepare_tiles,
// tiler.cpp:131-279 / 369-439, which the reference's GPU frame runs as bin.comp and
// propagate.comp).  A path's tiles belong to it alone, so one CTA bins all of a path's leaf
// lines in shared memory: it counts fills and backdrop deltas per tile, propagates the
// backdrops down each column, scans the counts into fill offsets (reserving the path's block
// of fills with one atomic), and walks the lines again to write the fills grouped by tile.
// No tile needs clearing, there is no frame-wide scan over tiles and no global atomic per
// fill.  Paths too large for a CTA (class 3) take global passes: counts with atomics, a CTA
// per path for backdrops and offsets, then the writes with atomics.

// Size classes by shared-memory words: one per tile (fill count in bits 0-23, the int8 sum of
// backdrop deltas in bits 24-31, later the tile's write cursor) and one per column (deltas
// landing above the rect, summed as int32).
constexpr int kCtaClasses = 3;
// Small CTAs for the small classes: a path's barriers then hold few warps, and more paths are in
// flight per SM (A/B on the 512-scene batch, binning: 21.56 ms with 256-thread CTAs, 6 per SM, for
// classes 0 and 1; 20.80 ms with 128-thread CTAs, 12 per SM; 20.72 ms with class 0 at 64 threads,
// 24 per SM).  Class 2 keeps 384 threads: its shared words allow 3 CTAs per SM (256 or 512 threads
// ran slower).
// a class's words, and up to 3 before the tiles and 3 after them
__host__ __device__ constexpr size_t class_smem(int c) { return (size_t(class_words(c)) + 8) * 4; }
__host__ __device__ constexpr int class_threads(int c) { return c == 2 ? 384 : c == 1 ? 128 : 64; }
// CTAs per SM the register budget is set for (shared memory allows 3 of class 2, 12 of class 1).
// Binning of 256 scenes / 20,000 paths: class 0 at 16, 18, 20 and 22 CTAs 7.63 / 0.696, 7.61 / 0.706, 7.64
// / 0.718 and 8.13 / 0.868 ms (more CTAs leave too few registers and spill); class 1 at 7, 8, 9 and 10
// 7.70, 7.64, 7.64 and 7.75 ms.
__host__ __device__ constexpr int class_min_ctas(int c) { return c == 2 ? 3 : c == 1 ? 8 : 18; }
// Tile visits with fills a CTA stages during its count walk (12 bytes each, in its own slice of a
// global buffer that stays in L2, an equal part for each of its warps): the fills are then placed
// without walking the lines again.  A path with more than this walks its lines twice.
__host__ __device__ constexpr uint32_t class_stage(int c) { return c == 0 ? 3072u : c == 1 ? 6144u : 12288u; }
// One line gives a tile at most two fills (the walk visits a tile once, with at most one
// extra fill for a vertical crossing), so with at most 2^22 lines per CTA-binned path the
// 24-bit counters cannot carry into the delta byte (kCtaMaxLeaves).
// bin_ctl slots: paths per list (the CTA classes, the small one, the cluster one), work tickets of the
// CTA classes and of the cluster one, tickets of the class-3 zeroing and set-up passes, and at slot
// 12 a 64-bit word: class-3 paths << 40 | their lines.
enum : int { kCtlCount = 0, kCtlTicket = 5, kCtlTicketCluster = 8, kCtlTicketZero = 9, kCtlTicketPrep = 10, kCtl3 = 12 };
// and from slot 16 the lists' paths counted by log2 of their leaf lines (5 x 32), then the write
// cursors of those buckets (5 x 32): each list runs from its largest paths to its smallest, so the
// last to start take the shortest paths
constexpr int kListSmall = kCtaClasses, kListCluster = kCtaClasses + 1, kLists = kCtaClasses + 2;
enum : int {
    kCtlBucket = 16,
    kCtlCursor = 16 + kLists * 32,
    kCtlWords = 16 + 2 * kLists * 32,
    kCtlCompTicket = kCtlWords
};
static_assert((kCtlCompTicket + 1) * 4 <= kBinCtlBytes, "bin_ctl is too small");
// The list of a class (-1: none, class 3 has its own); lists 3 and 4 lie behind class 3's two rows.
__device__ __forceinline__ int class_list(int cls) {
    return cls == kSmallClass ? kListSmall : cls == kClusterClass ? kListCluster : cls < kCtaClasses ? cls : -1;
}
__device__ __forceinline__ uint32_t *list_row(const Batch &b, int list) {
    return b.bin_list + (size_t)(list < kCtaClasses ? list : list + 2) * b.n_paths;
}
constexpr uint64_t kLow40 = (1ull << 40) - 1;

constexpr uint32_t kSmallLines = 384;  // most lines of a path that a warp bins

__device__ __forceinline__ unsigned long long *ctl3_word(const Batch &b) {
    return reinterpret_cast<unsigned long long *>(b.bin_ctl + kCtl3);
}
__device__ __forceinline__ unsigned long long *fill_total(const Batch &b) {
    return reinterpret_cast<unsigned long long *>(b.status + kStFill64);
}

// -1: no columns (nothing can land); kSmallClass: a warp; 0-2: CTA classes; kClusterClass: a cluster
// of CTAs; 3: global passes.  A
// class holds the path's words; a larger one is taken where the smaller one's warps would have to
// walk more than warp_lines lines each (bin_warp_lines), and a warp takes no more than it can stage.
__device__ __forceinline__ int path_class(const PathDev &P, uint32_t leaves, uint32_t warp_lines) {
    const int32_t rw = max(P.rx1 - P.rx0, 0), rh = max(P.ry1 - P.ry0, 0);
    if (rw == 0) return -1;
    if (leaves > kCtaMaxLeaves) return 3;
    int c = rect_class((uint32_t)rw, (uint32_t)rh);
    if (c == kSmallClass && leaves > min(warp_lines, kSmallLines)) c = 0;
    if (c == 0 && leaves > class_threads(0) / 32 * warp_lines) c = 1;
    if (c == 1 && leaves > class_threads(1) / 32 * warp_lines) c = 2;
    return c;
}

// The lines a warp would get if the frame's were spread evenly over the binning warps the GPU holds
// (36 per SM), at least 64 (two rounds).  A path of far more lines for its size than that - a
// dashed outline, or any path of a frame too small to fill the GPU - is the frame's critical path,
// so it gets a CTA of more warps.
__device__ __forceinline__ uint32_t bin_warp_lines(const Batch &b, bool learned) {
    return max(64u, b.status[learned ? kStLeafCount : kStLeaves] / (36u * b.n_sms));
}

// The leaf lines of one path: its region of the leaf buffer, then (learned frame) its lines
// in the spill pool, listed by k_pool_scatter.
struct PathLeaves {
    uint32_t first, nreg, pool0, n;
    __device__ __forceinline__ uint32_t index(const Batch &b, uint32_t k) const {
        return k < nreg ? first + k : b.leaf_pool_first + b.pool_idx[pool0 + (k - nreg)];
    }
};

__device__ __forceinline__ PathLeaves path_leaves(const Batch &b, uint32_t p) {
    const uint2 r = b.path_leaf_range[p];
    PathLeaves L{r.x, r.y - r.x, 0u, r.y - r.x};
    if (b.pool_cnt) {
        L.pool0 = b.pool_cnt[(int64_t)p - 1];
        L.n += b.pool_cnt[p] - L.pool0;
    }
    return L;
}

// Lines a warp of a CTA (or cluster) of `warps` takes at a time: 32, one a lane, or fewer where they are
// long.  A closed outline crosses its rect there and back, so its n lines span at least 2 (rw + rh) / n
// tiles on average; past long_line the warp walks its lines one after the other, and so many lines fill
// its part of the stage.  They are then dealt out evenly.  (Binning of 2,000 paths of 40 points, about
// 375 x 375 tiles each: 8.75 ms by groups of 32, 4.80 so; 300 quadrilaterals on 8,192 px 3.61 and 3.09.)
__device__ __forceinline__ uint32_t line_group(const Batch &b, uint32_t rw, uint32_t rh, uint32_t n, uint32_t warps) {
    const bool spread = (float)(2u * (rw + rh)) > b.long_line * (float)n;
    return spread ? min(32u, max(1u, (n + warps - 1u) / warps)) : 32u;
}

// Whether a walk of this frame hit its bound (the frame then ends with that error).  The lane form walks
// such a line through other tiles than walk_line, so its counts are not to be filled by a second walk,
// nor the fills read.  Past a barrier, a block sees what its own walks have found.  The CTA classes ask
// while the block of fills is being reserved (20,000 paths 1,432.9 us without, 1,430.3 so; asked at the
// second walk instead, 1.7% more, as its code then changes the kernel's), a warp only before its second
// walk (150,000 glyphs 986 and 989 us; asked by every path, 1,130).
__device__ __forceinline__ bool walk_failed(const uint32_t *status) {
    return (*(const volatile uint32_t *)status & kErrWalk) != 0;
}

__device__ __forceinline__ WalkCtx walk_ctx(const Batch &b, const PathDev &P) {
    const SceneDev &S = b.scenes[P.scene];
    WalkCtx w;
    w.rx0 = P.rx0;
    w.ry0 = P.ry0;
    w.rx1 = P.rx1;
    w.ry1 = P.ry1;
    w.rw = max(P.rx1 - P.rx0, 0);
    w.rh = max(P.ry1 - P.ry0, 0);
    w.vb_left = S.vb_left;
    w.vb_right = S.vb_right;
    w.vb_bottom = S.vb_bottom;
    return w;
}

// Adds an int8 delta to the low byte of a 16-bit tile state (class-3 count pass; the high
// byte is still zero).  A compare-and-swap on the enclosing word: every failed round means
// another thread's update went in, and the loop is bounded all the same.
__device__ __forceinline__ void add_delta_u16(uint16_t *a, int d, uint32_t *status) {
    uint32_t *word = reinterpret_cast<uint32_t *>(reinterpret_cast<uintptr_t>(a) & ~uintptr_t(3));
    const int sh = (reinterpret_cast<uintptr_t>(a) & 2) ? 16 : 0;
    uint32_t old = *word;
    for (int it = 0; it < (1 << 20); it++) {
        const uint32_t byte = ((old >> sh) + (uint32_t)d) & 0xffu;
        const uint32_t want = (old & ~(0xffu << sh)) | (byte << sh);
        const uint32_t seen = atomicCAS(word, old, want);
        if (seen == old) return;
        old = seen;
    }
    atomicOr(status, kErrWalk);
}

// The paths' leaf ranges, size classes and lists.  A listed path's key is its list and the log2 of
// its leaf lines; the lists are filled bucket by bucket, largest first, from the buckets' counts.
// Class-3 paths take a 64-bit atomic that also hands out their offsets in the class-3 line
// numbering the global passes stride over.
__device__ __forceinline__ uint32_t path_lines(const Batch &b, uint32_t p, uint2 range) {
    uint32_t n = range.y - range.x;
    if (b.pool_cnt) n += b.pool_cnt[p] - b.pool_cnt[(int64_t)p - 1];
    return n;
}

// Classifies path p; its key, or -1 when it is on no list.
__device__ __forceinline__ int bin_classify(const Batch &b, uint32_t p, bool learned, uint32_t warp_lines) {
    const PathDev P = b.paths[p];
    uint2 range;
    if (learned) {
        const uint32_t f = b.path_leaf_first[p];
        range = make_uint2(f, f + min(b.path_leaf_cursor[p], b.path_leaf_budget[p]));
    } else {
        const uint2 pc = b.path_contours[p];
        range = make_uint2(b.seg_leaves[b.contour_segs[pc.x]], b.seg_leaves[b.contour_segs[pc.y]]);
    }
    b.path_leaf_range[p] = range;
    const uint32_t n = path_lines(b, p, range);
    const int cls = path_class(P, n, warp_lines), list = class_list(cls);
    b.path_cls[p] = (uint8_t)cls;
    if (cls < 0) b.path_fill[p] = 0;
    if (cls == 3) {
        const unsigned long long old = atomicAdd(ctl3_word(b), (1ull << 40) | (unsigned long long)n);
        const uint32_t item = (uint32_t)(old >> 40);
        b.bin_list[(size_t)3 * b.n_paths + item] = p;
        b.bin_list[(size_t)4 * b.n_paths + item] = (uint32_t)(old & kLow40);
    }
    return list >= 0 ? list * 32 + (31 - __clz(max(n, 1u))) : -1;
}

// One warp per list: the buckets' first slots, largest lines first, into start[]; lane 31 returns
// the list's length.
__device__ __forceinline__ uint32_t bucket_starts(const uint32_t *count, uint32_t *start, int list, int lane) {
    const uint32_t v = count[list * 32 + 31 - lane];
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    start[list * 32 + 31 - lane] = incl - v;
    return incl;
}

__device__ __forceinline__ void copy_status(const Batch &b, const StatusCopy &copy) {
    for (uint32_t i = threadIdx.x; i < kStHostWords; i += blockDim.x)
        copy.host[i] = *(const volatile uint32_t *)(b.status + i);
}

// A frame of many paths: a pass that classifies and counts, and one that places.
__global__ void __launch_bounds__(kThreads) k_bin_classify(Batch b, bool learned) {
    __shared__ uint32_t s_bucket[kLists * 32];
    if (threadIdx.x < kLists * 32) s_bucket[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t p = global_tid();
    const int key = p < b.n_paths ? bin_classify(b, p, learned, bin_warp_lines(b, learned)) : -1;
    if (key >= 0) atomicAdd(&s_bucket[key], 1u);
    __syncthreads();
    if (threadIdx.x < kLists * 32 && s_bucket[threadIdx.x])
        atomicAdd(&b.bin_ctl[kCtlBucket + threadIdx.x], s_bucket[threadIdx.x]);
}

__global__ void __launch_bounds__(kThreads) k_bin_scatter(Batch b, StatusCopy copy) {
    __shared__ uint32_t s_start[kLists * 32];
    __shared__ bool s_last;
    const uint32_t p = global_tid();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < kLists) {
        const uint32_t n = bucket_starts(b.bin_ctl + kCtlBucket, s_start, warp, lane);
        if (blockIdx.x == 0 && lane == 31) b.bin_ctl[kCtlCount + warp] = n;
    }
    int key = -1;
    if (p < b.n_paths) {
        const int list = class_list((int)(int8_t)b.path_cls[p]);
        if (list >= 0) key = list * 32 + (31 - __clz(max(path_lines(b, p, b.path_leaf_range[p]), 1u)));
    }
    const unsigned g = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(g) - 1;
    uint32_t base = 0;
    if (key >= 0 && lane == leader) base = atomicAdd(&b.bin_ctl[kCtlCursor + key], (uint32_t)__popc(g));
    base = __shfl_sync(0xffffffffu, base, leader);
    __syncthreads();
    if (key >= 0) list_row(b, key >> 5)[s_start[key] + base + __popc(g & ((1u << lane) - 1u))] = p;
    if (!copy.host) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(copy.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        copy_status(b, copy);
    }
}

// A frame of few paths: both in one block (of up to kOneBlockPaths; 3,000 paths took 12 us in three
// launches).
constexpr uint32_t kOneBlockPaths = 4096;
constexpr int kOneBlockThreads = 1024;

__global__ void __launch_bounds__(kOneBlockThreads) k_bin_lists(Batch b, bool learned, StatusCopy copy) {
    __shared__ uint32_t s_bucket[kLists * 32], s_start[kLists * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < kLists * 32) s_bucket[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t warp_lines = bin_warp_lines(b, learned);
    int key[kOneBlockPaths / kOneBlockThreads];
#pragma unroll
    for (int k = 0; k < (int)(kOneBlockPaths / kOneBlockThreads); k++) {
        const uint32_t p = k * kOneBlockThreads + threadIdx.x;
        key[k] = p < b.n_paths ? bin_classify(b, p, learned, warp_lines) : -1;
        if (key[k] >= 0) atomicAdd(&s_bucket[key[k]], 1u);
    }
    __syncthreads();
    if (warp < kLists) {
        const uint32_t n = bucket_starts(s_bucket, s_start, warp, lane);
        if (lane == 31) b.bin_ctl[kCtlCount + warp] = n;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < (int)(kOneBlockPaths / kOneBlockThreads); k++)
        if (key[k] >= 0) list_row(b, key[k] >> 5)[atomicAdd(&s_start[key[k]], 1u)] = k * kOneBlockThreads + threadIdx.x;
    if (!copy.host) return;
    __threadfence_block();
    __syncthreads();
    copy_status(b, copy);
}

// The fills of one tile visit, as a binning warp stages them: the visit's points and a word with
// the tile (below 2^16) and which fills are kept - the tile's fill, the vertical crossing's extra
// one, and whether that runs from the tile's corner (going down) or to it.
constexpr uint32_t kVisitFill = 1u << 16, kVisitExtra = 1u << 17, kVisitDown = 1u << 18;

template <int kCls>
__global__ void __launch_bounds__(class_threads(kCls), class_min_ctas(kCls)) k_bin_fused(Batch b) {
    constexpr int kThr = class_threads(kCls), kWarps = kThr / 32;
    constexpr uint32_t kStage = class_stage(kCls) / kWarps;  // fills a warp stages
    static_assert(class_words(kCls) <= 65536u, "a staged fill holds its tile in 16 bits");
    extern __shared__ __align__(16) uint32_t sm[];
    __shared__ uint32_t s_item, s_base, s_write, s_next, s_over;
    __shared__ uint32_t s_slot[kWarps];
    __shared__ int32_t s_seg[kThr];
    __shared__ uint32_t s_warp[kWarps];
    __shared__ unsigned long long s_wsum[kWarps];
    const uint32_t tid = threadIdx.x;
    const int lane = (int)(tid & 31), warp = (int)(tid >> 5);
    const unsigned below = (1u << lane) - 1u;
    uint2 *const stage = b.stage + ((size_t)blockIdx.x * kWarps + warp) * kStage;
    uint32_t *const stage_tile = b.stage_tile + ((size_t)blockIdx.x * kWarps + warp) * kStage;
    const uint32_t *list = b.bin_list + (size_t)kCls * b.n_paths;
    const uint32_t n_items = b.bin_ctl[kCtlCount + kCls];
    uint32_t *const err = &b.status[kStErr];
    for (;;) {
        if (tid == 0) s_item = atomicAdd(&b.bin_ctl[kCtlTicket + kCls], 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= n_items) return;
        const uint32_t p = list[item];
        const PathDev P = b.paths[p];
        const WalkCtx w = walk_ctx(b, P);
        const uint32_t rw = (uint32_t)w.rw, rh = (uint32_t)w.rh, T = rw * rh, tb = P.tile_first, cb = P.col_first;
        // the tiles start as many words into the array as their records in global memory lie past a
        // multiple of four, so that the passes over them take 16 bytes at a time on both sides; the
        // words before and after them stay zero
        const uint32_t pad = tb & 3u, end4 = (pad + T + 3u) & ~3u;
        uint32_t *cnt = sm + pad;                                 // per tile: count | delta << 24, then cursor
        int32_t *above = reinterpret_cast<int32_t *>(sm + end4);  // per column
        const PathLeaves L = path_leaves(b, p);
        for (uint32_t t = 4 * tid; t < end4 + rw; t += 4 * kThr)
            *reinterpret_cast<uint4 *>(&sm[t]) = make_uint4(0u, 0u, 0u, 0u);
        if (tid == 0) {
            s_next = 0;
            s_over = 0;
        }
        __syncthreads();

        // 1. fill counts and backdrop deltas, the fills staged with their tiles.  Warps take
        //    the lines a group at a time, so a warp that drew short lines takes more.
        //    A line of many tiles (a contour's closing line spans the canvas) would hold its
        //    warp, and at the barrier its CTA, for tens of steps: such lines are walked by the
        //    whole warp after its short lines.
        uint32_t nstage = 0;  // visits this warp staged (the same in every lane)
        auto on_fill = [&](int32_t local, uint2 q) {
            atomicAdd(&cnt[local], 1u);
            const uint32_t slot = atomicAdd(&s_slot[warp], 1u);
            if (slot < kStage) {
                stage[slot] = q;
                stage_tile[slot] = (uint32_t)local | kVisitFill;
            }
        };
        auto on_delta = [&](int32_t where, int d) {
            if (where >= 0) atomicAdd(&cnt[where], (uint32_t)d << 24);
            else atomicAdd(&above[-1 - where], d);
        };
        auto on_above = [&](int32_t x, int d) { atomicAdd(&above[x], d); };
        auto begin_single = [&]() {
            if (lane == 0) s_slot[warp] = nstage;
            __syncwarp();
        };
        auto end_single = [&]() {
            __syncwarp();
            nstage = s_slot[warp];
        };
        // a step of the warp's lines: one atomic per lane for its tile, one stage slot per lane
        // with a fill
        auto visit = [&](bool live, bool m, bool e, uint32_t pa, uint32_t pb, bool down, uint32_t local,
                         uint32_t inc) {
            const unsigned keep = __ballot_sync(0xffffffffu, live && (m || e));
            if (live && inc) atomicAdd(&cnt[local], inc);
            const uint32_t slot = nstage + __popc(keep & below);
            if ((keep >> lane & 1u) && slot < kStage) {
                stage[slot] = make_uint2(pa, pb);
                stage_tile[slot] = local | (m ? kVisitFill : 0u) | (e ? kVisitExtra : 0u) | (down ? kVisitDown : 0u);
            }
            nstage += __popc(keep);
        };
        const uint32_t group = line_group(b, rw, rh, L.n, kWarps);
        for (;;) {
            uint32_t k0 = 0;
            if (lane == 0) k0 = atomicAdd(&s_next, group);
            k0 = __shfl_sync(0xffffffffu, k0, 0);
            if (k0 >= L.n) break;
            const uint32_t k = k0 + (uint32_t)lane;
            const bool have = (uint32_t)lane < group && k < L.n;
            const float4 f = have ? b.leaves[L.index(b, k)] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            walk_lines(w, f, have, b.long_line, visit, on_above, on_fill, on_delta, begin_single, end_single, err);
        }
        if (lane == 0 && nstage > kStage) s_over = 1;
        __syncthreads();

        // 2. the count of each warp's chunk of tiles; thread 0 reserves the path's block of
        //    fills with one atomic whose result it reads only after the column pass
        const uint32_t chunk = ((end4 + kWarps - 1) / kWarps + 127u) & ~127u;
        const uint32_t c0 = min(end4, (uint32_t)warp * chunk), c1 = min(end4, c0 + chunk);
        uint32_t lsum = 0;  // under 2^8 tiles a lane
        for (uint32_t t = c0 + 4 * lane; t < c1; t += 128) {
            const uint4 q = *reinterpret_cast<const uint4 *>(&sm[t]);
            lsum += (q.x & 0xffffffu) + (q.y & 0xffffffu) + (q.z & 0xffffffu) + (q.w & 0xffffffu);
        }
        unsigned long long wsum = lsum;  // 64-bit: a path's fills need not fit 32 bits (it then overflows)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wsum += __shfl_down_sync(0xffffffffu, wsum, o);
        if (lane == 0) s_wsum[warp] = wsum;
        __syncthreads();
        unsigned long long base = 0, total = 0;
        bool failed = false;
        if (tid == 0) {
            failed = walk_failed(err);  // in flight with the atomic
            for (int k = 0; k < kWarps; k++) {
                const unsigned long long v = s_wsum[k];
                s_warp[k] = (uint32_t)total;
                total += v;
            }
            base = atomicAdd(fill_total(b), total);
        }

        // 3. backdrops down each column (tile backdrop = int8 of the running column sum before
        //    the tile's own delta); columns are cut into segments of rows so every thread has
        //    work: segment sums first, then each segment's walk from its starting sum.
        const uint32_t segs = rw >= (uint32_t)kThr ? 1u : (uint32_t)kThr / rw;
        const uint32_t seg_rows = (rh + segs - 1) / segs;
        if (segs > 1) {
            if (tid < rw * segs) {
                const uint32_t x = tid % rw, s = tid / rw;
                const uint32_t y0 = min(rh, s * seg_rows), y1 = min(rh, y0 + seg_rows);
                int32_t sum = 0;
                for (uint32_t y = y0; y < y1; y++) sum += (int8_t)(cnt[y * rw + x] >> 24);
                s_seg[tid] = sum;
            }
            __syncthreads();
        }
        for (uint32_t u = tid; u < rw * segs; u += kThr) {
            const uint32_t x = u % rw, s = u / rw;
            int32_t run = above[x];
            for (uint32_t k = 0; k < s; k++) run += s_seg[k * rw + x];
            const uint32_t y0 = min(rh, s * seg_rows), y1 = min(rh, y0 + seg_rows);
            for (uint32_t y = y0; y < y1; y++) {
                const uint32_t t = y * rw + x, c = cnt[t];
                b.tile_state[tb + t] = (uint16_t)((uint32_t)(uint8_t)(int8_t)run | ((c & 0xffffffu) ? 0x100u : 0u));
                run += (int8_t)(c >> 24);
            }
            if (s == segs - 1) b.col_final[cb + x] = run;
        }
        if (tid == 0) {
            const bool fits = base + total <= (unsigned long long)b.fill_cap;
            if (!fits) atomicOr(err, kErrOverflowFill);
            b.path_fill[p] = (uint32_t)base;
            s_base = (uint32_t)base;
            s_write = fits && total > 0 && !failed;
        }
        __syncthreads();

        // 4. each warp scans its chunk into write cursors (shared) and end offsets (global): a
        //    lane takes four consecutive tiles (16 bytes of both), and one warp scan covers 128.
        //    With the passes over the tiles (zeros, counts, offsets) 16 bytes wide on both sides
        //    binning takes 7.64 ms instead of 7.93 on 256 scenes, whose large rects have more
        //    tiles than fills
        uint32_t carry = s_base + s_warp[warp];
        for (uint32_t t0 = c0; t0 < c1; t0 += 128) {
            const uint32_t t = t0 + 4 * (uint32_t)lane;
            const bool in = t < c1;
            const uint4 q = in ? *reinterpret_cast<const uint4 *>(&sm[t]) : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t v[4] = {q.x & 0xffffffu, q.y & 0xffffffu, q.z & 0xffffffu, q.w & 0xffffffu};
            const uint32_t own = v[0] + v[1] + v[2] + v[3];
            uint32_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += n;
            }
            uint32_t e[5];
            e[0] = carry + incl - own;
#pragma unroll
            for (int j = 0; j < 4; j++) e[j + 1] = e[j] + v[j];
            if (in) {
                *reinterpret_cast<uint4 *>(&sm[t]) = make_uint4(e[0], e[1], e[2], e[3]);
                uint32_t *const fills = b.tile_fills + (tb - pad) + t;
                if (t >= pad && t + 4 <= pad + T) {
                    *reinterpret_cast<uint4 *>(fills) = make_uint4(e[1], e[2], e[3], e[4]);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (t + j >= pad && t + j < pad + T) fills[j] = e[j + 1];
                }
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();

        // 5. the fills, grouped by tile: each warp's from its stage (four loads in flight per
        //    lane), or, when a warp's stage was too small, by walking the lines again
        if (s_write && !s_over) {
            auto place = [&](uint2 v, uint32_t t) {
                const uint32_t m = t >> 16 & 1u, e = t >> 17 & 1u;
                const uint32_t at = atomicAdd(&cnt[t & 0xffffu], m + e);
                if (m) b.fills[at] = v;
                if (e) b.fills[at + m] = t & kVisitDown ? make_uint2(0u, v.x) : make_uint2(v.y, 0u);
            };
            uint32_t k = lane;
            for (; k + 96 < nstage; k += 128) {
                uint2 v[4];
                uint32_t t[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    v[j] = stage[k + j * 32];
                    t[j] = stage_tile[k + j * 32];
                }
#pragma unroll
                for (int j = 0; j < 4; j++) place(v[j], t[j]);
            }
            for (; k < nstage; k += 32) place(stage[k], stage_tile[k]);
        } else if (s_write) {
            for (uint32_t k = tid; k < L.n; k += kThr) {
                const float4 f = b.leaves[L.index(b, k)];
                walk_line(
                    w, f.x, f.y, f.z, f.w,
                    [&](int32_t local, uint2 q) { b.fills[atomicAdd(&cnt[local], 1u)] = q; },
                    [&](int32_t, int) {}, err);
            }
        }
        __syncthreads();
    }
}

// The small class: one warp bins a path, as k_bin_fused does with a CTA.  A glyph's path has some 60
// lines and 10 tiles; a CTA spends most of its time on it in barriers and in waiting for the path's
// record, while warps on paths of their own have no barriers and wait side by side.  Visits are
// staged in shared memory (the rest, if any, in the warp's slice of the global stage).  Binning
// 150,000 glyphs 0.47 -> 0.34 ms, 20,000 paths (half of them small) 0.73 -> 0.69 ms; 8 CTAs
// per SM leave 64 registers, and 68 bytes of spills; 10 (48 registers, more spills) take 0.37 ms, the next
// path's record loaded ahead 0.35 ms.
constexpr int kSmallThreads = 128, kSmallWarps = kSmallThreads / 32;
constexpr uint32_t kSmallStage = 160, kSmallSpill = 640;  // visits staged per warp: shared, then global

__global__ void __launch_bounds__(kSmallThreads, 8) k_bin_small(Batch b) {
    __shared__ __align__(16) uint32_t s_cnt[kSmallWarps][kSmallWords];
    __shared__ uint2 s_pts[kSmallWarps][kSmallStage];
    __shared__ uint32_t s_tile[kSmallWarps][kSmallStage], s_slot[kSmallWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    uint32_t *const cnt = s_cnt[warp], *const err = &b.status[kStErr];
    const uint32_t first = blockIdx.x * kSmallWarps + warp, stride = gridDim.x * kSmallWarps;
    uint2 *const spill = b.stage + (size_t)first * kSmallSpill;
    uint32_t *const spill_tile = b.stage_tile + (size_t)first * kSmallSpill;
    const uint32_t *list = list_row(b, kListSmall);
    const uint32_t n_items = b.bin_ctl[kCtlCount + kListSmall];
    uint32_t item = first;
    if (item >= n_items) return;
    uint32_t next_p = list[item];
    for (;;) {
        const uint32_t p = next_p;
        if (item + stride < n_items) next_p = list[item + stride];
        const PathDev P = b.paths[p];
        const PathLeaves L = path_leaves(b, p);
        const WalkCtx w = walk_ctx(b, P);
        const uint32_t rw = (uint32_t)w.rw, rh = (uint32_t)w.rh, T = rw * rh, tb = P.tile_first, cb = P.col_first;
        int32_t *const above = reinterpret_cast<int32_t *>(cnt + T);
        for (uint32_t t = lane; t < T + rw; t += 32) cnt[t] = 0;
        __syncwarp();

        // 1. fill counts and backdrop deltas, the visits staged
        uint32_t nstage = 0;
        auto stage = [&](uint32_t slot, uint2 pts, uint32_t tile) {
            if (slot < kSmallStage) {
                s_pts[warp][slot] = pts;
                s_tile[warp][slot] = tile;
            } else if (slot < kSmallStage + kSmallSpill) {
                spill[slot - kSmallStage] = pts;
                spill_tile[slot - kSmallStage] = tile;
            }
        };
        auto on_fill = [&](int32_t local, uint2 q) {
            atomicAdd(&cnt[local], 1u);
            stage(atomicAdd(&s_slot[warp], 1u), q, (uint32_t)local | kVisitFill);
        };
        auto on_delta = [&](int32_t where, int d) {
            if (where >= 0) atomicAdd(&cnt[where], (uint32_t)d << 24);
            else atomicAdd(&above[-1 - where], d);
        };
        auto on_above = [&](int32_t x, int d) { atomicAdd(&above[x], d); };
        auto begin_single = [&]() {
            if (lane == 0) s_slot[warp] = nstage;
            __syncwarp();
        };
        auto end_single = [&]() {
            __syncwarp();
            nstage = s_slot[warp];
        };
        auto visit = [&](bool live, bool m, bool e, uint32_t pa, uint32_t pb, bool down, uint32_t local,
                         uint32_t inc) {
            const unsigned keep = __ballot_sync(0xffffffffu, live && (m || e));
            if (live && inc) atomicAdd(&cnt[local], inc);
            if (keep >> lane & 1u)
                stage(nstage + __popc(keep & below), make_uint2(pa, pb),
                      local | (m ? kVisitFill : 0u) | (e ? kVisitExtra : 0u) | (down ? kVisitDown : 0u));
            nstage += __popc(keep);
        };
        for (uint32_t k0 = 0; k0 < L.n; k0 += 32) {
            const uint32_t k = k0 + (uint32_t)lane;
            const bool have = k < L.n;
            const float4 f = have ? b.leaves[L.index(b, k)] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            walk_lines(w, f, have, b.long_line, visit, on_above, on_fill, on_delta, begin_single, end_single, err);
        }
        __syncwarp();

        // 2. the path's block of fills: four consecutive tiles a lane
        uint32_t v[4], own = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = 4u * lane + j < T ? cnt[4 * lane + j] & 0xffffffu : 0u;
            own += v[j];
        }
        uint32_t incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(fill_total(b), (unsigned long long)total);

        // 3. backdrops down each column
        for (uint32_t x = lane; x < rw; x += 32) {
            int32_t run = above[x];
            for (uint32_t y = 0; y < rh; y++) {
                const uint32_t t = y * rw + x, c = cnt[t];
                b.tile_state[tb + t] = (uint16_t)((uint32_t)(uint8_t)(int8_t)run | ((c & 0xffffffu) ? 0x100u : 0u));
                run += (int8_t)(c >> 24);
            }
            b.col_final[cb + x] = run;
        }
        __syncwarp();

        // 4. write cursors (shared) and end offsets (global)
        base = __shfl_sync(0xffffffffu, base, 0);
        const bool fits = base + total <= (unsigned long long)b.fill_cap;
        if (lane == 0) {
            if (!fits) atomicOr(err, kErrOverflowFill);
            b.path_fill[p] = (uint32_t)base;
        }
        uint32_t at = (uint32_t)base + incl - own;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t t = 4 * lane + j;
            if (t < T) {
                cnt[t] = at;
                b.tile_fills[tb + t] = at + v[j];
            }
            at += v[j];
        }
        __syncwarp();

        // 5. the fills, grouped by tile
        if (fits && nstage <= kSmallStage + kSmallSpill) {
            for (uint32_t k = lane; k < nstage; k += 32) {
                const bool here = k < kSmallStage;
                const uint2 q = here ? s_pts[warp][k] : spill[k - kSmallStage];
                const uint32_t t = here ? s_tile[warp][k] : spill_tile[k - kSmallStage];
                const uint32_t m = t >> 16 & 1u, e = t >> 17 & 1u;
                const uint32_t slot = atomicAdd(&cnt[t & 0xffffu], m + e);
                if (m) b.fills[slot] = q;
                if (e) b.fills[slot + m] = t & kVisitDown ? make_uint2(0u, q.x) : make_uint2(q.y, 0u);
            }
        } else if (fits && !walk_failed(err)) {
            for (uint32_t k = lane; k < L.n; k += 32) {
                const float4 f = b.leaves[L.index(b, k)];
                walk_line(
                    w, f.x, f.y, f.z, f.w,
                    [&](int32_t local, uint2 q) { b.fills[atomicAdd(&cnt[local], 1u)] = q; },
                    [&](int32_t, int) {}, err);
            }
        }
        __syncwarp();
        if ((item += stride) >= n_items) return;
    }
}

// The cluster class: rects too large for one CTA's shared memory (beyond 2048 x 2048 px or so) are
// binned by four CTAs of a cluster, each holding the counters of a band of rows.  All four walk the
// path's lines, a quarter each, and add to each other's counters through distributed shared memory;
// the bands' column sums and totals are exchanged the same way.  The global passes that these
// rects took before walk every line twice with global atomics on two arrays (mixed 8,192 paths on
// 4095 x 4095, some 150 of such rects: binning 0.83 ms, of which 0.61 in those passes; now 0.38).
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// The address of a shared variable of the cluster's CTA `rank`, in the cluster's shared window.
__device__ __forceinline__ uint32_t cluster_addr(const void *p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_add(uint32_t addr, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t cluster_fetch_add(uint32_t addr, uint32_t v) {
    uint32_t old;
    asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ uint32_t cluster_load(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

constexpr int kClusterThreads = 384, kClusterWarps = kClusterThreads / 32;
constexpr uint32_t kClusterStage = 1024;  // visits staged per warp
constexpr size_t kClusterSmem = (kClusterTiles + 2 * kClusterCols) * 4;

__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 3) k_bin_cluster(Batch b) {
    extern __shared__ uint32_t sm[];
    uint32_t *const cnt = sm;                                              // this band's tiles
    int32_t *const above = reinterpret_cast<int32_t *>(sm + kClusterTiles);  // CTA 0: deltas above the rect
    int32_t *const colsum = above + kClusterCols;                          // this band's delta sums
    __shared__ uint32_t s_item, s_base, s_write, s_next, s_over;
    __shared__ uint32_t s_total[2 * kClusterCtas];  // every CTA's fills (64 bits each)
    __shared__ uint32_t s_slot[kClusterWarps], s_warp[kClusterWarps];
    __shared__ unsigned long long s_wsum[kClusterWarps];
    const uint32_t tid = threadIdx.x;
    const int lane = (int)(tid & 31), warp = (int)(tid >> 5);
    const unsigned below = (1u << lane) - 1u;
    const uint32_t rank = blockIdx.x % kClusterCtas;
    uint2 *const stage = b.stage + ((size_t)blockIdx.x * kClusterWarps + warp) * kClusterStage;
    uint32_t *const stage_tile = b.stage_tile + ((size_t)blockIdx.x * kClusterWarps + warp) * kClusterStage;
    const uint32_t *list = list_row(b, kListCluster);
    const uint32_t n_items = b.bin_ctl[kCtlCount + kListCluster];
    uint32_t *const err = &b.status[kStErr];
    for (;;) {
        if (rank == 0 && tid == 0) {
            const uint32_t t = atomicAdd(&b.bin_ctl[kCtlTicketCluster], 1u);
            for (uint32_t r = 0; r < kClusterCtas; r++) cluster_store(cluster_addr(&s_item, r), t);
        }
        cluster_sync();  // the ticket; and every CTA is done with the path before
        const uint32_t item = s_item;
        if (item >= n_items) return;
        const uint32_t p = list[item];
        const PathDev P = b.paths[p];
        const WalkCtx w = walk_ctx(b, P);
        const PathLeaves L = path_leaves(b, p);
        const uint32_t rw = (uint32_t)w.rw, rh = (uint32_t)w.rh;
        const uint32_t rows = cluster_rows(rh), band = rows * rw;  // tiles of a whole band
        const uint32_t y0 = min(rh, rank * rows), y1 = min(rh, y0 + rows), T = (y1 - y0) * rw;
        const uint32_t tb = P.tile_first + y0 * rw, cb = P.col_first;
        for (uint32_t t = tid; t < T; t += kClusterThreads) cnt[t] = 0;
        for (uint32_t x = tid; x < rw; x += kClusterThreads) above[x] = 0;
        if (tid == 0) {
            s_next = 0;
            s_over = 0;
        }
        cluster_sync();

        // 1. fill counts and backdrop deltas into the bands' counters, the visits staged.  CTA r
        //    takes every fourth group of lines from group r.
        auto tile_addr = [&](uint32_t local) {
            const uint32_t r = (uint32_t)(local >= band) + (uint32_t)(local >= 2 * band) + (uint32_t)(local >= 3 * band);
            return cluster_addr(cnt + (local - r * band), r);
        };
        uint32_t nstage = 0;
        auto on_fill = [&](int32_t local, uint2 q) {
            cluster_add(tile_addr((uint32_t)local), 1u);
            const uint32_t slot = atomicAdd(&s_slot[warp], 1u);
            if (slot < kClusterStage) {
                stage[slot] = q;
                stage_tile[slot] = (uint32_t)local | kVisitFill;
            }
        };
        auto on_above = [&](int32_t x, int d) { cluster_add(cluster_addr(above + x, 0), (uint32_t)d); };
        auto on_delta = [&](int32_t where, int d) {
            if (where >= 0) cluster_add(tile_addr((uint32_t)where), (uint32_t)d << 24);
            else on_above(-1 - where, d);
        };
        auto begin_single = [&]() {
            if (lane == 0) s_slot[warp] = nstage;
            __syncwarp();
        };
        auto end_single = [&]() {
            __syncwarp();
            nstage = s_slot[warp];
        };
        auto visit = [&](bool live, bool m, bool e, uint32_t pa, uint32_t pb, bool down, uint32_t local,
                         uint32_t inc) {
            const unsigned keep = __ballot_sync(0xffffffffu, live && (m || e));
            if (live && inc) cluster_add(tile_addr(local), inc);
            const uint32_t slot = nstage + __popc(keep & below);
            if ((keep >> lane & 1u) && slot < kClusterStage) {
                stage[slot] = make_uint2(pa, pb);
                stage_tile[slot] = local | (m ? kVisitFill : 0u) | (e ? kVisitExtra : 0u) | (down ? kVisitDown : 0u);
            }
            nstage += __popc(keep);
        };
        const uint32_t group = line_group(b, rw, rh, L.n, kClusterWarps * kClusterCtas);
        for (;;) {
            uint32_t g = 0;
            if (lane == 0) g = atomicAdd(&s_next, 1u);
            const uint32_t k0 = (__shfl_sync(0xffffffffu, g, 0) * kClusterCtas + rank) * group;
            if (k0 >= L.n) break;
            const uint32_t k = k0 + (uint32_t)lane;
            const bool have = (uint32_t)lane < group && k < L.n;
            const float4 f = have ? b.leaves[L.index(b, k)] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            walk_lines(w, f, have, b.long_line, visit, on_above, on_fill, on_delta, begin_single, end_single, err);
        }
        if (lane == 0 && nstage > kClusterStage) s_over = 1;
        cluster_sync();

        // 2. the band's fills (each warp's chunk of tiles) and column sums, told to every CTA
        const uint32_t chunk = ((T + kClusterWarps - 1) / kClusterWarps + 127u) & ~127u;
        const uint32_t c0 = min(T, (uint32_t)warp * chunk), c1 = min(T, c0 + chunk);
        unsigned long long wsum = 0;
        for (uint32_t t = c0 + lane; t < c1; t += 32) wsum += cnt[t] & 0xffffffu;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wsum += __shfl_down_sync(0xffffffffu, wsum, o);
        if (lane == 0) s_wsum[warp] = wsum;
        for (uint32_t x = tid; x < rw; x += kClusterThreads) {
            int32_t sum = 0;
            for (uint32_t t = x; t < T; t += rw) sum += (int8_t)(cnt[t] >> 24);
            colsum[x] = sum;
        }
        __syncthreads();
        if (tid == 0) {
            unsigned long long total = 0;
            for (int k = 0; k < kClusterWarps; k++) {
                const unsigned long long v = s_wsum[k];
                s_warp[k] = (uint32_t)total;
                total += v;
            }
            for (uint32_t r = 0; r < kClusterCtas; r++) {
                cluster_store(cluster_addr(&s_total[2 * rank], r), (uint32_t)total);
                cluster_store(cluster_addr(&s_total[2 * rank + 1], r), (uint32_t)(total >> 32));
            }
        }
        cluster_sync();
        unsigned long long before = 0, total = 0;  // fills of the bands above, of the path
        for (uint32_t r = 0; r < kClusterCtas; r++) {
            const unsigned long long v = s_total[2 * r] | (unsigned long long)s_total[2 * r + 1] << 32;
            if (r < rank) before += v;
            total += v;
        }
        if (rank == 0 && tid == 0) {
            const bool failed = walk_failed(err);  // in flight with the atomic
            const unsigned long long base = atomicAdd(fill_total(b), total);
            const bool fits = base + total <= (unsigned long long)b.fill_cap;
            if (!fits) atomicOr(err, kErrOverflowFill);
            b.path_fill[p] = (uint32_t)base;
            for (uint32_t r = 0; r < kClusterCtas; r++) {
                cluster_store(cluster_addr(&s_base, r), (uint32_t)base);
                cluster_store(cluster_addr(&s_write, r), fits && total > 0 && !failed ? 1u : 0u);
            }
        }

        // 3. backdrops down the band's columns, from the sums of the bands above
        for (uint32_t x = tid; x < rw; x += kClusterThreads) {
            int32_t run = (int32_t)cluster_load(cluster_addr(above + x, 0));
            for (uint32_t r = 0; r < rank; r++) run += (int32_t)cluster_load(cluster_addr(colsum + x, r));
            for (uint32_t t = x; t < T; t += rw) {
                const uint32_t c = cnt[t];
                b.tile_state[tb + t] = (uint16_t)((uint32_t)(uint8_t)(int8_t)run | ((c & 0xffffffu) ? 0x100u : 0u));
                run += (int8_t)(c >> 24);
            }
            if (rank == kClusterCtas - 1) b.col_final[cb + x] = run;
        }
        cluster_sync();  // the base; and the counters are read before they become cursors

        // 4. write cursors and end offsets: a warp scan of each warp's chunk
        uint32_t carry = s_base + (uint32_t)before + s_warp[warp];
        for (uint32_t t0 = c0; t0 < c1; t0 += 32) {
            const uint32_t t = t0 + (uint32_t)lane, own = t < c1 ? cnt[t] & 0xffffffu : 0u;
            uint32_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += n;
            }
            if (t < c1) {
                cnt[t] = carry + incl - own;
                b.tile_fills[tb + t] = carry + incl;
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        cluster_sync();

        // 5. the fills, grouped by tile, from this CTA's stages or by walking its lines again
        if (s_write && !s_over) {
            for (uint32_t k = lane; k < nstage; k += 32) {
                const uint2 q = stage[k];
                const uint32_t t = stage_tile[k], m = t >> 16 & 1u, e = t >> 17 & 1u;
                const uint32_t at = cluster_fetch_add(tile_addr(t & 0xffffu), m + e);
                if (m) b.fills[at] = q;
                if (e) b.fills[at + m] = t & kVisitDown ? make_uint2(0u, q.x) : make_uint2(q.y, 0u);
            }
        } else if (s_write) {
            // the lines that this CTA's warps counted: every fourth group, from group `rank`
            for (uint32_t j = tid;; j += kClusterThreads) {
                const uint32_t k = (j / group * kClusterCtas + rank) * group + j % group;
                if (k >= L.n) break;
                const float4 f = b.leaves[L.index(b, k)];
                walk_line(
                    w, f.x, f.y, f.z, f.w,
                    [&](int32_t local, uint2 q) { b.fills[cluster_fetch_add(tile_addr((uint32_t)local), 1u)] = q; },
                    [&](int32_t, int) {}, err);
            }
        }
        __syncwarp();  // whole warps at the barrier
    }
}

// Class 3: clear the counters, deltas and column sums of the paths' tiles.
__global__ void k_bin_zero_large(Batch b) {
    __shared__ uint32_t s_item;
    const uint32_t n3 = (uint32_t)(*ctl3_word(b) >> 40);
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(&b.bin_ctl[kCtlTicketZero], 1u);
        __syncthreads();
        const uint32_t item = s_item;
        __syncthreads();
        if (item >= n3) return;
        const PathDev P = b.paths[b.bin_list[(size_t)3 * b.n_paths + item]];
        const uint32_t rw = (uint32_t)(P.rx1 - P.rx0), T = rw * (uint32_t)max(P.ry1 - P.ry0, 0);
        for (uint32_t t = threadIdx.x; t < T; t += blockDim.x) {
            b.tile_fills[P.tile_first + t] = 0;
            b.tile_state[P.tile_first + t] = 0;
        }
        for (uint32_t x = threadIdx.x; x < rw; x += blockDim.x) b.col_above[P.col_first + x] = 0;
    }
}

// Class 3, per line (strided over the class-3 numbering of lines): count (global atomics on
// the tile counters, deltas into the low byte of the tile state) or write (the counters have
// become cursors).
template <bool kWrite>
__global__ void __launch_bounds__(kThreads) k_bin_large(Batch b) {
    const unsigned long long c3 = *ctl3_word(b);
    const uint32_t n3 = (uint32_t)(c3 >> 40), total = (uint32_t)(c3 & kLow40);
    if (n3 == 0) return;
    if (kWrite && (b.status[kStErr] & kErrOverflowFill)) return;
    const uint32_t *list = b.bin_list + (size_t)3 * b.n_paths, *first = b.bin_list + (size_t)4 * b.n_paths;
    for (uint32_t j = global_tid(); j < total; j += gridDim.x * blockDim.x) {
        const uint32_t item = upper_bound(first, n3, j) - 1;
        const uint32_t p = list[item];
        const PathDev P = b.paths[p];
        const PathLeaves L = path_leaves(b, p);
        const float4 f = b.leaves[L.index(b, j - first[item])];
        const WalkCtx w = walk_ctx(b, P);
        const uint32_t tb = P.tile_first, cb = P.col_first;
        if (kWrite) {
            walk_line(
                w, f.x, f.y, f.z, f.w,
                [&](int32_t local, uint2 q) { b.fills[atomicAdd(&b.tile_fills[tb + (uint32_t)local], 1u)] = q; },
                [&](int32_t, int) {}, &b.status[kStErr]);
        } else {
            walk_line(
                w, f.x, f.y, f.z, f.w, [&](int32_t local, uint2) { atomicAdd(&b.tile_fills[tb + (uint32_t)local], 1u); },
                [&](int32_t where, int d) {
                    if (where >= 0) add_delta_u16(&b.tile_state[tb + (uint32_t)where], d, &b.status[kStErr]);
                    else atomicAdd(&b.col_above[cb + (uint32_t)(-1 - where)], d);
                },
                &b.status[kStErr]);
        }
    }
}

// Class 3, one CTA per path: backdrops down each column, then the path's block of fills and
// the counts scanned into write cursors.
constexpr int kPrepThreads = 256;

__global__ void __launch_bounds__(kPrepThreads) k_bin_large_prep(Batch b) {
    constexpr int kWarps = kPrepThreads / 32;
    __shared__ uint32_t s_item, s_base;
    __shared__ unsigned long long s_red[kWarps];
    __shared__ uint32_t s_warp[kWarps];
    const uint32_t tid = threadIdx.x;
    const int lane = (int)(tid & 31), warp = (int)(tid >> 5);
    const uint32_t n3 = (uint32_t)(*ctl3_word(b) >> 40);
    for (;;) {
        if (tid == 0) s_item = atomicAdd(&b.bin_ctl[kCtlTicketPrep], 1u);
        __syncthreads();
        const uint32_t item = s_item;
        if (item >= n3) return;
        const uint32_t p = b.bin_list[(size_t)3 * b.n_paths + item];
        const PathDev P = b.paths[p];
        const uint32_t rw = (uint32_t)max(P.rx1 - P.rx0, 0), rh = (uint32_t)max(P.ry1 - P.ry0, 0), T = rw * rh;
        const uint32_t tb = P.tile_first, cb = P.col_first;
        unsigned long long sum = 0;
        for (uint32_t x = tid; x < rw; x += kPrepThreads) {
            int32_t run = b.col_above[cb + x];
            uint32_t y = 0;
            // eight rows at a time: their counters and deltas are loaded before any of the
            // eight states is rewritten, so the loads overlap instead of following each store
            for (; y + 8 <= rh; y += 8) {
                uint32_t cnt[8];
                uint16_t state[8];
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint32_t t = tb + (y + k) * rw + x;
                    cnt[k] = b.tile_fills[t];
                    state[k] = b.tile_state[t];
                }
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint32_t t = tb + (y + k) * rw + x;
                    b.tile_state[t] = (uint16_t)((uint32_t)(uint8_t)(int8_t)run | (cnt[k] ? 0x100u : 0u));
                    run += (int8_t)(state[k] & 0xffu);
                    sum += cnt[k];
                }
            }
            for (; y < rh; y++) {
                const uint32_t t = tb + y * rw + x, c = b.tile_fills[t];
                const int8_t delta = (int8_t)(b.tile_state[t] & 0xffu);
                b.tile_state[t] = (uint16_t)((uint32_t)(uint8_t)(int8_t)run | (c ? 0x100u : 0u));
                run += delta;
                sum += c;
            }
            b.col_final[cb + x] = run;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
        if (lane == 0) s_red[warp] = sum;
        __syncthreads();
        if (tid == 0) {
            unsigned long long total = 0;
            for (int k = 0; k < kWarps; k++) total += s_red[k];
            const unsigned long long base = atomicAdd(fill_total(b), total);
            if (base + total > (unsigned long long)b.fill_cap) atomicOr(&b.status[kStErr], kErrOverflowFill);
            b.path_fill[p] = (uint32_t)base;
            s_base = (uint32_t)base;
        }
        __syncthreads();
        // exclusive scan of the counters into write cursors, four consecutive tiles a thread
        uint32_t carry = s_base;
        for (uint32_t t0 = 0; t0 < T; t0 += 4 * kPrepThreads) {
            const uint32_t t = t0 + 4 * tid;
            uint32_t v[4], own = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v[k] = t + k < T ? b.tile_fills[tb + t + k] : 0u;
                own += v[k];
            }
            uint32_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += n;
            }
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            uint32_t before = 0, chunk_total = 0;
            for (int k = 0; k < kWarps; k++) {
                if (k < warp) before += s_warp[k];
                chunk_total += s_warp[k];
            }
            uint32_t cur = carry + before + incl - own;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (t + k < T) b.tile_fills[tb + t + k] = cur;
                cur += v[k];
            }
            carry += chunk_total;
            __syncthreads();
        }
    }
}

// Learned frame: list the spill pool's lines by path (count, scan, scatter), so each path's
// CTA finds its pooled lines.
__global__ void k_pool_count(Batch b) {
    const uint32_t n = min(b.status[kStPoolUsed], b.leaf_pool_cap);
    for (uint32_t j = global_tid(); j < n; j += gridDim.x * blockDim.x) atomicAdd(&b.pool_cnt[b.pool_path[j]], 1u);
}

__global__ void k_pool_scatter(Batch b) {
    const uint32_t n = min(b.status[kStPoolUsed], b.leaf_pool_cap);
    for (uint32_t j = global_tid(); j < n; j += gridDim.x * blockDim.x)
        b.pool_idx[atomicAdd(&b.pool_cnt[b.pool_path[j]], 1u)] = j;
}

// ---------------------------------------------------------------------------
// Per framebuffer-tile row of each scene: the scene's paths whose tile rect spans the row, in path
// order.  A block takes kRowWindow rows of a scene and a chunk of its paths (row_chunk of them, 256
// at a time, one per thread), counts the paths of each row into row_mat[scene][row][chunk], and,
// once that is scanned, writes them from there: the matrix is in the order of the lists, so the
// scan gives every chunk its place in every row and path order needs no sort.  A block's cost is its
// paths plus its rows, wherever the paths lie.  (One block per row, testing every path of the
// scene, took 0.83 ms of the 2.3 ms frame of 150,000 glyphs on 128 rows, and 0.12 ms of 2.0 ms with
// 20,000 paths on 256 rows.)

constexpr int kRowThreads = 256, kRowWarps = kRowThreads / 32;
// Row-entry flag of a clipped path; mask sources of a clipped tile.
constexpr uint32_t kRowClipped = 16u;
enum : uint32_t { kMaskOwn = 0, kMaskClip = 1, kMaskBoth = 2 };

template <bool kWrite>
__global__ void __launch_bounds__(kRowThreads) k_rows(Batch b) {
    __shared__ int s_cnt[kRowWarps][kRowWindow + 1];  // per warp: the rows' paths (as differences, then summed)
    __shared__ uint32_t s_out[kRowWindow];            // the rows' next entries (kWrite), or counts so far
    const uint32_t blk = b.rblk_base + blockIdx.x;
    const uint32_t s = upper_bound(b.scene_rblk_first + b.scene_base, b.n_scenes + 1, blk) - 1 + b.scene_base;
    const SceneDev &S = b.scenes[s];
    const uint32_t paths = S.path_end - S.path_first, chunks = max(1u, (paths + b.row_chunk - 1) / b.row_chunk);
    const uint32_t local = blk - S.rblk_first, chunk = local % chunks;
    const int32_t y0 = (int32_t)(local / chunks * kRowWindow), rows = min((int32_t)S.fbh - y0, kRowWindow);
    uint32_t *const mat = b.row_mat + (S.rmat_first - b.rmat_base) + (size_t)y0 * chunks + chunk;
    const uint32_t p0 = S.path_first - b.path_base + chunk * b.row_chunk;
    const uint32_t p1 = min(p0 + b.row_chunk, S.path_end - b.path_base);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    if (tid < rows) s_out[tid] = kWrite ? mat[(size_t)tid * chunks] : 0u;
    if (kWrite && chunk == 0 && tid < rows) b.row_first[S.row_first - b.row_base + y0 + tid] = mat[(size_t)tid * chunks];
    if (kWrite && blockIdx.x == 0 && tid == 0) b.row_first[b.n_rows] = b.status[kStRows];
    uint32_t seen = 0;  // lane 0: a bit per binning class
    for (uint32_t base = p0; base < p1; base += kRowThreads) {
        for (int k = lane; k <= kRowWindow; k += 32) s_cnt[warp][k] = 0;
        __syncwarp();
        // the path's rows in this window, its columns inside the framebuffer
        const uint32_t p = base + tid;
        PathDev P{};
        int32_t cx0 = 0, cx1 = 0, a = 0, e = 0;
        if (p < p1) {
            P = b.paths[p];
            if (kWrite) {
                P.tile_first = b.path_tiles[p];
                if (y0 == 0) {  // one block of the chunk leaves them to the kernels that follow
                    b.paths[p].tile_first = P.tile_first;
                    b.paths[p].col_first = b.path_cols[p];
                }
            }
            cx0 = max(P.rx0, 0);
            cx1 = min(P.rx1, (int32_t)S.fbw);
            if (cx0 < cx1 && !(P.flags & kPathIsClip)) {
                a = max(P.ry0 - y0, 0);
                e = min(P.ry1 - y0, rows);
            }
        }
        if (!kWrite && y0 == 0) {
            // which binning classes the rects ask for
            const uint32_t w = (uint32_t)max(P.rx1 - P.rx0, 0), h = (uint32_t)max(P.ry1 - P.ry0, 0);
            const uint32_t classes = __reduce_or_sync(0xffffffffu, w ? 1u << rect_class(w, h) : 0u);
            if (lane == 0) seen |= classes;
        }
        const bool spans = a < e;
        if (spans) {
            atomicAdd(&s_cnt[warp][a], 1);
            atomicAdd(&s_cnt[warp][e], -1);
        }
        __syncwarp();
        // differences to counts: two rows a lane
        {
            const int u = s_cnt[warp][2 * lane], v = s_cnt[warp][2 * lane + 1];
            int incl = u + v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int n = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += n;
            }
            s_cnt[warp][2 * lane] = incl - v;
            s_cnt[warp][2 * lane + 1] = incl;
        }
        __syncthreads();
        // per row: the warps' first entries (kWrite), and the rows' totals
        if (tid < rows) {
            uint32_t run = s_out[tid];
            for (int k = 0; k < kRowWarps; k++) {
                const uint32_t c = (uint32_t)s_cnt[k][tid];
                s_cnt[k][tid] = (int)run;
                run += c;
            }
            s_out[tid] = run;
        }
        __syncthreads();
        if (kWrite) {
            const int lo = __reduce_min_sync(0xffffffffu, spans ? a : kRowWindow);
            const int hi = __reduce_max_sync(0xffffffffu, spans ? e : 0);
            const bool clipped = spans && b.path_clip_cat && b.path_clip_rel[p] != kNone;
            const uint32_t flags = P.flags | (clipped ? kRowClipped : 0u), rw = (uint32_t)(P.rx1 - P.rx0);
            // tile index of column 0 of a row in the path's numbering (may underflow by rx0;
            // adding fx >= rx0 brings it back into range)
            uint32_t row_tile = P.tile_first + (uint32_t)(y0 + lo - P.ry0) * rw - (uint32_t)P.rx0;
            for (int r = lo; r < hi; r++, row_tile += rw) {
                const bool in = spans && a <= r && r < e;
                const unsigned m = __ballot_sync(0xffffffffu, in);
                const uint32_t at = (uint32_t)s_cnt[warp][r] + __popc(m & below);
                // flags: bit 0 even-odd, bit 1 occludes, bit 2 the rect's first tile (its first
                // row, first column) is in this row of the framebuffer, bit 4 the path is clipped
                const bool first = y0 + r == P.ry0 && P.rx0 >= 0;
                if (in && at < b.row_cap)
                    b.row_paths[at] = make_uint4(p, (uint32_t)cx0 | ((uint32_t)cx1 << 16), row_tile,
                                                 flags | (first ? 4u : 0u));
            }
            __syncthreads();  // the counts are read before the next paths clear them
        }
    }
    if (kWrite) return;
    if (tid < rows) mat[(size_t)tid * chunks] = s_out[tid];
    for (int c = 0; c <= kClusterClass; c++)
        if (seen >> c & 1u) b.status[kStRectClass + c] = 1;
}

// ---------------------------------------------------------------------------
// Coverage of one alpha tile, accumulated by a warp into shared memory.
//
// A fill contributes, to the pixel (i, j) of its tile, the signed area inside the pixel
// between the fill and the tile bottom (the quantity fill.comp:51-100 looks up in its area
// LUT).  Along a pixel column that area steps from 0 (rows above the line) to the fill's
// x-extent (rows below it), so the fill is stored as per-row differences: every piece of
// the fill inside one cell (i, r) with x-width w and mean in-row depth m adds w(1-m) to
// row r and w*m to row r+1; a prefix sum down the column restores the area.  Values are
// int32 fixed point (kCovShift fraction bits), so the result does not depend on fill order.

// 16 rows of 16 cells, and a row below them for what the bottom row passes on (never read)
constexpr int kCovCells = 17 * 16;

// an area as int32 fixed point, rounded to nearest even: the low bits of a sum with 1.5 * 2^23, as
// areas are at most 1 (the product is exact)
__device__ __forceinline__ int cov_fixed(float v) {
    return (int)(__float_as_uint(__fmaf_rn(v, (float)(1 << kCovShift), kMagic)) - __float_as_uint(kMagic));
}

// Per-fill set-up shared by the (fill, column) work items of one alpha tile, as the lanes read it:
// two 16-byte loads.
struct alignas(16) FillPrep {
    float xl, yl, xr, yr, dydx, s;
    int off;  // work item k is pixel column off + k
    int pad;
};

// The piece of fill `fp` inside pixel column i: per-row differences into D, one addition per row
// (a cell's part for its own row with what the cell above passes on).  Rows the piece crosses from
// top to bottom all get the same part.  (Two additions per row, each with its own bounds check and
// padded index, and a search for the item's fill: the composite took 292 us on 20,000 paths, of
// which half here; now 235 us.  Clipped batch 455 -> 400 us.)
__device__ __forceinline__ void raster_column(const FillPrep &fp, int i, int *D) {
    const float xa = fmaxf(fp.xl, (float)i), xb = fminf(fp.xr, (float)(i + 1));
    const float w = xb - xa;
    if (!(w > 0.0f)) return;
    const float ya = xa == fp.xl ? fp.yl : fp.yl + fp.dydx * (xa - fp.xl);
    const float yb = xb == fp.xr ? fp.yr : fp.yl + fp.dydx * (xb - fp.xl);
    const float ylo = fminf(ya, yb), yhi = fmaxf(ya, yb);
    const float rf = floorf(ylo);
    const float sw = fp.s * w, hi = fminf(yhi, rf + 1.0f);
    int *cell = D + ((int)rf * 16 + i);
    const float m = 0.5f * (ylo + hi) - rf;
    float wr = sw;
    if (yhi <= rf + 1.0f) {
        atomicAdd(cell, cov_fixed(wr * (1.0f - m)));
        atomicAdd(cell + 16, cov_fixed(wr * m));
        return;
    }
    const float inv_h = 1.0f / (yhi - ylo);
    wr = sw * (hi - ylo) * inv_h;
    atomicAdd(cell, cov_fixed(wr * (1.0f - m)));
    int pass = cov_fixed(wr * m);
    const int whole = cov_fixed(sw * inv_h * 0.5f);
    const float last = fminf(ceilf(yhi) - 1.0f, 15.0f);
    float r = rf + 1.0f;
    for (; r < last; r += 1.0f) {
        cell += 16;
        atomicAdd(cell, pass + whole);
        pass = whole;
    }
    const float lo = r, end = fminf(yhi, r + 1.0f);
    wr = sw * (end - lo) * inv_h;
    const float me = 0.5f * (lo + end) - r;
    atomicAdd(cell + 16, pass + cov_fixed(wr * (1.0f - me)));
    atomicAdd(cell + 32, cov_fixed(wr * me));
}

// Warp computes the coverage of the 8 pixels of every lane (column lane&15, rows
// (lane>>4)*8 .. +7) of an alpha tile; D must be zero on entry and is left zero.
// Fills are rasterised as (fill, pixel column) work items spread over the lanes, 32 fills
// at a time, so a tile of a few wide fills still keeps the warp busy.  The kernel is bound by
// instructions, and a tile has few fills (5.6 on 20,000 paths), so what is done per round of 32
// items counts: an item's fill comes from a mask of the items that begin one (a binary search over
// the fills' first items was five dependent shared loads), its set-up in two loads.
// backdrop + the fills' area sums (fixed point) of the warp's 8 pixels per lane, before the fill rule
// src: the tile's n fills; q: with kLoaded this lane's fill of the first 32 (any value from lane n on),
// else not read.
// lane: the caller's, passed down because the composite spills more when each of these functions asks
// for its own (256 scenes, composite 2.90 -> 2.83 ms).
template <bool kLoaded>
__device__ __forceinline__ void coverage_raw(int lane, const uint2 *src, uint32_t n, uint2 q, int8_t bd, int *D,
                                             FillPrep *prep, int raw[8]) {
    const unsigned below = (1u << lane) - 1u;
    for (uint32_t base = 0; base < n; base += 32) {
        const uint32_t left = n - base;
        int items = 0;
        FillPrep fp;
        if ((uint32_t)lane < left) {
            if (!kLoaded || base > 0) q = src[base + lane];
            const float x0 = (float)(q.x & 0xffffu) * (1.0f / 256.0f), y0 = (float)(q.x >> 16) * (1.0f / 256.0f);
            const float x1 = (float)(q.y & 0xffffu) * (1.0f / 256.0f), y1 = (float)(q.y >> 16) * (1.0f / 256.0f);
            fp.s = x0 > x1 ? 1.0f : -1.0f;
            fp.xl = fminf(x0, x1);
            fp.xr = fmaxf(x0, x1);
            fp.yl = x0 < x1 ? y0 : y1;
            fp.yr = x0 < x1 ? y1 : y0;
            // xr - xl >= 1/256 (vertical fills are culled when quantised): the fast divide is
            // within 2 ulp, far inside the coverage tolerance
            fp.dydx = __fdividef(fp.yr - fp.yl, fp.xr - fp.xl);
            const int i0 = max((int)floorf(fp.xl), 0);
            items = max(min((int)ceilf(fp.xr), 16) - i0, 0);
            fp.off = i0;
        }
        int incl = items;
        for (uint32_t d = 1; d < min(left, 32u); d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (int)d) incl += t;
        }
        const int total = __shfl_sync(0xffffffffu, incl, (int)min(left, 32u) - 1);
        const int first = incl - items;
        // the fills with items, without gaps
        const unsigned some = __ballot_sync(0xffffffffu, items > 0);
        if (items > 0) {
            fp.off -= first;
            prep[__popc(some & below)] = fp;
        }
        __syncwarp();
        int begun = 0;  // fills whose items began in the rounds before
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int at = first - k0;
            const unsigned starts = __reduce_or_sync(0xffffffffu, items > 0 && at >= 0 && at < 32 ? 1u << at : 0u);
            const int k = k0 + lane;
            if (k < total) {
                const FillPrep g = prep[begun + __popc(starts & (below | 1u << lane)) - 1];
                raster_column(g, g.off + k, D);
            }
            begun += __popc(starts);
        }
        __syncwarp();
    }
    // read and clear: the next tile starts from zero cells.  The halves of the warp read their rows
    // in pairs of opposite order, so that they are in opposite halves of the banks.
    const int col = lane & 15, h = lane >> 4;
    int *const cells = D + h * 128 + col;
    int acc[8];
    int run = 0;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        int *const c0 = cells + (k + h) * 16, *const c1 = cells + (k + 1 - h) * 16;
        const int a = *c0, b = *c1;
        *c0 = 0;
        *c1 = 0;
        acc[k] = run + (h ? b : a);
        run += a + b;
        acc[k + 1] = run;
    }
    const int upper = __shfl_sync(0xffffffffu, run, col);  // rows 0..7 total of this column
    const int base = (h ? upper : 0) + ((int)bd << kCovShift);
#pragma unroll
    for (int k = 0; k < 8; k++) raw[k] = base + acc[k];
}

// The fill rule (fill.comp:133-140): nonzero min(|c|, 1), even-odd 1 - |1 - (c mod 2)|.
__device__ __forceinline__ void coverage_rule(const int raw[8], bool eo, float cov[8]) {
    const float scale = 1.0f / (float)(1 << kCovShift);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int c = raw[k];
        if (!eo) {
            cov[k] = fminf(fabsf((float)c) * scale, 1.0f);
        } else {
            const float t = (float)(c & ((2 << kCovShift) - 1)) * scale;
            cov[k] = __saturatef(1.0f - fabsf(1.0f - t));
        }
    }
}

__device__ __forceinline__ void alpha_coverage(const Batch &b, uint32_t f0, uint32_t f1, int8_t bd, bool eo, int *D,
                                               FillPrep *prep, float cov[8]) {
    int raw[8];
    const uint32_t lane = threadIdx.x & 31;
    const uint2 q = lane < f1 - f0 ? b.fills[f0 + lane] : make_uint2(0u, 0u);
    coverage_raw<true>((int)lane, b.fills + f0, f1 - f0, q, bd, D, prep, raw);
    coverage_rule(raw, eo, cov);
}

__device__ __forceinline__ void zero_cells(int *D) {
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < kCovCells; k += 32) D[k] = 0;
    __syncwarp();
}

constexpr int kCompWarps = 1;

// One framebuffer tile: walk the paths spanning its row from the topmost down, test 32
// candidates at a time (one per lane), and visit the visible tiles in order.  A visible tile
// is an alpha tile or a solid tile with a nonzero backdrop (scene_builder.cpp:57-63); the
// walk ends at the first occluding tile - a solid, opaque tile whose fill rule covers it
// (the d3d11 z-buffer rule, propagate.comp:190-205) - so the tiles visited are exactly the
// framebuffer tile's composite list after z-culling (sort.comp:49-83), in reverse order.
// With kFetch, every visible candidate also loads its colour and (alpha tiles) its fill
// range in parallel before the visits, so a visit waits on its fills alone; with kAhead, the next
// candidate's first fills are loaded during the visit before it.
// visit(candidate) returns true to stop the walk.
struct Cand {
    uint32_t p, gt, st, flags;  // st: the tile state, with a clipped tile's mask source in bits 9-10
                                // and (kMaskBoth) the draw tile's own backdrop in bits 16-23
    uint32_t f0, f1, color;     // kFetch only (kMaskClip: the clip tile's fills)
    uint2 q;                    // kFetch: this lane's fill of the first 32
    uint32_t gc;                // kMaskClip, kMaskBoth: the clip tile
};

__device__ __forceinline__ uint32_t mask_mode(uint32_t st) { return (st >> 9) & 3u; }

// A clipped draw tile against the clip path's tile at the same coordinates
// (Tiler::prepare_tiles, pathfinder/core/d3d9/tiler.cpp:386-431): culled outside the clip's
// rect or over a blank clip tile; a solid tile over a clip alpha tile takes the clip's mask and
// backdrop; an alpha tile over a clip alpha tile keeps its mask, to be combined with the clip's,
// and its backdrop is zeroed; otherwise unchanged.  Updates c.st (and c.f0/f1, c.gc).
__device__ __forceinline__ void apply_clip(const Batch &b, uint32_t p, int32_t tx, int32_t ty, Cand &c) {
    const uint32_t cp = b.path_clip_rel[p];
    const PathDev C = b.paths[cp];
    if (tx < C.rx0 || tx >= C.rx1 || ty < C.ry0 || ty >= C.ry1) {
        c.st = 0;
        return;
    }
    const uint32_t gc = C.tile_first + (uint32_t)((ty - C.ry0) * (C.rx1 - C.rx0) + (tx - C.rx0));
    const uint32_t cs = b.tile_state[gc];
    const bool ca = (cs & 0x100u) != 0, da = (c.st & 0x100u) != 0;
    const int8_t cbd = (int8_t)(cs & 0xffu), dbd = (int8_t)(c.st & 0xffu);
    if (ca && da) {
        c.st = 0x100u | kMaskBoth << 9 | (uint32_t)(uint8_t)dbd << 16;
        c.gc = gc;
    } else if (ca && dbd != 0) {
        c.st = 0x100u | kMaskClip << 9 | (uint32_t)(uint8_t)cbd;
        c.f0 = gc == C.tile_first ? b.path_fill[cp] : b.tile_fills[gc - 1];
        c.f1 = b.tile_fills[gc];
        c.gc = gc;
    } else if (!ca && cbd == 0) {
        c.st = 0;
    }
}

template <bool kFetch, bool kClip, bool kAhead, class Visit>
__device__ __forceinline__ void walk_fb_tile(const Batch &b, int lane, uint32_t row, uint32_t fx, uint32_t fy,
                                             Visit &&visit, uint32_t &chunks) {
    const uint32_t k_lo = b.row_first[row], k_hi = b.row_first[row + 1];
    for (uint32_t top = k_hi; top > k_lo; top = top > k_lo + 32 ? top - 32 : k_lo) {
        chunks++;
        const int64_t k = (int64_t)top - 1 - lane;
        Cand c{0, 0, 0, 0, 0, 0, 0, make_uint2(0u, 0u), kNone};
        bool vis = false;
        if (k >= (int64_t)k_lo) {
            const uint4 e = b.row_paths[k];
            if (fx >= (e.y & 0xffffu) && fx < (e.y >> 16)) {
                c.p = e.x;
                c.flags = e.w;
                c.gt = e.z + fx;
                c.st = b.tile_state[c.gt];
                if (kClip && (c.flags & kRowClipped)) apply_clip(b, c.p, (int32_t)fx, (int32_t)fy, c);
                vis = c.st != 0;
                if (kFetch && vis) {
                    c.color = b.color[b.path_base + c.p];
                    if ((c.st & 0x100u) && mask_mode(c.st) != kMaskClip) {
                        // the first tile of a path starts the path's block of fills
                        const bool first = (c.flags & 4u) && fx == (e.y & 0xffffu);
                        c.f0 = first ? b.path_fill[c.p] : b.tile_fills[c.gt - 1];
                        c.f1 = b.tile_fills[c.gt];
                    }
                }
            }
        }
        uint32_t mask = __ballot_sync(0xffffffffu, vis);
        uint32_t nf0 = 0, nf1 = 0;
        uint2 nq = make_uint2(0u, 0u);
        auto next_fills = [&]() {
            const int l = __ffs(mask) - 1;
            nf0 = __shfl_sync(0xffffffffu, c.f0, l);
            nf1 = __shfl_sync(0xffffffffu, c.f1, l);
            if ((uint32_t)lane < nf1 - nf0) nq = b.fills[nf0 + lane];
        };
        if (kFetch && kAhead && mask) next_fills();
        while (mask) {
            const int l = __ffs(mask) - 1;
            mask &= mask - 1;
            Cand v;
            v.p = __shfl_sync(0xffffffffu, c.p, l);
            v.gt = __shfl_sync(0xffffffffu, c.gt, l);
            v.st = __shfl_sync(0xffffffffu, c.st, l);
            v.flags = __shfl_sync(0xffffffffu, c.flags, l);
            if (kFetch) {
                if (!kAhead) {
                    v.f0 = __shfl_sync(0xffffffffu, c.f0, l);
                    v.f1 = __shfl_sync(0xffffffffu, c.f1, l);
                } else {
                    v.f0 = nf0;
                    v.f1 = nf1;
                    v.q = nq;
                }
                v.color = __shfl_sync(0xffffffffu, c.color, l);
                if (kClip) v.gc = __shfl_sync(0xffffffffu, c.gc, l);
                if (kAhead && mask) next_fills();
            }
            if (visit(v)) return;
        }
    }
}

__device__ __forceinline__ bool solid_hidden(bool eo, int8_t bd) { return eo && ((bd < 0 ? -bd : bd) & 1) == 0; }

// First fill of tile gt of path p: the path's block starts at path_fill[p]; every other tile
// starts where the tile before it ends.
__device__ __forceinline__ uint32_t fill_begin(const Batch &b, uint32_t p, uint32_t gt) {
    return gt == b.path_tiles[p] ? b.path_fill[p] : b.tile_fills[gt - 1];
}

// The colour (straight alpha) a gradient gives the pixel centred at (x, y): tile.comp's colour
// texture coordinate (computeTileVaryings, tile.comp:694-724: the half-float transform times
// the pixel centre), filterRadialGradient (tile.comp:319-347) for radial gradients, then a
// linearly filtered fetch of the 256-texel ramp (clamped, or repeated for PF_WRAP_REPEAT).
__device__ __forceinline__ float4 gradient_color(const Batch &b, uint32_t g, float x, float y) {
    const float4 *m = b.grad_meta + 4 * g;
    const float4 m0 = m[0], m1 = m[1], m3 = m[3];
    const uint32_t type = __float_as_uint(m3.x);
    const bool repeat = __float_as_uint(m3.y) == PF_WRAP_REPEAT;
    float u;
    if (type == PF_PAINT_LINEAR) {
        u = m0.x * x + m0.z * y + m1.x;
    } else {
        const float4 m2 = m[2];
        const float cx = m0.x * x + m0.z * y + m1.x, cy = m0.y * x + m0.w * y + m1.y;
        const float dpx = cx - m1.z, dpy = cy - m1.w, dcx = m2.x, dcy = m2.y;
        const float r0 = m2.z, dr = m2.w - r0;
        const float a = dcx * dcx + dcy * dcy - dr * dr;
        const float bb = dpx * dcx + dpy * dcy + r0 * dr;
        const float c = dpx * dpx + dpy * dpy - r0 * r0;
        const float disc = bb * bb - a * c;
        if (!(disc > 0.0f)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // no real t (or the shader's 0)
        const float sq = sqrtf(disc);
        float t0 = (sq + bb) / a, t1 = (-sq + bb) / a;
        if (t0 > t1) {
            const float tmp = t0;
            t0 = t1;
            t1 = tmp;
        }
        u = t0 >= 0.0f ? t0 : t1;
    }
    if (!isfinite(u)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (repeat) u -= floorf(u);
    const float s = u * 256.0f - 0.5f, f0 = floorf(s), f = s - f0;
    int i0 = (int)fmaxf(fminf(f0, 1e9f), -1e9f), i1 = i0 + 1;
    if (repeat) {
        i0 &= 255;
        i1 &= 255;
    } else {
        i0 = min(max(i0, 0), 255);
        i1 = min(max(i1, 0), 255);
    }
    const uint32_t *ramp = b.grad_ramp + 256 * (size_t)g;
    const uint32_t p0 = __ldg(ramp + i0), p1 = __ldg(ramp + i1);
    const float inv = 1.0f / 255.0f;
    float4 o;
    o.x = ((float)(p0 & 0xffu) + ((float)(p1 & 0xffu) - (float)(p0 & 0xffu)) * f) * inv;
    o.y = ((float)((p0 >> 8) & 0xffu) + ((float)((p1 >> 8) & 0xffu) - (float)((p0 >> 8) & 0xffu)) * f) * inv;
    o.z = ((float)((p0 >> 16) & 0xffu) + ((float)((p1 >> 16) & 0xffu) - (float)((p0 >> 16) & 0xffu)) * f) * inv;
    o.w = ((float)(p0 >> 24) + ((float)(p1 >> 24) - (float)(p0 >> 24)) * f) * inv;
    return o;
}

// Warps per SM the registers are capped for.
__host__ __device__ constexpr int comp_warps(bool clip, bool paint) { return paint ? 20 : clip ? 24 : 32; }

// kClip: the batch has clip paths; kPaint: it has gradient paints; kTicket: resident warps
// take tiles by ticket (b.comp_ticket > 0).  Variants of their own, so that code one frame does
// not need costs it no registers.  The loop over tiles costs the ticketed ones registers, so they keep
// their place in the queue in shared memory, ask for their lane in every tile and don't load the next
// candidate's fills ahead (with all that in registers 276 and 236 bytes of spills, without and with clips,
// now 192 and 92; 256 scenes, a ticket per tile: 3.65 -> 3.09 ms, with clips 4.34 -> 3.62, with gradients
// 6.63 -> 6.10).
template <bool kClip, bool kPaint, bool kTicket>
__global__ void __launch_bounds__(kCompWarps * 32, comp_warps(kClip, kPaint) / kCompWarps) k_composite(Batch b) {
    __shared__ int cells[kCompWarps][kCovCells];
    __shared__ FillPrep prep[kCompWarps][32];
    __shared__ int park[kCompWarps][8][32];  // kMaskBoth: the clip tile's |coverage|
    // a frame whose leaf lines or fills overran their buffers is redone, one with a walk that hit its
    // bound is an error; nothing to read here
    if (b.status[kStErr] & (kErrOverflowLeaf | kErrOverflowFill | kErrWalk)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *D = cells[warp];
    zero_cells(D);  // once: coverage_raw leaves the cells it reads zero
    const float inv255 = 1.0f / 255.0f;
    uint32_t entries = 0, comp_fills = 0, chunks = 0;
    // one framebuffer tile per warp, or (kTicket) warps that stay and take comp_ticket
    // consecutive tiles at a time from a frame-wide ticket counter
    __shared__ uint32_t s_next[kCompWarps], s_left[kCompWarps];
    if (kTicket && lane == 0) s_left[warp] = 0;
    __syncwarp();
    for (uint32_t round = 0;; round++) {
        uint32_t fb;
        if (!kTicket) {
            if (round > 0) break;
            fb = blockIdx.x * kCompWarps + warp;
        } else {
            if (lane == 0) {
                if (s_left[warp] == 0) {
                    s_next[warp] = atomicAdd(&b.bin_ctl[kCtlCompTicket], b.comp_ticket);
                    s_left[warp] = b.comp_ticket;
                }
                s_left[warp]--;
            }
            __syncwarp();
            fb = s_next[warp];
            __syncwarp();
            if (lane == 0) s_next[warp] = fb + 1;
        }
        if (fb >= b.n_fb) break;
        int ln = lane;
        if (kTicket) asm volatile("mov.u32 %0, %%laneid;" : "=r"(ln));
        const int col = ln & 15, h = ln >> 4;
        const uint32_t fbg = b.fb_base + fb;
        const uint32_t s = b.fb_scene[fbg];
        const SceneDev &S = b.scenes[s];
        const uint32_t local = fbg - S.fb_first;
        const uint32_t fx = local % S.fbw, fy = local / S.fbw;
        // front to back: acc = sum of T * premultiplied source, T = product of (1 - a) above;
        // the accumulated alpha is 1 - T
        float ar[8], ag[8], ab[8], tr[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            ar[k] = ag[k] = ab[k] = 0.0f;
            tr[k] = 1.0f;
        }
        walk_fb_tile<true, kClip, !kTicket>(b, ln, S.row_first - b.row_base + fy, fx, fy, [&](const Cand &v) -> bool {
            const bool eo = (v.flags & 1u) != 0;
            const int8_t bd = (int8_t)(v.st & 0xffu);
            float cov[8];
            bool stop = false;
            entries++;
            if (!(v.st & 0x100u)) {
                if (solid_hidden(eo, bd)) return false;
#pragma unroll
                for (int k = 0; k < 8; k++) cov[k] = 1.0f;
                stop = (v.flags & 2u) != 0;
            } else {
                // the tile's own mask; kMaskClip (a solid tile over a clip alpha tile): the clip's;
                // kMaskBoth: the clip's mask first, parked, then the tile's own, combined as
                // tile_clip_combine.frag does - min(|draw + its backdrop|, |clip + its backdrop|) -
                // before the draw path's fill rule
                bool both = kClip && mask_mode(v.st) == kMaskBoth, combined = false;
                uint32_t f0 = v.f0, f1 = v.f1;
                int8_t tbd = bd;
                uint2 q = v.q;
                if (both) {
                    const uint32_t cp = b.path_clip_rel[v.p];
                    f0 = fill_begin(b, cp, v.gc);
                    f1 = b.tile_fills[v.gc];
                    if (!kTicket && (uint32_t)lane < f1 - f0) q = b.fills[f0 + lane];
                    tbd = (int8_t)(b.tile_state[v.gc] & 0xffu);
                }
                int raw[8];
                for (;;) {
                    comp_fills += f1 - f0;
                    coverage_raw<!kTicket>(ln, b.fills + f0, f1 - f0, q, tbd, D, prep[warp], raw);
                    __syncwarp();
                    if (!both) break;
#pragma unroll
                    for (int k = 0; k < 8; k++) park[warp][k][lane] = abs(raw[k]);
                    both = false;
                    combined = true;
                    f0 = v.f0;
                    f1 = v.f1;
                    q = v.q;
                    tbd = (int8_t)(v.st >> 16);
                }
                if (combined) {
#pragma unroll
                    for (int k = 0; k < 8; k++) raw[k] = min(abs(raw[k]), park[warp][k][lane]);
                }
                coverage_rule(raw, eo, cov);
            }
            const uint32_t color = v.color;
            float pr = (float)(color & 0xffu) * inv255, pg = (float)((color >> 8) & 0xffu) * inv255,
                  pb = (float)((color >> 16) & 0xffu) * inv255, pa = (float)(color >> 24) * inv255;
            const uint32_t grad = kPaint ? b.path_grad[b.path_base + v.p] : kNone;
            bool opaque = true;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (kPaint && grad != kNone) {  // SrcIn over the opaque white base colour
                    const float4 g = gradient_color(b, grad, (float)(fx * 16 + col) + 0.5f,
                                                    (float)(fy * 16 + h * 8 + k) + 0.5f);
                    pr = g.x;
                    pg = g.y;
                    pb = g.z;
                    pa = g.w;
                }
                const float a = pa * cov[k], w = tr[k] * a;
                ar[k] += w * pr;
                ag[k] += w * pg;
                ab[k] += w * pb;
                tr[k] *= 1.0f - a;
                opaque &= tr[k] == 0.0f;
            }
            return stop || __all_sync(0xffffffffu, opaque);
        }, chunks);
        // the scene's image fields in registers before the stores: a store through the image
        // pointer may alias the scene table as far as the compiler knows, and would make it
        // load them again for every pixel
        const uint32_t img_w = S.img_w, img_h = S.img_h, clear = S.clear;
        const bool load_dst = S.load == PF_LOAD_LOAD;
        uchar4 *const img = reinterpret_cast<uchar4 *>(b.image + S.img_offset);
        const uint32_t px = fx * 16 + (uint32_t)col;
        if (px < img_w) {
            float cr = (float)(clear & 0xffu) * inv255, cg = (float)((clear >> 8) & 0xffu) * inv255,
                  cb = (float)((clear >> 16) & 0xffu) * inv255, ca = (float)(clear >> 24) * inv255;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t py = fy * 16 + (uint32_t)(h * 8 + k);
                if (py < img_h) {
                    if (load_dst) {
                        // LOAD_ACTION_LOAD (tile.comp:744-757): start from the pixel already there
                        const uchar4 d = img[(size_t)py * img_w + px];
                        cr = (float)d.x * inv255;
                        cg = (float)d.y * inv255;
                        cb = (float)d.z * inv255;
                        ca = (float)d.w * inv255;
                    }
                    img[(size_t)py * img_w + px] =
                        make_uchar4((unsigned char)__float2uint_rn(__saturatef(ar[k] + tr[k] * cr) * 255.0f),
                                    (unsigned char)__float2uint_rn(__saturatef(ag[k] + tr[k] * cg) * 255.0f),
                                    (unsigned char)__float2uint_rn(__saturatef(ab[k] + tr[k] * cb) * 255.0f),
                                    (unsigned char)__float2uint_rn(__saturatef(1.0f - tr[k] + tr[k] * ca) * 255.0f));
                }
            }
        }
    }
    if (b.counters) {
        // one reduction per block into the frame counters
        __shared__ uint32_t red[kCompWarps][3];
        if (lane == 0) {
            red[warp][0] = entries;
            red[warp][1] = comp_fills;
            red[warp][2] = chunks;
        }
        __syncthreads();
        if (threadIdx.x < 3) {
            uint32_t v = 0;
            for (int w = 0; w < kCompWarps; w++) v += red[w][threadIdx.x];
            const int slot = threadIdx.x == 0 ? kStEntries : (threadIdx.x == 1 ? kStListFills : kStWalkChunks);
            if (v) atomicAdd(&b.status[slot], v);
        }
    }
}

// Frame counters: the draw paths' alpha tiles and visible tiles (an alpha tile or a nonzero
// backdrop: the tiles build_tile_batches keeps, core/d3d9/scene_builder.cpp:57-63).  One block
// per path, over its tile states.
__global__ void __launch_bounds__(kThreads) k_tile_counts(Batch b) {
    __shared__ uint32_t red[2][kThreads / 32];
    const uint32_t p = blockIdx.x;
    const PathDev P = b.paths[p];
    uint32_t alpha = 0, visible = 0;
    if (!(P.flags & kPathIsClip)) {
        const uint32_t T = (uint32_t)max(P.rx1 - P.rx0, 0) * (uint32_t)max(P.ry1 - P.ry0, 0);
        for (uint32_t t = threadIdx.x; t < T; t += kThreads) {
            const uint32_t st = b.tile_state[P.tile_first + t];
            alpha += (st >> 8) & 1u;
            visible += (st & 0x1ffu) != 0;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        alpha += __shfl_down_sync(0xffffffffu, alpha, o);
        visible += __shfl_down_sync(0xffffffffu, visible, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = alpha;
        red[1][threadIdx.x >> 5] = visible;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        uint32_t v = 0;
        for (int w = 0; w < kThreads / 32; w++) v += red[threadIdx.x][w];
        if (v) atomicAdd(&b.status[threadIdx.x == 0 ? kStAlphaTiles : kStVisible], v);
    }
}

// Composite lists and z per framebuffer tile for the canonical output (not part of a frame):
// the same walk as k_composite, written back to front.
template <bool kWrite>
__global__ void __launch_bounds__(kCompWarps * 32) k_list_dump(Batch b) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t fb = blockIdx.x * kCompWarps + warp;
    if (fb >= b.n_fb) return;
    const uint32_t fbg = b.fb_base + fb;
    const uint32_t s = b.fb_scene[fbg];
    const SceneDev &S = b.scenes[s];
    const uint32_t local = fbg - S.fb_first;
    const uint32_t fx = local % S.fbw, fy = local / S.fbw;
    uint32_t n = 0, first = 0, count = 0, n_chunks = 0;
    int32_t z = -1;
    if (kWrite) {
        first = b.fb_count[fb];
        count = b.fb_count[fb + 1] - first;
    }
    walk_fb_tile<false, true, false>(b, threadIdx.x & 31, S.row_first - b.row_base + fy, fx, fy, [&](const Cand &v) -> bool {
        if (kWrite && lane == 0) b.list[first + count - 1 - n] = v.gt;
        n++;
        const int8_t bd = (int8_t)(v.st & 0xffu);
        if (!(v.st & 0x100u) && (v.flags & 2u) && !solid_hidden((v.flags & 1u) != 0, bd)) {
            z = (int32_t)v.p;
            return true;
        }
        return false;
    }, n_chunks);
    if (lane == 0) {
        if (kWrite) b.z[fb] = z;
        else b.fb_count[fb] = n;
    }
}

// Every tile of the frame after the clip rules, for the canonical output (not part of a frame):
// the state the composite's walk sees - apply_clip, the same function, on each tile of a
// clipped path - and the clip tile whose mask it takes (kNone if none).  state[t] holds the
// int8 backdrop in bits 0-7, the alpha flag in bit 8, the mask source in bits 9-10 and, for
// kMaskBoth, the draw tile's own backdrop in bits 16-23.  One thread per tile.
__global__ void __launch_bounds__(kThreads) k_clip_dump(Batch b, uint32_t n_tiles, uint32_t *state, uint32_t *clip) {
    const uint32_t t = global_tid();
    if (t >= n_tiles) return;
    const uint32_t p = upper_bound(b.path_tiles, b.n_paths + 1, t) - 1;
    Cand c{0, t, b.tile_state[t], 0, 0, 0, 0, make_uint2(0u, 0u), kNone};
    if (b.path_clip_rel[p] != kNone && !(b.paths[p].flags & kPathIsClip)) {
        const PathDev P = b.paths[p];
        const uint32_t local = t - P.tile_first, rw = (uint32_t)(P.rx1 - P.rx0);
        apply_clip(b, p, P.rx0 + (int32_t)(local % rw), P.ry0 + (int32_t)(local / rw), c);
        if (mask_mode(c.st) == kMaskOwn) c.gc = kNone;
    }
    state[t] = c.st;
    clip[t] = c.gc;
}

// Coverage of listed alpha tiles after the fill rule (test output; one warp per tile).
__global__ void __launch_bounds__(kCompWarps * 32) k_coverage_dump(Batch b, const uint32_t *tiles, uint32_t n,
                                                                   float *out) {
    __shared__ int cells[kCompWarps][kCovCells];
    __shared__ FillPrep prep[kCompWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t k = blockIdx.x * kCompWarps + warp;
    if (k >= n) return;
    int *D = cells[warp];
    const uint32_t gt = tiles[k];
    const uint32_t p = upper_bound(b.path_tiles, b.n_paths + 1, gt) - 1;
    zero_cells(D);
    float cov[8];
    alpha_coverage(b, fill_begin(b, p, gt), b.tile_fills[gt], (int8_t)(b.tile_state[gt] & 0xffu),
                   (b.paths[p].flags & 1u) != 0, D, prep[warp], cov);
    const int col = lane & 15, h = lane >> 4;
#pragma unroll
    for (int r = 0; r < 8; r++) out[(size_t)k * 256 + (h * 8 + r) * 16 + col] = cov[r];
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers

static std::atomic<uint64_t> g_launches{0};
uint64_t launches() { return g_launches.load(); }
void count_launches(uint32_t n) { g_launches += n; }

#define PF_LAUNCH(...)           \
    do {                         \
        __VA_ARGS__;             \
        count_launches(1);       \
    } while (0)

cudaError_t launch_paths(const Batch &b, uint2 *path_contours, cudaStream_t st) {
    if (b.n_paths) PF_LAUNCH(k_paths<<<grid_for(b.n_paths, kPathThreads / 32), kPathThreads, 0, st>>>(b, path_contours));
    return cudaGetLastError();
}

cudaError_t launch_contour_segments(const Batch &b, uint64_t n_points, bool write, cudaStream_t st) {
    if (!b.n_contours) return cudaSuccess;
    const uint32_t sample = b.n_contours / 2048 + 1;
    if (n_points <= uint64_t(b.n_contours) * 40) {
        const unsigned grid = grid_for(b.n_contours, kThreads / 8);
        if (write) PF_LAUNCH(k_contour_segments<true, 8><<<grid, kThreads, 0, st>>>(b, sample));
        else PF_LAUNCH(k_contour_segments<false, 8><<<grid, kThreads, 0, st>>>(b, sample));
    } else {
        const unsigned grid = grid_for(b.n_contours, kThreads / 32);
        if (write) PF_LAUNCH(k_contour_segments<true, 32><<<grid, kThreads, 0, st>>>(b, sample));
        else PF_LAUNCH(k_contour_segments<false, 32><<<grid, kThreads, 0, st>>>(b, sample));
    }
    return cudaGetLastError();
}

// The warp-shared flattening runs as many blocks as fit on every SM (they take segments by
// ticket).  Groups of 32 segments, or of the power of two below that leaves 8 groups to every
// resident warp (20,000 paths, 700,000 segments: 0.48 ms of flattening with 16 groups a warp, 0.46
// with 8, 0.49 with 4; 240 paths, 4,000 segments, one to a group: 0.13 ms with one lane per
// segment -> 0.066).
template <int kMode>
static cudaError_t launch_flatten_pool(const Batch &b, uint32_t n_segs, cudaStream_t st) {
    int dev = 0, sms = 152, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (const cudaError_t e =
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_flatten_pool<kMode>, kPoolWarps * 32, 0))
        return e;
    const uint64_t resident = uint64_t(std::max(1, per_sm)) * uint64_t(sms);
    int shift = 0;
    while (shift < 5 && (uint64_t(16) << shift) * resident * kPoolWarps <= n_segs) shift++;
    const uint64_t groups = ((uint64_t(n_segs) - 1) >> shift) + 1;
    const uint64_t blocks = std::min<uint64_t>(resident, (groups + kPoolWarps - 1) / kPoolWarps);
    PF_LAUNCH(k_flatten_pool<kMode><<<(unsigned)blocks, kPoolWarps * 32, 0, st>>>(b, n_segs, shift));
    return cudaGetLastError();
}

// Exact frame.  Segments that bisect deeply are shared by the lanes of a warp; where nearly all are
// shallow (under 1 in 1,024 of the sampled ones takes more than 8 lines), one segment per thread keeps
// more of them in flight (count and write pass with their segments, GB300: 150,000 glyphs, none
// deep, 0.22 ms against 0.36 shared; stroked batch, 1.8 lines per segment but between 1 in 64 and 1 in
// 256 deep, 0.69 against 0.57; 20,000 paths, 25 per segment, 0.80 against 0.44).
cudaError_t launch_flatten(const Batch &b, uint32_t n_segs, bool write, bool shallow, cudaStream_t st) {
    if (!n_segs) return cudaSuccess;
    if (!shallow)
        return write ? launch_flatten_pool<kPoolWrite>(b, n_segs, st) : launch_flatten_pool<kPoolCount>(b, n_segs, st);
    if (write) PF_LAUNCH(k_flatten<true><<<grid_for(n_segs), kThreads, 0, st>>>(b, n_segs));
    else PF_LAUNCH(k_flatten<false><<<grid_for(n_segs), kThreads, 0, st>>>(b, n_segs));
    return cudaGetLastError();
}

cudaError_t launch_flatten_budget(const Batch &b, uint32_t n_segs, cudaStream_t st) {
    if (!n_segs) return cudaSuccess;
    return launch_flatten_pool<kPoolLearned>(b, n_segs, st);
}

cudaError_t launch_bin_lists(const Batch &b, bool learned, const StatusCopy &copy, cudaStream_t st) {
    if (b.n_paths <= kOneBlockPaths) {
        PF_LAUNCH(k_bin_lists<<<1, kOneBlockThreads, 0, st>>>(b, learned, copy));
    } else {
        PF_LAUNCH(k_bin_classify<<<grid_for(b.n_paths), kThreads, 0, st>>>(b, learned));
        PF_LAUNCH(k_bin_scatter<<<grid_for(b.n_paths), kThreads, 0, st>>>(b, copy));
    }
    return cudaGetLastError();
}

// CTAs of a class that one SM holds.
template <int kCls>
static cudaError_t fused_per_sm(int *per_sm) {
    const size_t smem = class_smem(kCls);
    static std::atomic<uint64_t> configured{0};  // devices the kernel's shared memory is set up on, and
    static std::atomic<int> known[64];           // what fits there
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && (configured.load() >> dev & 1u)) {
        *per_sm = known[dev].load();
        return cudaSuccess;
    }
    e = cudaFuncSetAttribute(k_bin_fused<kCls>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_bin_fused<kCls>, class_threads(kCls), smem);
    if (e != cudaSuccess) return e;
    *per_sm = std::max(1, *per_sm);
    if (dev < 64) {
        known[dev].store(*per_sm);
        configured.fetch_or(uint64_t(1) << dev);
    }
    return cudaSuccess;
}

// Grid of a CTA class: as many CTAs as fit on every SM (they take paths by ticket), or
// per_sm_wanted per SM when that is nonzero and fits; no more than there are paths.
template <int kCls>
static cudaError_t fused_grid(unsigned *grid, uint32_t n_sms, uint32_t n_paths, uint32_t per_sm_wanted) {
    int per_sm = 0;
    const cudaError_t e = fused_per_sm<kCls>(&per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm_wanted) per_sm = std::min(per_sm, (int)per_sm_wanted);
    *grid = std::min((unsigned)per_sm * n_sms, std::max(n_paths, 1u));
    return cudaSuccess;
}

template <int kCls>
static cudaError_t launch_fused(const Batch &b, unsigned grid, cudaStream_t st) {
    PF_LAUNCH(k_bin_fused<kCls><<<grid, class_threads(kCls), class_smem(kCls), st>>>(b));
    return cudaGetLastError();
}

// The small class's grid: as many CTAs as fit on every SM, a path per warp at least.
static cudaError_t small_grid(unsigned *grid, uint32_t n_sms, uint32_t n_paths) {
    static std::atomic<int> per_sm{0};  // the same on every device of the one architecture this is built for
    int n = per_sm.load();
    if (!n) {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_bin_small, kSmallThreads, 0);
        if (e != cudaSuccess) return e;
        per_sm.store(n = std::max(n, 1));
    }
    *grid = std::min((unsigned)n * n_sms, std::max(1u, (n_paths + kSmallWarps - 1) / kSmallWarps));
    return cudaSuccess;
}

// The cluster class's grid: as many clusters as the GPU holds, a path each at least.
static cudaError_t cluster_grid(unsigned *grid, uint32_t n_paths) {
    static std::atomic<uint64_t> configured{0};  // devices the kernel's shared memory is set up on, and
    static std::atomic<int> known[64];           // the clusters that fit there
    int dev = 0, clusters = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 64 && (configured.load() >> dev & 1u)) {
        clusters = known[dev].load();
    } else {
        e = cudaFuncSetAttribute(k_bin_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kClusterCtas);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = kClusterSmem;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kClusterCtas;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if ((e = cudaOccupancyMaxActiveClusters(&clusters, k_bin_cluster, &cfg)) != cudaSuccess) return e;
        clusters = std::max(clusters, 1);
        if (dev < 64) {
            known[dev].store(clusters);
            configured.fetch_or(uint64_t(1) << dev);
        }
    }
    *grid = std::min((unsigned)clusters, std::max(n_paths, 1u)) * kClusterCtas;
    return cudaSuccess;
}

// The grids of the classes that can have paths, and their slices of the stage.  Classes of one stream run
// one after the other and share a slice: on their own streams the cluster class with class 1, and class
// 0 with the small one; all of them in a frame that runs them in turn.  Where there is a class 3, whose
// passes come first on the main stream, the cluster class has a stream of its own: binning of three paths
// of 4,000 long lines, two of them of class 3, 3.86 -> 2.53 ms, of 100 quadrilaterals on 6,000 px 1.93 ->
// 1.82; on class 2's stream it held that up (20,000 paths, 0.66 -> 0.72).  (A slice for each of the five
// classes, whether the frame has it or not: a first frame of 240 paths took 178 MB and 614 us, now 68 MB
// and 550 us, one of 20,000 paths 4.07 ms, now 2.25; later frames are the same.)
cudaError_t bin_launch(const Tuning &t, uint32_t n_sms, const BinClasses &has, bool at_once, BinLaunch &l) {
    cudaError_t e = cudaSuccess;
    if (has.cta[0]) e = fused_grid<0>(&l.cta[0], n_sms, has.cta[0], t.bin_ctas_per_sm[0]);
    if (e == cudaSuccess && has.cta[1]) e = fused_grid<1>(&l.cta[1], n_sms, has.cta[1], t.bin_ctas_per_sm[1]);
    if (e == cudaSuccess && has.cta[2]) e = fused_grid<2>(&l.cta[2], n_sms, has.cta[2], t.bin_ctas_per_sm[2]);
    if (e == cudaSuccess && has.small) e = small_grid(&l.small, n_sms, has.small);
    if (e == cudaSuccess && has.cluster) e = cluster_grid(&l.cluster, has.cluster);
    if (e != cudaSuccess) return e;
    const size_t cluster = size_t(l.cluster) * kClusterWarps * kClusterStage;
    l.cluster_aside = at_once && has.large;
    const size_t own = std::max(size_t(l.cta[1]) * class_stage(1), l.cluster_aside ? 0 : cluster);
    const size_t side0 = size_t(l.cta[2]) * class_stage(2);
    const size_t side1 = std::max(size_t(l.cta[0]) * class_stage(0), size_t(l.small) * kSmallWarps * kSmallSpill);
    if (at_once) {
        l.first[2] = own;
        l.first[0] = l.first_small = own + side0;
        l.slots = own + side0 + side1;
        if (l.cluster_aside) {
            l.first_cluster = l.slots;
            l.slots += cluster;
        }
    } else {
        l.slots = std::max(own, std::max(side0, side1));
    }
    return cudaSuccess;
}

cudaError_t bin_class_max_ctas(int out[3]) {
    cudaError_t e = fused_per_sm<0>(&out[0]);
    if (e == cudaSuccess) e = fused_per_sm<1>(&out[1]);
    if (e == cudaSuccess) e = fused_per_sm<2>(&out[2]);
    return e;
}

// Class 3, the cluster class, the CTA classes, largest rects first, and the small class, those that can
// have paths; at once (bs not null) on streams of their own, joined before the composite, so that the
// block scheduler fills the SMs that one class's last paths leave idle with the others'.
cudaError_t launch_bin_paths(const Batch &b, const BinLaunch &l, const BinClasses &has, const BinStreams *bs,
                             cudaStream_t st) {
    if (!b.n_paths) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    const int sides = l.cluster_aside ? 3 : 2;
    if (bs) {
        if ((e = cudaEventRecord(bs->fork, st)) != cudaSuccess) return e;
        for (int k = 0; k < sides; k++)
            if ((e = cudaStreamWaitEvent(bs->side[k], bs->fork, 0)) != cudaSuccess) return e;
    }
    if (has.large) {
        PF_LAUNCH(k_bin_zero_large<<<b.n_sms * 2, 256, 0, st>>>(b));
        PF_LAUNCH(k_bin_large<false><<<b.n_sms * 8, kThreads, 0, st>>>(b));
        PF_LAUNCH(k_bin_large_prep<<<b.n_sms * 2, kPrepThreads, 0, st>>>(b));
        PF_LAUNCH(k_bin_large<true><<<b.n_sms * 8, kThreads, 0, st>>>(b));
    }
    auto slice = [&](size_t first) {
        Batch c = b;
        c.stage += first;
        c.stage_tile += first;
        return c;
    };
    cudaStream_t const st2 = bs ? bs->side[0] : st, st0 = bs ? bs->side[1] : st;
    if (has.cluster) {
        PF_LAUNCH(k_bin_cluster<<<l.cluster, kClusterThreads, kClusterSmem, l.cluster_aside ? bs->side[2] : st>>>(
            slice(l.first_cluster)));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (has.cta[2] && (e = launch_fused<2>(slice(l.first[2]), l.cta[2], st2)) != cudaSuccess) return e;
    if (has.cta[1] && (e = launch_fused<1>(slice(l.first[1]), l.cta[1], st)) != cudaSuccess) return e;
    if (has.cta[0] && (e = launch_fused<0>(slice(l.first[0]), l.cta[0], st0)) != cudaSuccess) return e;
    if (has.small) {
        PF_LAUNCH(k_bin_small<<<l.small, kSmallThreads, 0, st0>>>(slice(l.first_small)));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    for (int k = 0; bs && k < sides; k++) {
        if ((e = cudaEventRecord(bs->join[k], bs->side[k])) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(st, bs->join[k], 0)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_pool_lists(const Batch &b, bool scatter, cudaStream_t st) {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (scatter) PF_LAUNCH(k_pool_scatter<<<sms * 2, kThreads, 0, st>>>(b));
    else PF_LAUNCH(k_pool_count<<<sms * 2, kThreads, 0, st>>>(b));
    return cudaGetLastError();
}

// Status words to pinned host memory by a kernel rather than a copy-engine transfer, so a
// frame's readback never queues behind a large device-to-host copy (pf_read_images_async).
__global__ void k_copy_words(uint32_t *dst, const uint32_t *src, uint32_t n) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

cudaError_t launch_copy_words(uint32_t *dst, const uint32_t *src, uint32_t n, cudaStream_t st) {
    if (n) PF_LAUNCH(k_copy_words<<<1, 64, 0, st>>>(dst, src, n));
    return cudaGetLastError();
}

// Small device reads (totals, flags, per-scene bounds) into mapped host memory the same way.
__global__ void k_copy_bytes(uint8_t *dst, const uint8_t *src, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[i];
}

__global__ void k_gather_words(uint32_t *dst, WordSources s) {
    if (threadIdx.x < s.n) dst[threadIdx.x] = *s.p[threadIdx.x];
}

// Spreads a mapped host buffer over device buffers.  Bound by the link's latency and rate; 16 bytes a
// thread, so that even a small upload has all its reads in flight.
__global__ void __launch_bounds__(256) k_unstage(const uint8_t *src, CopySegs c) {
    const uint32_t step = gridDim.x * blockDim.x * 16u, end = c.s[c.n - 1].end;
    uint32_t k = 0;
    for (uint32_t at = (c.s[0].first & ~15u) + (blockIdx.x * blockDim.x + threadIdx.x) * 16u; at < end; at += step) {
        while (c.s[k].end <= at) k++;  // ends: the last range's end is above at
        const uint32_t lo = max(at, c.s[k].first), hi = min(at + 16u, c.s[k].end);
        uint8_t *const dst = c.s[k].dst + ((int64_t)at - (int64_t)c.s[k].first);
        if (hi - lo == 16u && lo < hi) {
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(src + at);
        } else {
            for (uint32_t i = lo; i < hi; i++) dst[i - at] = src[i];
        }
    }
}

cudaError_t launch_unstage(const uint8_t *src, const CopySegs &c, cudaStream_t st) {
    if (!c.n) return cudaSuccess;
    const uint32_t units = (c.s[c.n - 1].end - (c.s[0].first & ~15u) + 15) / 16;
    PF_LAUNCH(k_unstage<<<std::min<uint32_t>((units + 255) / 256, 1216), 256, 0, st>>>(src, c));
    return cudaGetLastError();
}

cudaError_t launch_copy_bytes(uint8_t *dst, const uint8_t *src, uint32_t n, cudaStream_t st) {
    if (n) PF_LAUNCH(k_copy_bytes<<<std::min<uint32_t>((n + 255) / 256, 64), 256, 0, st>>>(dst, src, n));
    return cudaGetLastError();
}

cudaError_t launch_gather_words(uint32_t *dst, const WordSources &s, cudaStream_t st) {
    if (s.n) PF_LAUNCH(k_gather_words<<<1, 32, 0, st>>>(dst, s));
    return cudaGetLastError();
}

cudaError_t launch_rows(const Batch &b, bool write, cudaStream_t st) {
    if (!b.n_rblks) return cudaSuccess;
    if (write) PF_LAUNCH(k_rows<true><<<b.n_rblks, kRowThreads, 0, st>>>(b));
    else PF_LAUNCH(k_rows<false><<<b.n_rblks, kRowThreads, 0, st>>>(b));
    return cudaGetLastError();
}

// Grid of the composite: a warp per framebuffer tile, or (ticketed) as many resident blocks as
// fit on every SM.  With no tickets asked for (comp_ticket 0) the frame decides: gradients and clips make
// some tiles many times as long as others, and in a frame of many tiles resident warps that take the next
// one are ahead of the block scheduler's order.  The lines, in tiles per resident warp (20 per SM with
// gradients, 24 with clips): 4 with gradients (4,096 tiles, 1.3 a warp, 0-5% slower with a ticket a tile;
// from 16,384 on, 5 a warp, 4-14% faster; 512 scenes 14.43 -> 12.16 ms), 64 with clips alone (below, from
// 15% slower to 7% faster; from 230,000 tiles on 1-9% faster; 512 scenes 7.63 -> 6.93 ms); without either
// it never pays (64 scenes 0.91 -> 1.03 ms, 512 the same).
template <bool kClip, bool kPaint>
static cudaError_t launch_composite_variant(const Batch &b, cudaStream_t st) {
    Batch c = b;
    const uint64_t resident = uint64_t(comp_warps(kClip, kPaint)) * b.n_sms;
    if (!c.comp_ticket && (kPaint || kClip) && b.n_fb >= resident * (kPaint ? 4 : 64)) c.comp_ticket = 1;
    if (!c.comp_ticket) {
        PF_LAUNCH(k_composite<kClip, kPaint, false><<<grid_for(b.n_fb, kCompWarps), kCompWarps * 32, 0, st>>>(c));
        return cudaGetLastError();
    }
    int dev = 0, sms = 152, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_composite<kClip, kPaint, true>, kCompWarps * 32, 0);
    if (e != cudaSuccess) return e;
    const unsigned grid =
        std::min<unsigned>(grid_for(b.n_fb, kCompWarps), (unsigned)std::max(per_sm, 1) * (unsigned)sms);
    PF_LAUNCH(k_composite<kClip, kPaint, true><<<grid, kCompWarps * 32, 0, st>>>(c));
    return cudaGetLastError();
}

cudaError_t launch_composite(const Batch &b, cudaStream_t st) {
    if (!b.n_fb) return cudaSuccess;
    if (b.path_clip_cat && b.path_grad) return launch_composite_variant<true, true>(b, st);
    if (b.path_clip_cat) return launch_composite_variant<true, false>(b, st);
    if (b.path_grad) return launch_composite_variant<false, true>(b, st);
    return launch_composite_variant<false, false>(b, st);
}

// One block per scene: its framebuffer tiles get its index.
__global__ void k_fb_scene(const uint32_t *scene_fb_first, uint32_t *fb_scene) {
    const uint32_t s = blockIdx.x, a = scene_fb_first[s], e = scene_fb_first[s + 1];
    for (uint32_t t = a + threadIdx.x; t < e; t += blockDim.x) fb_scene[t] = s;
}

cudaError_t launch_fb_scene(const uint32_t *scene_fb_first, uint32_t n_scenes, uint32_t *fb_scene, cudaStream_t st) {
    if (n_scenes) PF_LAUNCH(k_fb_scene<<<n_scenes, kThreads, 0, st>>>(scene_fb_first, fb_scene));
    return cudaGetLastError();
}

cudaError_t launch_tile_counts(const Batch &b, cudaStream_t st) {
    if (b.n_paths) PF_LAUNCH(k_tile_counts<<<b.n_paths, kThreads, 0, st>>>(b));
    return cudaGetLastError();
}

cudaError_t launch_list_dump(const Batch &b, bool write, cudaStream_t st) {
    if (!b.n_fb) return cudaSuccess;
    if (write) PF_LAUNCH(k_list_dump<true><<<grid_for(b.n_fb, kCompWarps), kCompWarps * 32, 0, st>>>(b));
    else PF_LAUNCH(k_list_dump<false><<<grid_for(b.n_fb, kCompWarps), kCompWarps * 32, 0, st>>>(b));
    return cudaGetLastError();
}

cudaError_t launch_clip_dump(const Batch &b, uint32_t n_tiles, uint32_t *state, uint32_t *clip, cudaStream_t st) {
    if (n_tiles && b.path_clip_cat) PF_LAUNCH(k_clip_dump<<<grid_for(n_tiles), kThreads, 0, st>>>(b, n_tiles, state, clip));
    return cudaGetLastError();
}

cudaError_t launch_coverage_dump(const Batch &b, const uint32_t *tiles, uint32_t n, float *out, cudaStream_t st) {
    if (n) PF_LAUNCH(k_coverage_dump<<<grid_for(n, kCompWarps), kCompWarps * 32, 0, st>>>(b, tiles, n, out));
    return cudaGetLastError();
}

}  // namespace pfc
