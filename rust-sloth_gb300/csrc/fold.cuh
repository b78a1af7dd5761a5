// fold.cuh -- drawing without tiles: every triangle's samples folded straight into the
// frame's global depth keys.
//
// The tile raster (raster_common.cuh) pays for itself when the samples are many: a tile
// count, a scan, an entry per triangle and tile, a sort and a walk per tile, in six or
// seven launches that each wait for the one before.  A draw of a few thousand triangles over few
// samples is all launches.  Here it takes two: fold_triangles sets up 32 triangles per
// block and walks their samples (direct.cuh) with every warp of the block, and queues the
// triangles of more than kFoldBlockSamples samples; fold_queue_walk walks those with the
// warps of the whole GPU.  The minimum of a cell's keys does not depend on the order of
// the folds, so the frame is the tile raster's bit for bit.  The newline rows go straight
// into the frame's segment tree, whose nodes are maxima.
//
// Every tile's keys must be current (cleared or written since the clear) before the folds.
#pragma once

#include "fold_items.h"
#include "raster_common.cuh"
#include "record.cuh"

namespace sloth {

// Triangles a block sets up (one per lane of its first warp).
constexpr int kFoldTris = 32;
// Triangles of more samples than this (rows times walked columns) are queued: the block
// that set one up would walk it alone while the rest of the GPU is idle.
constexpr uint32_t kFoldBlockSamples = 128;
// A queued triangle is cut into items of every parts-th group of rows: kFoldParts groups of
// kFoldRows for the large ones (one group each up to 1024 rows), kFoldMidParts of kFoldMidRows
// for those of at most kFoldWarpSamples samples, or, when there is one for every warp, one item
// of all their rows, 32 at a time.  Items are numbered part after part and a warp's lanes
// look at 32 of them at once, so the items past a triangle's last row cost next to nothing.
// The walk is as long as its longest item, so a large one's groups are small, where the others'
// would only be more items (rows of a group, large / other: 8 / 8, 4 / 4, 2 / 4, 2 / 8; us a
// frame of 16 models at 1280x720 205, 182, 171, 163; of 10 of 5k at 1149x567 180, 180, 181,
// 159; of 20k triangles at 640x360 27.8, 24.9, 23.5, 23.3).
// A warp walks kFoldUnroll steps of 32 samples at once: the row searches, edge values and
// key loads of a step are one chain, and the walk waits on its latency.
constexpr uint32_t kFoldWarpSamples = 4096;
constexpr int kFoldRows = 2, kFoldMidRows = 8;
constexpr int kFoldUnroll = 4;

// With more queued triangles than this, cells that already hold a nearer key are left out
// before the reduction (they may overdraw each other many times); with fewer, the load
// would only lengthen each step.
constexpr uint32_t kFoldFilterMin = 512;

// Dynamic shared memory of a fold block: one direct stage and each lane's triangle's first
// sample (-1: none), and the samples of all.
constexpr size_t kFoldSmemBytes = (kDirectStageWords + 33) * 4;

// Triangles too large for their block: draw index and frame (batches; null otherwise), the
// large ones from the front of the cap entries, the others from the back; count[0] and
// count[1] are their numbers.
struct FoldQueue {
    uint32_t *tri;
    uint32_t *frame;
    uint32_t *count;
    uint32_t cap;
};

// Queue slot of a lane's triangle (called by all 32 lanes; -1 for lanes without one).
__device__ __forceinline__ int fold_queue_slot(const FoldQueue &q, bool mid, bool large)
{
    const int lane = threadIdx.x & 31;
    const unsigned ml = __ballot_sync(0xffffffffu, large), mm = __ballot_sync(0xffffffffu, mid);
    if (!(ml | mm)) return -1;
    uint32_t l0 = 0, m0 = 0;
    if (lane == 0) {
        if (ml) l0 = atomicAdd(&q.count[0], (uint32_t)__popc(ml));
        if (mm) m0 = atomicAdd(&q.count[1], (uint32_t)__popc(mm));
    }
    l0 = __shfl_sync(0xffffffffu, l0, 0);
    m0 = __shfl_sync(0xffffffffu, m0, 0);
    const unsigned lt = (1u << lane) - 1u;
    if (large) return (int)(l0 + __popc(ml & lt));
    if (mid) return (int)(q.cap - 1u - (m0 + __popc(mm & lt)));
    return -1;
}

// How a triangle that build_record kept is walked: by its block (mine), by one warp (mid) or
// by many (large).  A triangle the direct walk does not size (no edge of dy > 0,
// non-finite, or more than 2^31 samples) is left to the row walk.
struct FoldClass {
    bool mine, mid, large;
};
__device__ __forceinline__ FoldClass fold_class(const TriRecord &r, const DirectWalk &dw)
{
    const uint64_t walked = (uint64_t)(r.xe + 1 - r.x0) * (uint32_t)(r.y1 - r.y0);
    FoldClass c;
    c.mine = dw.direct && walked <= kFoldBlockSamples;
    c.mid = !c.mine && walked <= kFoldWarpSamples;
    c.large = !c.mine && !c.mid;
    return c;
}

// Newline rows [y0, y1) of draw index v into the frame's tree (nltree_update with
// reductions, which return nothing to wait for).
__device__ __forceinline__ void nltree_reduce(int32_t *tree, int n, int y0, int y1, int32_t v)
{
    auto put = [&](int i) { asm volatile("red.global.max.s32 [%0], %1;" ::"l"(tree + i), "r"(v) : "memory"); };
    int l = y0 + n, r = y1 + n;
    while (l < r) {
        if (l & 1) put(l++);
        if (r & 1) put(--r);
        l >>= 1;
        r >>= 1;
    }
}

// The newline rows of a warp's 32 triangles into the frame's tree.  The tree is a few
// kilobytes that every SM writes, and its reductions queue up at L2: with each triangle's
// own nodes a frame of 82k triangles at 640x360 took 22.3 us, by rows of the warp
// (warp_row_last) 15.9.
__device__ __forceinline__ void nltree_reduce_warp(int32_t *tree, int n, int y0, int y1, int32_t v)
{
    int lo;
    int32_t last;
    if (warp_row_last(y0, y1, v, lo, last)) {
        const int i = n + lo + (int)(threadIdx.x & 31);
        if (last >= 0) asm volatile("red.global.max.s32 [%0], %1;" ::"l"(tree + i), "r"(last) : "memory");
    } else if (y0 < y1) {
        nltree_reduce(tree, n, y0, y1, v);
    }
}

// Positions p0 .. p0+31 of setup's order of the mesh, by a block of kWarps warps: records,
// newline rows, samples folded or the triangle queued.  base: draw index of the mesh's
// first triangle.  Bound by latency at the sizes it serves (the first warp's chain index ->
// vertex -> record, then the walk), so the samples of 32 triangles are spread over kWarps
// warps instead of one.
template <int kWarps>
__device__ __forceinline__ void fold_triangles(const MeshDev &mesh, const Mat4 &M, uint32_t p0, uint32_t base,
                                               const FrameGeom &g, const FrameBuffers &fb, const FoldQueue &queue,
                                               uint32_t frame)
{
    int *starts = reinterpret_cast<int *>(setup_smem + kDirectStageWords);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (wid == 0) {
        const uint32_t p = p0 + lane;
        FoldClass c{false, false, false};
        int4 row4 = make_int4(0, 0, 0, 0);
        uint32_t gtri = 0;
        DirectWalk dw{false, 0, 0u};
        TriRecord r;
        if (p < mesh.ntri) {
            const uint32_t t = mesh_triangle(mesh, p);
            gtri = base + t;
            uint32_t i1, i2, i3;
            mesh_corners(mesh, p, t, i1, i2, i3);
            const float4 p1 = transform_vertex(mesh, M, i1), p2 = transform_vertex(mesh, M, i2),
                         p3 = transform_vertex(mesh, M, i3);
            const uint32_t rgb = load_rgb(mesh.rgb, t);
            const bool keep = needs_setup(p1, p2, p3, g.w, g.h, row4);
            if (keep) {
                r = build_record(p1, p2, p3, rgb, g.w, g.h, INT_MAX, &dw);
                if (r.x0 < r.xe) {
                    c = fold_class(r, dw);
                    store_record(fb.records + gtri, r, true);
                }
            }
        }
        if (g.image) nltree_reduce_warp(fb.nltree, g.nl_size, row4.z, row4.w, (int32_t)gtri);
        const int q = fold_queue_slot(queue, c.mid, c.large);
        if (q >= 0) {
            queue.tri[q] = gtri;
            if (queue.frame) queue.frame[q] = frame;
        }
        int start;
        const int n = c.mine ? direct_columns(r, dw.xend, dw.exit_mask) * (r.y1 - r.y0) : 0;
        const int all = direct_stage_warp(c.mine, n, r, gtri, dw.xend, dw.exit_mask, 0u, start);
        starts[lane] = c.mine ? start : -1;
        if (lane == 0) starts[32] = all;
    }
    if (kWarps > 1) block_sync();
    else __syncwarp();
    const int start = starts[lane];
    const uint32_t frags = direct_walk(start >= 0, start, starts[32], wid * 32, kWarps * 32, g.w, g.pitch, g.tw,
                                       reinterpret_cast<unsigned long long *>(fb.keys), 0u);
    add_frags_warp(frags, fb.fragments);
}

// One edge's columns on one row, as edge_row_span, for rows as wide as the frame: past a
// few steps from the estimate (edges of huge coordinates, whose real-valued crossing is
// only a guess) the first column that fails is found by bisection, since the columns that
// pass are a prefix (dy > 0) or a suffix (dy < 0) of the row.
__device__ __forceinline__ void fold_row_span(float dx, float dy, float ax, float ay, float py, int &lo, int &hi)
{
    if (lo >= hi) return;
    auto pass = [&](int x) { return edge_eval(dx, dy, ax, ay, (float)x, py) >= 0.0f; };
    if (dy == 0.0f) {
        if (!pass(lo)) hi = lo;
        return;
    }
    const float cross = ax + __fdividef(fmul(dx, fsub(py, ay)), dy);   // estimate only
    if (dy > 0.0f) {
        int t = (int)fminf(fmaxf(floorf(cross), (float)(lo - 1)), (float)(hi - 1)) + 1;
        for (int k = 0; k < 3 && t < hi && pass(t); ++k) ++t;
        if (t < hi && pass(t)) t = first_true(t + 1, hi, [&](int x) { return !pass(x); });
        hi = t;
    } else {
        int t = (int)fminf(fmaxf(ceilf(cross), (float)lo), (float)hi) - 1;
        for (int k = 0; k < 3 && t >= lo && pass(t); ++k) --t;
        if (t >= lo && pass(t)) t = first_true(lo, t, [&](int x) { return pass(x); }) - 1;
        lo = t + 1;
    }
}

// One warp's share of a queued triangle: the groups of kRows rows part, part + parts, ...,
// each row cut to the columns that can pass all three edges, the spans of a group walked 32
// samples at a time with the exact test for every sample.  With filter, a covered sample
// whose cell already holds a nearer key is dropped before the reduction: the plain load may
// be older than the key in L2, and keys only fall, so it can only keep a sample that was not
// needed.  Returns the covered samples; with kCountKept those the filter did not drop (16k
// triangles over 480x270, 14 covered samples a cell: 22% of them).
template <int kRows, bool kCountKept = true, int kUnroll = kFoldUnroll>
__device__ __forceinline__ uint32_t fold_queued(uint32_t gtri, uint32_t part, uint32_t parts, bool filter,
                                                const FrameGeom &g, const FrameBuffers &fb)
{
    const int lane = threadIdx.x & 31;
    const float4 *rp = reinterpret_cast<const float4 *>(fb.records + gtri);
    const int4 xr = *(reinterpret_cast<const int4 *>(rp) + 4);
    if (xr.z + (int)part * kRows >= xr.w) return 0;
    const float4 q0 = rp[0], q1 = rp[1], q5 = rp[5];
    TriRecord r;
    r.v1x = q0.x; r.v1y = q0.y; r.v2x = q0.z; r.v2y = q0.w; r.v3x = q1.x; r.v3y = q1.y;
    r.dx0 = fsub(r.v3x, r.v2x); r.dy0 = fsub(r.v3y, r.v2y);
    r.dx1 = fsub(r.v1x, r.v3x); r.dy1 = fsub(r.v1y, r.v3y);
    r.dx2 = fsub(r.v2x, r.v1x); r.dy2 = fsub(r.v2y, r.v1y);
    r.v1z = q5.x; r.dz2 = q5.y; r.dz3 = q5.z; r.a = q5.w;
    // the reference's right end (row 4 may hold the shorter end the walk was sized by)
    const int x1 = sat_hi(ceilf(fminf(fmul(fmaxf(r.v1x, fmaxf(r.v2x, r.v3x)), 2.0f), (float)(g.w - 1))));
    const float big = 1e18f;
    const bool finite = fabsf(r.v1x) < big && fabsf(r.v1y) < big && fabsf(r.v2x) < big && fabsf(r.v2y) < big &&
                        fabsf(r.v3x) < big && fabsf(r.v3y) < big;
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(fb.keys);
    uint32_t frags = 0;
    for (int ya = xr.z + (int)part * kRows; ya < xr.w; ya += (int)parts * kRows) {
        int lo = xr.x, hi = lane < kRows && ya + lane < xr.w ? x1 : xr.x;
        if (finite) {
            const float py = (float)(ya + lane);
            fold_row_span(r.dx0, r.dy0, r.v2x, r.v2y, py, lo, hi);
            fold_row_span(r.dx1, r.dy1, r.v3x, r.v3y, py, lo, hi);
            fold_row_span(r.dx2, r.dy2, r.v1x, r.v1y, py, lo, hi);
        }
        const int len = max(hi - lo, 0);
        int end = len;
#pragma unroll
        for (int d = 1; d < kRows; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, end, d);
            if (lane >= d) end += o;
        }
        const int total = __shfl_sync(0xffffffffu, end, kRows - 1), xoff = lo - (end - len);
        for (int base = 0; base < total; base += 32 * kUnroll) {
            int row[kUnroll];   // the rows whose spans end at or before the sample
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) row[u] = 0;
#pragma unroll
            for (int step = kRows / 2; step > 0; step >>= 1)
#pragma unroll
                for (int u = 0; u < kUnroll; ++u)
                    if (__shfl_sync(0xffffffffu, end, row[u] + step - 1) <= base + 32 * u + lane) row[u] += step;
            unsigned long long *kp[kUnroll], key[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const int k = base + 32 * u + lane, y = ya + row[u];
                const int x = k + __shfl_sync(0xffffffffu, xoff, row[u]);
                key[u] = kEmptyKey;
                kp[u] = keys;
                if (k >= total) continue;
                const EdgeVals e = eval_edges(r, (float)x, (float)y);
                if (e.w0 >= 0.0f && e.w1 >= 0.0f && e.w2 >= 0.0f) {
                    ++frags;   // a sample the filter drops is taken off again
                    const float z = interp_z(r.v1z, r.dz2, r.dz3, r.a, e.w1, e.w2);
                    if (z < kFltMax) {
                        const uint32_t nw = 2 * x < g.w ? 1u : 0u;
                        kp[u] = keys + (size_t)(nw ? y : y + 1) * g.pitch + key_col(nw ? 2 * x : 2 * x - g.w, g.tw);
                        key[u] = make_key(z, gtri, nw);
                    }
                }
            }
            if (filter) {
                unsigned long long cur[kUnroll];
#pragma unroll
                for (int u = 0; u < kUnroll; ++u) cur[u] = key[u] != kEmptyKey ? *kp[u] : 0ull;
#pragma unroll
                for (int u = 0; u < kUnroll; ++u)
                    if (key[u] >= cur[u] && key[u] != kEmptyKey) {
                        key[u] = kEmptyKey;
                        if (kCountKept) --frags;
                    }
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                if (key[u] != kEmptyKey) red_min_u64(kp[u], key[u]);
        }
    }
    return frags;
}

// The queued triangles of one frame or many, over the warps of a grid (this is warp `warp` of
// nwarps): frame_of(q) gives the frame of queue entry q as a pair of its geometry and buffers.
// Index: FoldItems.
template <class Index, class FrameOf>
__device__ __forceinline__ uint32_t fold_queue_walk(const FoldQueue &queue, uint32_t warp, uint32_t nwarps,
                                                    FrameOf frame_of)
{
    const int lane = threadIdx.x & 31;
    const uint32_t large = queue.count[0], mid = queue.count[1];
    const bool whole = mid > nwarps;   // a warp for each of the smaller ones
    const FoldItems<Index> items(large, mid, queue.cap, whole);
    const bool filter = large + mid > kFoldFilterMin;
    uint32_t frags = 0;
    for (Index base = warp; base < items.all; base += (Index)32 * nwarps) {
        // lane l holds item base + l*nwarps: neighbouring items go to neighbouring warps
        const Index it = base + (Index)lane * nwarps;
        uint32_t q = 0, part = 0, tri = 0;
        bool live = it < items.all;
        if (live) {
            q = items.entry(it, part);
            tri = queue.tri[q];
            const int4 xr = *(reinterpret_cast<const int4 *>(frame_of(q).fb.records + tri) + 4);
            live = xr.z + (int)part * (it < items.cut ? kFoldRows : kFoldMidRows) < xr.w;
            // a large one's part carries the class (the walk below has no register to spare)
            if (it < items.cut) part |= 0x80000000u;
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, live); todo; todo &= todo - 1u) {
            const int src = __ffs(todo) - 1;
            const uint32_t wq = __shfl_sync(0xffffffffu, q, src), wt = __shfl_sync(0xffffffffu, tri, src),
                           wp = __shfl_sync(0xffffffffu, part, src);
            const auto &f = frame_of(wq);
            if (wp >> 31) frags += fold_queued<kFoldRows>(wt, wp & 0x7fffffffu, kFoldParts, filter, f.g, f.fb);
            else if (!whole) frags += fold_queued<kFoldMidRows>(wt, wp, kFoldMidParts, filter, f.g, f.fb);
            else frags += fold_queued<32>(wt, 0u, 1u, filter, f.g, f.fb);
        }
    }
    return frags;
}

}  // namespace sloth
