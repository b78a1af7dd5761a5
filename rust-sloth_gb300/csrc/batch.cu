// batch.cu -- kernels of the batched path: many frames (views, meshes, viewports) in one
// pass of each stage, and one persistent raster kernel over a device-side (frame, tile)
// work queue.  Every per-triangle, per-tile and per-cell step is the single-frame one
// (record.cuh, bin_common.cuh, raster_common.cuh, resolve_common.cuh) applied to the
// item's frame, so each frame is bit-identical to drawing it alone.
#include <algorithm>

#include "batch_kernels.h"
#include "bin_common.cuh"
#include "direct.cuh"
#include "fold.cuh"
#include "launch.cuh"
#include "newline.cuh"
#include "raster_common.cuh"
#include "record.cuh"
#include "resolve_common.cuh"

namespace sloth {

__device__ __forceinline__ Viewport vp_batch(const FrameGeom &g)
{
    return Viewport{g.w, g.h, g.image, g.tw, g.th, g.ntx, g.nty, g.pitch};
}

// The three vertices of triangle t of draw d, at position p of setup's order of the mesh,
// transformed by the draw's matrix M in place (the vertex kernel's operations): a mesh
// shared by many views stays in L2, and no transformed-vertex buffer is written and read
// back.
__device__ __forceinline__ void batch_triangle_vertices(const BatchDraw &d, const Mat4 &M, uint32_t p, uint32_t t,
                                                        float4 &p1, float4 &p2, float4 &p3)
{
    uint32_t i1, i2, i3;
    mesh_corners(d.mesh, p, t, i1, i2, i3);
    p1 = transform_vertex(d.mesh, M, i1);
    p2 = transform_vertex(d.mesh, M, i2);
    p3 = transform_vertex(d.mesh, M, i3);
}

// One triangle t of draw d with transformed vertices p1, p2, p3 and packed colour rgb
// (live false: none; every lane of the warp calls it): record, small-triangle tile
// counts, fill list or large queue, and the direct folds of the smallest triangles.
template <bool kDirect>
__device__ __forceinline__ void batch_setup_triangle(const BatchDev &b, const BatchDraw &d, const BatchFrame &f,
                                                     bool live, uint32_t t, float4 p1, float4 p2, float4 p3,
                                                     uint32_t rgb, uint32_t stage)
{
    bool large = false, direct = false;
    DirectWalk dw{false, 0, 0u};
    TriRecord r;
    TileSpan sp{};
    const Viewport vp = vp_batch(f.g);
    if (live) {
        r = build_record(p1, p2, p3, rgb, f.g.w, f.g.h, kDirect ? f.g.direct_max : 0, kDirect ? &dw : nullptr);
        direct = dw.direct;
        if (!direct) sp = tile_span(vp, r);   // a direct triangle is not binned
        // a triangle with nothing to rasterize is never read back here (the fill walks the
        // fill list, the newline the packed rows): its record is not written
        if (direct || sp.ntiles != 0) store_record(f.fb.records + d.local_base + t, r, direct);
        large = sp.large;
    }
    const bool binned = live && !large && !direct && sp.ntiles != 0;
    uint32_t hits;
    const uint32_t slot1 = count_small_tiles_warp(binned, r, vp, sp, b.bb.tile_count + f.tile_off,
                                                  b.bb.tile_cursor + f.tile_off, hits);
    // the fill's work list: one atomic per warp
    const unsigned bm = __ballot_sync(0xffffffffu, binned);
    if (bm) {
        const int lane = threadIdx.x & 31;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(b.fill_count, (uint32_t)__popc(bm));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bm & ((1u << lane) - 1u));
        if (binned) {
            b.bb.fill_list[at] = fill_entry(r, sp, d.local_base + t, slot1, f.tile_off, vp.ntx, d.frame);
            b.bb.fill_meta[at] = fill_meta(sp, hits, vp.ntx);
        }
    }
    if (__any_sync(0xffffffffu, large)) {
        const int q = large_slot(large, sp.ntiles, b.bb.large_count, b.bb.large_cap);
        if (q >= 0) {
            b.bb.large_queue[q] = d.local_base + t;   // frame-local draw index
            b.large_frame[q] = d.frame;
        }
    }
    // the smallest triangles fold their samples into the frame's global keys (direct.cuh)
    if (kDirect && __any_sync(0xffffffffu, direct)) {
        const uint32_t frags = direct_raster_warp(direct, r, d.local_base + t, f.g.w, f.g.pitch, f.g.tw,
                                                  reinterpret_cast<unsigned long long *>(f.fb.keys), dw.xend,
                                                  dw.exit_mask, stage);
        add_frags_warp(frags, f.fb.fragments);
    }
}

// batch_setup_triangle for a frame drawn without tiles (fold.cuh): the record, the samples
// of a small triangle folded by the warp, a larger one queued.
__device__ __forceinline__ void batch_fold_triangle(const BatchDev &b, const BatchDraw &d, const BatchFrame &f,
                                                    bool live, uint32_t t, float4 p1, float4 p2, float4 p3,
                                                    uint32_t rgb, uint32_t stage)
{
    FoldClass c{false, false, false};
    DirectWalk dw{false, 0, 0u};
    TriRecord r;
    if (live) {
        r = build_record(p1, p2, p3, rgb, f.g.w, f.g.h, INT_MAX, &dw);
        if (r.x0 < r.xe) {
            c = fold_class(r, dw);
            store_record(f.fb.records + d.local_base + t, r, true);
        }
    }
    const FoldQueue queue{b.bb.large_queue, b.large_frame, b.bb.large_count, b.bb.large_cap};
    const int q = fold_queue_slot(queue, c.mid, c.large);
    if (q >= 0) {
        queue.tri[q] = d.local_base + t;
        queue.frame[q] = d.frame;
    }
    if (__any_sync(0xffffffffu, c.mine)) {
        const uint32_t frags = direct_raster_warp(c.mine, r, d.local_base + t, f.g.w, f.g.pitch, f.g.tw,
                                                  reinterpret_cast<unsigned long long *>(f.fb.keys), dw.xend,
                                                  dw.exit_mask, stage);
        add_frags_warp(frags, f.fb.fragments);
    }
}

// blocks[i] = (draw, first triangle): b.tpb triangles of the draw in the single-frame
// setup's chunks and two phases (setup.cu): the range and the back-face proof for every
// triangle, the rest of the setup for the ones queued in shared memory with their vertices.
// kFold: every frame is drawn without tiles.
template <bool kDirect, bool kChunks, bool kFold = false>
__global__ void __launch_bounds__(kSetupThreads, kDirect ? kSetupMinBlocks : kFillMinBlocks) batch_setup_kernel(BatchDev b, const int2 *__restrict__ blocks)
{
    __shared__ uint32_t sq_n;
    // the draw's and frame's descriptors in shared memory: read there, their fields are not
    // reloaded from global memory after each of the block's record stores
    __shared__ BatchDraw sd;
    __shared__ BatchFrame sf;
    __shared__ Mat4 sm;
    const int2 blk = blocks[blockIdx.x];
    if (threadIdx.x < 16) sm.m[threadIdx.x] = b.mats[blk.x].m[threadIdx.x];
    const uint32_t cap = (uint32_t)setup_chunk(b.tpb);
    const SetupStash st{cap};
    if (threadIdx.x == 0) {
        sq_n = 0;
        sd = b.draws[blk.x];
        sf = b.frames[sd.frame];
    }
    block_sync();
    const BatchDraw &d = sd;
    const BatchFrame &f = sf;
    const uint32_t t0 = (uint32_t)blk.y, t_end = min(d.mesh.ntri, t0 + (uint32_t)b.tpb);
    uint32_t base = 0;
    for (uint32_t c0 = t0; c0 < t_end; c0 += cap) {
        // two triangles per round, their vertex loads issued together (the same trip count
        // in every lane)
        // (positions p and q of setup's order: triangles tp and tq; the packed rows are
        // stored by position, everything else by triangle)
        for (uint32_t p = c0 + threadIdx.x; p < c0 + cap; p += 2 * blockDim.x) {
            const uint32_t q = p + blockDim.x;
            const bool lt = p < t_end, lu = q < c0 + cap && q < t_end;
            float4 a1, a2, a3, b1, b2, b3;
            uint32_t tp = 0, tq = 0;
            if (lt) {
                tp = mesh_triangle(d.mesh, p);
                batch_triangle_vertices(d, sm, p, tp, a1, a2, a3);
            }
            if (lu) {
                tq = mesh_triangle(d.mesh, q);
                batch_triangle_vertices(d, sm, q, tq, b1, b2, b3);
            }
            int4 row4;
            const bool kt = lt && needs_setup(a1, a2, a3, f.g.w, f.g.h, row4);
            if (lt) f.fb.rows[d.local_base + p] = pack_rows(row4.z, row4.w);
            stash_push(st, &sq_n, base, kt, tp, a1, a2, a3);
            const bool ku = lu && needs_setup(b1, b2, b3, f.g.w, f.g.h, row4);
            if (lu) f.fb.rows[d.local_base + q] = pack_rows(row4.z, row4.w);
            stash_push(st, &sq_n, base, ku, tq, b1, b2, b3);
        }
        block_sync();
        const uint32_t total = sq_n, nq = total - base;
        for (uint32_t q0 = 0; q0 < nq; q0 += blockDim.x) {
            const uint32_t q = q0 + threadIdx.x;
            float4 p1, p2, p3;
            uint32_t rgb = 0, t = 0;
            if (q < nq) {
                t = st.get(q, p1, p2, p3);
                rgb = load_rgb(d.mesh.rgb, t);
            }
            const uint32_t stage = 10u * cap + (threadIdx.x >> 5) * (uint32_t)kDirectStageWords;
            if constexpr (kFold) batch_fold_triangle(b, d, f, q < nq, t, p1, p2, p3, rgb, stage);
            else batch_setup_triangle<kDirect>(b, d, f, q < nq, t, p1, p2, p3, rgb, stage);
        }
        if (!kChunks) break;
        base = total;
        if (c0 + cap < t_end) block_sync();   // the next chunk refills the stash
    }
}

// blocks[i] = (draw, first triangle): 32 triangles of a draw by a block of kWarps warps
// (fold_triangles; few triangles in all, where the spread over blocks counts).
template <int kWarps>
__global__ void __launch_bounds__(32 * kWarps) batch_fold_setup_kernel(BatchDev b, const int2 *__restrict__ blocks)
{
    __shared__ BatchDraw sd;
    __shared__ BatchFrame sf;
    __shared__ Mat4 sm;
    const uint32_t zero = pdl_begin();
    const int2 blk = blocks[blockIdx.x + zero];
    if (threadIdx.x < 16) sm.m[threadIdx.x] = b.mats[blk.x].m[threadIdx.x];
    if (threadIdx.x == 0) {
        sd = b.draws[blk.x];
        sf = b.frames[sd.frame];
    }
    block_sync();
    const FoldQueue queue{b.bb.large_queue, b.large_frame, b.bb.large_count, b.bb.large_cap};
    fold_triangles<kWarps>(sd.mesh, sm, (uint32_t)blk.y, sd.local_base, sf.g, sf.fb, queue, sd.frame);
}

// newline_block of a chunk of a draw.
template <bool kShared>
__device__ __forceinline__ void batch_newline_block(const BatchDev &b, int2 blk, int32_t *stree)
{
    const BatchDraw &d = b.draws[blk.x];
    const BatchFrame &f = b.frames[d.frame];
    const uint32_t lo = (uint32_t)blk.y, hi = min(d.mesh.ntri, lo + b.newline_chunk);
    newline_block<kShared>(stree, f.g.nl_size, lo, hi, d.mesh.order, f.fb.rows + d.local_base, d.local_base,
                           f.fb.nltree);
}

// The queued triangles of every frame (fold_large_kernel), after nnl blocks of newline chunks.
__global__ void __launch_bounds__(256) batch_fold_large_kernel(BatchDev b, const int2 *__restrict__ nl, uint32_t nnl)
{
    extern __shared__ int32_t stree[];
    uint32_t blk = blockIdx.x;
    if (blk < nnl) {
        batch_newline_block<true>(b, nl[blk], stree);
        return;
    }
    blk -= nnl;
    const uint32_t first = (blk * blockDim.x + threadIdx.x) >> 5;
    const FoldQueue queue{b.bb.large_queue, b.large_frame, b.bb.large_count, b.bb.large_cap};
    const uint32_t frags = fold_queue_walk<uint64_t>(queue, first, ((gridDim.x - nnl) * blockDim.x) >> 5,
                                           [&](uint32_t q) -> const BatchFrame & { return b.frames[b.large_frame[q]]; });
    add_frags_warp(frags, b.frames[0].fb.fragments);   // the batch's one counter
}

// Everything a render starts from: counters, tile counts and generations, the newline
// trees, the matrices, and the keys when the setup folds into them.  One launch instead of
// nine memsets and a copy, each of them a node of the graph that the next one waited for.
__global__ void __launch_bounds__(256) batch_reset_kernel(BatchReset r)
{
    const uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t mask = r.half_shift < 63u ? (1ull << r.half_shift) - 1ull : ~0ull;
    const uint4 empty = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (uint64_t i = i0; i < r.nmats; i += step) r.mats[i] = r.mats_host[i];
    if (i0 == 0) {
        r.large_count[0] = r.large_count[1] = 0u;
        *r.fill_count = 0u;
        *r.fragments = 0ull;
    }
    for (uint64_t i = i0; i < r.ntiles; i += step) {
        r.tile_count[i] = r.tile_cursor[i] = 0u;
        r.tile_gen[i] = r.gen;
    }
    for (uint64_t i = i0; i < r.nnl; i += step) r.nltree[i] = -1;
    for (uint64_t v = i0; v < r.n4; v += step)
        r.keys[r.half_shift < 63u ? ((v >> r.half_shift) << (r.half_shift + 1)) | (v & mask) : v] = empty;
}

// blocks[i] = (draw, first triangle of a chunk): the newline rows in a launch of their own.
template <bool kShared>
__global__ void __launch_bounds__(1024) batch_newline_kernel(BatchDev b, const int2 *__restrict__ blocks)
{
    extern __shared__ int32_t stree[];
    batch_newline_block<kShared>(b, blocks[blockIdx.x], stree);
}

// One warp per part of a queued large triangle, any frame: warp `warp` of nwarps.
template <bool kFill>
__device__ __forceinline__ void batch_large_items(const BatchDev &b, uint32_t warp, uint32_t nwarps)
{
    const int lane = threadIdx.x & 31;
    const uint32_t items = large_items(b.bb.large_count);
    for (uint32_t it = warp; it < items; it += nwarps) {
        uint32_t q, part, nparts;
        if (!large_item(it, b.bb.large_count, b.bb.large_cap, q, part, nparts)) break;
        const BatchFrame &f = b.frames[b.large_frame[q]];
        const uint32_t gtri = b.bb.large_queue[q];
        bin_large_warp<kFill>(f.fb.records + gtri, gtri, vp_batch(f.g), b.bb.tile_count + f.tile_off,
                              b.bb.tile_cursor + f.tile_off, b.bb.entries, b.bb.capacity, lane, part, nparts);
    }
}

__global__ void __launch_bounds__(256) batch_count_large_kernel(BatchDev b)
{
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    batch_large_items<false>(b, warp, (gridDim.x * blockDim.x) >> 5);
}

__device__ __forceinline__ uint32_t frame_of_tile(const BatchDev &b, uint32_t tile)
{
    // last frame whose first tile is <= tile
    uint32_t lo = 0, hi = b.nframes;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (b.frame_tile_off[mid] <= tile) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Global tile t: the tile's raster items (tile, slice); a tile rasterized in
// slices gets its keys cleared and its generation set first (bin_tile_items, per frame),
// and so does every tile when the entries outgrew their buffer (batch_overflow_fold).
__device__ __forceinline__ void batch_tile_items(const BatchDev &b, uint32_t t)
{
    const uint32_t nt = b.total_tiles;
    const bool live = t < nt, outgrew = b.bb.tile_offset[nt] > b.bb.capacity;
    const SplitParams sp{b.bb.slice_offset[nt + 1], b.bb.slice_offset[nt + 2]};
    const uint32_t cnt = live ? b.bb.tile_count[t] : 0u;
    if (live) {
        const uint32_t ns = tile_slices(cnt, sp), off = item_offset(b.bb.slice_offset, nt, t, cnt, sp.threshold);
        for (uint32_t k = 0; k < ns && off + k < b.bb.item_capacity; ++k) b.bb.items[off + k] = make_uint2(t, k);
    }
    bool empty = live && (cnt > sp.threshold || outgrew);
    const BatchFrame &f = b.frames[empty ? frame_of_tile(b, t) : 0u];
    const uint32_t lt = t - f.tile_off;
    empty = empty && f.fb.tile_gen[lt] != f.fb.gen;
    const int tr = (int)lt / f.g.ntx, tc = (int)lt - tr * f.g.ntx;
    empty_tiles_warp(empty, f.fb.keys + (size_t)tr * f.g.th * f.g.pitch + (size_t)tc * f.g.tw, f.g);
    if (empty) f.fb.tile_gen[lt] = f.fb.gen;
}

// A fill's blocks, part after part (bin_fill_kernel): newline chunks, large triangles, tiles'
// raster items, the rest the small triangles setup listed.  A warp's lanes may hold triangles
// of different frames; their tiles are global tile indices.
struct BatchFillParts {
    uint32_t newline, large, items;
};

__global__ void __launch_bounds__(kSetupThreads, kFillMinBlocks)
batch_fill_kernel(BatchDev b, const int2 *__restrict__ nl, BatchFillParts parts)
{
    extern __shared__ int32_t stree[];
    uint32_t blk = blockIdx.x;
    if (blk < parts.newline) {
        batch_newline_block<true>(b, nl[blk], stree);
        return;
    }
    blk -= parts.newline;
    if (blk < parts.large) {
        batch_large_items<true>(b, (blk * blockDim.x + threadIdx.x) >> 5, (parts.large * blockDim.x) >> 5);
        return;
    }
    blk -= parts.large;
    if (blk < parts.items) {
        const uint32_t t = blk * blockDim.x + threadIdx.x;
        if (t == 0) *b.queue = 0u;   // the persistent raster's item counter
        batch_tile_items(b, t);
        return;
    }
    blk -= parts.items;
    const uint32_t n = *b.fill_count, step = (gridDim.x - parts.newline - parts.large - parts.items) * blockDim.x;
    for (uint32_t i = blk * blockDim.x + threadIdx.x; i < n; i += step) {
        const uint4 e = b.bb.fill_list[i];
        const uint32_t meta = b.bb.fill_meta[i];
        if (!(meta & kFillReread)) {
            fill_listed(e, meta, b.bb.tile_offset, b.bb.tile_cursor, b.bb.entries, b.bb.capacity);
        } else {
            const BatchFrame &f = b.frames[e.z];
            const Viewport vp = vp_batch(f.g);
            const TriRecord r = load_record(f.fb.records, e.x);
            fill_small(r, e.x, vp, tile_span(vp, r), b.bb.tile_offset, b.bb.tile_cursor, b.bb.entries, b.bb.capacity,
                       e.y, f.tile_off);
        }
    }
}

// Raster item i (a tile, or a slice of a split tile, of any frame) of the item list built by
// the fill; false when its key load gave up (raster_tile).
template <int TW, int TH>
__device__ __forceinline__ bool batch_raster_item(TileSmem<TW, TH> &S, const BatchDev &b, uint32_t i, uint32_t &phase)
{
    const uint2 it = b.bb.items[i];
    const BatchFrame &f = b.frames[frame_of_tile(b, it.x)];
    const uint32_t all = b.bb.tile_count[it.x];
    const uint32_t thr = b.bb.slice_offset[b.total_tiles + 1], slice = b.bb.slice_offset[b.total_tiles + 2];
    const bool split = all > thr;
    const uint32_t first = split ? it.y * slice : 0u;
    const uint32_t cnt = split ? min(slice, all - first) : all;
    return raster_tile<TW, TH>(S, f.g, f.fb, (int)(it.x - f.tile_off), cnt,
                               b.bb.entries + b.bb.tile_offset[it.x] + first, b.depth_cull, phase, split);
}

// A render whose entries outgrew their buffer (its fill wrote what fitted) is rasterized
// without tiles: every binned triangle is in the fill list or the large queue, and the
// warps of the grid fold their samples straight into the keys, which the fill has
// made current.  The frames are exact, so nothing has to wait for the count; the host grows
// the buffer before a later render.  Not inlined: the raster keeps its registers.
__device__ __noinline__ void batch_overflow_fold(const BatchDev &b)
{
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    uint32_t frags = 0;
    const uint32_t n = *b.fill_count;
    for (uint32_t i = warp; i < n; i += nwarps) {
        const uint4 e = b.bb.fill_list[i];
        const BatchFrame &f = b.frames[(b.bb.fill_meta[i] & kFillReread) ? e.z : frame_of_tile(b, e.w)];
        frags += fold_queued<32, false, 1>(e.x, 0u, 1u, true, f.g, f.fb);
    }
    const OverflowItems items(b.bb.large_count[0], b.bb.large_count[1], b.bb.large_cap);
    for (uint64_t i = warp; i < items.all; i += nwarps) {
        uint32_t part;
        const uint32_t q = items.entry(i, part);
        const BatchFrame &f = b.frames[b.large_frame[q]];
        frags += fold_queued<8, false, 1>(b.bb.large_queue[q], part, kOverflowParts, true, f.g, f.fb);
    }
    add_frags_warp(frags, b.frames[0].fb.fragments);
}

// Raster over every frame's tiles in one launch.  Persistent form (the default): a grid of
// SMs x resident CTAs, each CTA taking the next item of the device-side (frame, tile)
// queue -- the item list, split tiles' slices first -- from a counter (b.queue, zeroed by
// the fill) until the queue is empty.  The item is claimed by thread 0 and read
// by every thread after a barrier, so the whole CTA leaves the loop together.  The other
// form launches one CTA per item and leaves the balancing to the hardware block scheduler.
template <int TW, int TH, bool kPersistent>
__global__ void __launch_bounds__(kRasterThreads, kRasterMinBlocks) batch_raster_kernel(BatchDev b)
{
    __shared__ TileSmem<TW, TH> S;
    __shared__ uint32_t s_item;
    const uint32_t blk = blockIdx.x;
    if (b.bb.tile_offset[b.total_tiles] > b.bb.capacity) {
        if (blk == 0 && threadIdx.x == 0) b.status[0] = 1;
        batch_overflow_fold(b);
        return;
    }
    const uint32_t nitems = min(b.bb.slice_offset[b.total_tiles], b.bb.item_capacity);
    if (!kPersistent && blk >= nitems) return;
    uint32_t phase = 0;
    if (!kPersistent) {
        if (!batch_raster_item<TW, TH>(S, b, blk, phase) && threadIdx.x == 0) b.status[1] = 1;
        return;
    }
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(b.queue, 1u);
        block_sync();
        const uint32_t i = s_item;   // thread 0 writes the next claim only after raster_tile's last barrier
        if (i >= nitems) break;
        if (!batch_raster_item<TW, TH>(S, b, i, phase)) {
            if (threadIdx.x == 0) b.status[1] = 1;
            break;
        }
    }
}

// blocks[i] = (frame, first cell): runs of kBatchRun frame cells per lane (resolve_run),
// written with one store per buffer when the frame's outputs are aligned.  Eight resident
// blocks per SM (32 registers): the winners' record loads are latency-bound, and the warps
// that wait on them at once count more than the loads each has in flight (uneven batch:
// four blocks with four pairs of cells a thread 297 us, eight blocks with two 229).
constexpr int kBatchRun = 2;
static_assert(kBatchNewlineChunk == kNewlineChunk && kBatchNewlineFillChunk == kNewlineFillChunk, "the same chunks");
static_assert(kFoldBlockTris == kFoldTris, "the host's table steps by the block's triangles");
static_assert(kBatchResolveChunk % (kBatchRun * 256) == 0 && kBatchResolveSmall % (kBatchRun * 256) == 0,
              "whole runs, the same trip count in every warp");

constexpr int kBatchPairs = 2;   // pairs of cells per thread of an even-width frame

// kOdd: the batch has frames of odd width.
template <bool kOdd>
__global__ void __launch_bounds__(256, 8) batch_resolve_kernel(BatchDev b, const int2 *__restrict__ blocks)
{
    // the frame's descriptor in shared memory, a word a thread: read there, its fields are
    // not reloaded from global memory after each of the block's output stores
    __shared__ BatchFrame sf;
    constexpr uint32_t kWords = sizeof(BatchFrame) / 4;
    static_assert(sizeof(BatchFrame) % 4 == 0 && kWords <= 256, "a word a thread");
    const int2 blk = blocks[blockIdx.x];
    if (threadIdx.x < kWords)
        reinterpret_cast<uint32_t *>(&sf)[threadIdx.x] =
            reinterpret_cast<const uint32_t *>(b.frames + blk.x)[threadIdx.x];
    block_sync();
    const BatchFrame &f = sf;
    const uint32_t ncells = frame_cells(f.g), first = (uint32_t)blk.y;
    const uint32_t end = min(ncells - first, b.resolve_chunk) + first;   // chunks start on runs
    if (!kOdd || !(f.g.w & 1)) {
        const uint32_t pend = end / 2 + (end & 1u);
        for (uint32_t p0 = first / 2; p0 < pend; p0 += kBatchPairs * blockDim.x)
            resolve_even<kBatchPairs>(f.g, f.fb, p0 + threadIdx.x, blockDim.x, pend, f.vec != 0);
        return;
    }
    const int lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < b.resolve_chunk / kBatchRun; i += blockDim.x) {
        const uint32_t p = first / kBatchRun + i;
        resolve_run<kBatchRun>(f.g, f.fb, p, kBatchRun * p < end, lane, f.vec != 0);
    }
}

cudaError_t prepare_batch_kernels()
{
    const int bytes = (int)setup_smem_bytes(kMaxTrianglesPerBlock, true);
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(batch_setup_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) ||
        (e = cudaFuncSetAttribute(batch_setup_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) ||
        (e = cudaFuncSetAttribute(batch_setup_kernel<true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) ||
        (e = cudaFuncSetAttribute(batch_setup_kernel<true, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)))
        return e;
    return cudaFuncSetAttribute(batch_newline_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kNewlineSharedBytes);
}

cudaError_t launch_batch_setup(const BatchDev &b, const int2 *blocks, uint32_t nblocks, cudaStream_t s)
{
    if (!nblocks) return cudaSuccess;
    if (!valid_triangles_per_block(b.tpb)) return cudaErrorInvalidValue;
    const size_t smem = setup_smem_bytes(b.tpb, b.direct_max > 0);   // prepare_batch_kernels: above 48 KB
    const bool chunks = b.tpb > kSetupChunk;
    return launch(b.direct_max > 0 ? (chunks ? batch_setup_kernel<true, true> : batch_setup_kernel<true, false>)
                                       : (chunks ? batch_setup_kernel<false, true> : batch_setup_kernel<false, false>),
                      dim3(nblocks), dim3(setup_block_threads(b.tpb)), smem, s, b, blocks);
}

cudaError_t launch_batch_fold_setup(const BatchDev &b, const int2 *blocks, uint32_t nblocks, int warps,
                                    cudaStream_t s)
{
    if (!nblocks) return cudaSuccess;
    if (warps == 4) return launch_pdl(batch_fold_setup_kernel<4>, dim3(nblocks), dim3(128), kFoldSmemBytes, s, b, blocks);
    if (warps == 1) return launch_pdl(batch_fold_setup_kernel<1>, dim3(nblocks), dim3(32), kFoldSmemBytes, s, b, blocks);
    if (!valid_triangles_per_block(b.tpb)) return cudaErrorInvalidValue;
    const size_t smem = setup_smem_bytes(b.tpb, true);
    return launch(b.tpb > kSetupChunk ? batch_setup_kernel<true, true, true> : batch_setup_kernel<true, false, true>,
                      dim3(nblocks), dim3(setup_block_threads(b.tpb)), smem, s, b, blocks);
}

bool batch_newline_part(uint64_t ntri, int max_nl)
{
    return ntri <= kNewlinePartTriangles && newline_tree_bytes(max_nl) <= kNewlinePartBytes;
}

cudaError_t launch_batch_fold_large(const BatchDev &b, const int2 *newline, uint32_t nnewline, int max_nl, cudaStream_t s)
{
    return launch(batch_fold_large_kernel, dim3(nnewline + 4u * (unsigned)device_sm_count()), dim3(256),
                      nnewline ? newline_tree_bytes(max_nl) : 0, s, b, newline, nnewline);
}

cudaError_t launch_batch_reset(const BatchReset &r, cudaStream_t s)
{
    const uint64_t most = std::max<uint64_t>(std::max<uint64_t>(r.nmats, r.ntiles), std::max<uint64_t>(r.nnl, r.n4));
    const uint64_t blocks = std::min<uint64_t>((most + 255) / 256, 16ull * (uint64_t)device_sm_count());
    return launch(batch_reset_kernel, dim3((unsigned)std::max<uint64_t>(blocks, 1)), dim3(256), 0, s, r);
}

cudaError_t launch_batch_newline(const BatchDev &b, const int2 *blocks, uint32_t nblocks, int max_nl,
                                 cudaStream_t s)
{
    if (!nblocks) return cudaSuccess;
    const size_t smem = newline_tree_bytes(max_nl);
    if (smem <= kNewlineSharedBytes)
        return launch(batch_newline_kernel<true>, dim3(nblocks), dim3(1024), smem, s, b, blocks);
    return launch(batch_newline_kernel<false>, dim3(nblocks), dim3(1024), 0, s, b, blocks);
}

cudaError_t launch_batch_count_large(const BatchDev &b, cudaStream_t s)
{
    // eight CTAs of 8 warps per SM; the warps stride over the items
    return launch(batch_count_large_kernel, dim3(8u * (unsigned)device_sm_count()), dim3(256), 0, s, b);
}

cudaError_t launch_batch_fill(const BatchDev &b, const int2 *newline, uint32_t nnewline, int max_nl, cudaStream_t s)
{
    const uint32_t sms = (uint32_t)device_sm_count();
    const BatchFillParts parts{nnewline, 4u * sms, (b.total_tiles + kSetupThreads - 1) / kSetupThreads};
    return launch(batch_fill_kernel, dim3(parts.newline + parts.large + parts.items + 2u * kFillMinBlocks * sms),
                      dim3(kSetupThreads), nnewline ? newline_tree_bytes(max_nl) : 0, s, b, newline, parts);
}

// Resident CTAs per SM of a raster kernel (looked up once per kernel and device).
template <class K>
static int resident_ctas(K kernel)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kRasterThreads, 0) != cudaSuccess || n < 1) n = 1;
    return n;
}

cudaError_t launch_batch_raster(const BatchDev &b, int tw, int th, bool persistent, cudaStream_t s)
{
    if (!b.total_tiles) return cudaSuccess;
    // persistent: SMs x resident CTAs take items from the queue; otherwise one CTA per
    // possible raster item, CTAs past the item count exiting at once
#define SLOTH_BATCH_RASTER_CASE(W_, H_)                                                        \
    if (tw == W_ && th == H_) {                                                                \
        if (persistent) {                                                                      \
            static int per_sm[64];                                                             \
            int dev = 0;                                                                       \
            cudaGetDevice(&dev);                                                               \
            if (dev >= 0 && dev < 64 && !per_sm[dev]) per_sm[dev] = resident_ctas(batch_raster_kernel<W_, H_, true>); \
            const uint32_t slots = (uint32_t)device_sm_count() * (dev >= 0 && dev < 64 ? per_sm[dev] : 1); \
            const uint32_t grid = slots < b.bb.item_capacity ? slots : b.bb.item_capacity;     \
            return launch(batch_raster_kernel<W_, H_, true>, dim3(grid), dim3(kRasterThreads), 0, s, b); \
        }                                                                                      \
        return launch(batch_raster_kernel<W_, H_, false>, dim3(b.bb.item_capacity), dim3(kRasterThreads), 0, s, b); \
    }
    SLOTH_TILE_SHAPES(SLOTH_BATCH_RASTER_CASE)
#undef SLOTH_BATCH_RASTER_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_batch_resolve(const BatchDev &b, const int2 *blocks, uint32_t nblocks, bool odd, cudaStream_t s)
{
    if (!nblocks) return cudaSuccess;
    return launch(odd ? batch_resolve_kernel<true> : batch_resolve_kernel<false>, dim3(nblocks), dim3(256), 0, s, b, blocks);
}

}  // namespace sloth
