// bin.cu -- binning of one frame's triangles into target-cell tiles.
//
// The reference visits every sample of every triangle's range in one sequential loop
// (src/rasterizer.rs:69-70).  Here each triangle is listed in the tiles whose depth
// cells it can write: count (setup kernel for small triangles, one warp per large
// triangle here), exclusive scan over tiles, then fill (bin_common.cuh).
#include <algorithm>

#include "bin_common.cuh"
#include "launch.cuh"
#include "newline.cuh"
#include "record.cuh"
#include "sloth_kernels.h"

namespace sloth {

__device__ __forceinline__ Viewport vp_of(const FrameGeom &g)
{
    return Viewport{g.w, g.h, g.image, g.tw, g.th, g.ntx, g.nty, g.pitch};
}

// Warps over the parts of the queued large triangles: warp `warp` of nwarps.
template <bool kFill>
__device__ __forceinline__ void bin_large_items(uint32_t tri_base, const FrameGeom &g, const FrameBuffers &fb,
                                                const BinBuffers &bb, uint32_t warp, uint32_t nwarps)
{
    const int lane = threadIdx.x & 31;
    const uint32_t items = large_items(bb.large_count);
    const Viewport vp = vp_of(g);
    for (uint32_t it = warp; it < items; it += nwarps) {
        uint32_t q, part, nparts;
        if (!large_item(it, bb.large_count, bb.large_cap, q, part, nparts)) break;
        const uint32_t gtri = tri_base + bb.large_queue[q];
        bin_large_warp<kFill>(fb.records + gtri, gtri, vp, bb.tile_count, bb.tile_cursor, bb.entries,
                              bb.capacity, lane, part, nparts);
    }
}

__global__ void __launch_bounds__(256)
bin_count_large_kernel(uint32_t tri_base, FrameGeom g, FrameBuffers fb, BinBuffers bb)
{
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x + pdl_begin()) >> 5;
    bin_large_items<false>(tri_base, g, fb, bb, warp, (gridDim.x * blockDim.x) >> 5);
}

__device__ __forceinline__ SplitParams split_params(const BinBuffers &bb, uint32_t n)
{
    return SplitParams{bb.slice_offset[n + 1], bb.slice_offset[n + 2]};
}

// Exclusive scans of the tile entry counts (tile_count + tile_cursor: the entries with a
// counted slot and the others; offsets[n] = total) and of the raster items per tile, by one
// block, 4096 tiles per step with running carries.  Afterwards tile_count holds each tile's
// entries and tile_cursor the first slot after its counted ones.  A
// first pass sets the split threshold and the light threshold from the mean entries of a
// non-empty tile.  Items are numbered in three classes: split tiles' slices first (they
// start first), then the other tiles in tile order, then light tiles (fewer entries than
// a quarter of the mean: mostly the frame's nearly empty borders) last, so that the last
// wave of a launch is made of short CTAs.  slice_offset[t] is the tile's first item within
// its class; item_offset() adds the class base.
// The counted (tile_count) and other (tile_cursor) entries of tiles i0..i0+3, 0 past n;
// 16-byte loads when all four exist (i0 is a multiple of 4 and the arrays 16-byte aligned).
__device__ __forceinline__ void load_counts4(const BinBuffers &bb, uint32_t n, uint32_t i0, uint32_t c1[4],
                                             uint32_t c2[4])
{
    if (i0 + 4 <= n) {
        const uint4 a = *reinterpret_cast<const uint4 *>(bb.tile_count + i0);
        const uint4 b = *reinterpret_cast<const uint4 *>(bb.tile_cursor + i0);
        c1[0] = a.x; c1[1] = a.y; c1[2] = a.z; c1[3] = a.w;
        c2[0] = b.x; c2[1] = b.y; c2[2] = b.z; c2[3] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            c1[k] = i0 + k < n ? bb.tile_count[i0 + k] : 0u;
            c2[k] = i0 + k < n ? bb.tile_cursor[i0 + k] : 0u;
        }
    }
}

__global__ void __launch_bounds__(1024) bin_scan_kernel(uint32_t n, BinBuffers bb)
{
    constexpr int kV = 4;   // running sums: entries, split items, other items, light items
    __shared__ unsigned long long red_e[32];
    __shared__ uint32_t red_t[32];
    __shared__ uint32_t ws[kV][32];
    __shared__ uint32_t carry[kV];
    __shared__ SplitParams sp_s;
    __shared__ uint32_t light_s;
    const uint32_t tid = threadIdx.x + pdl_wait();   // its dependents would wait on the whole GPU meanwhile
    const int lane = tid & 31, wid = tid >> 5;
    // pass 1: entries and non-empty tiles, four consecutive tiles per thread and step as in
    // pass 2; the first step's counts stay in registers for pass 2
    unsigned long long se = 0;
    uint32_t st = 0;
    uint32_t c1_0[4], c2_0[4];
    for (uint32_t base = 0; base < n; base += 4 * 1024) {
        uint32_t c1[4], c2[4];
        load_counts4(bb, n, base + 4 * tid, c1, c2);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (base == 0) {
                c1_0[k] = c1[k];
                c2_0[k] = c2[k];
            }
            const uint32_t c = c1[k] + c2[k];   // counted and other entries
            se += c;
            st += c != 0u;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        se += __shfl_xor_sync(0xffffffffu, se, d);
        st += __shfl_xor_sync(0xffffffffu, st, d);
    }
    if (lane == 0) {
        red_e[wid] = se;
        red_t[wid] = st;
    }
    if (tid < kV) carry[tid] = 0;
    block_sync();
    unsigned long long te = 0;   // thread 0: all entries
    if (tid == 0) {
        uint32_t tt = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            te += red_e[w];
            tt += red_t[w];
        }
        const unsigned long long mean = (te + (tt ? tt : 1u) - 1) / (tt ? tt : 1u);
        // 4x the mean, but low enough that a launch of few tiles still yields about
        // kTargetItems items to spread over the GPU
        unsigned long long thr = mean * 4 < 2 * te / kTargetItems ? mean * 4 : 2 * te / kTargetItems;
        if (thr < kMinSplitEntries) thr = kMinSplitEntries;
        sp_s.threshold = (uint32_t)(thr < 0x40000000ull ? thr : 0x40000000ull);
        sp_s.slice = sp_s.threshold / 2;
        light_s = (uint32_t)(mean / 4 < sp_s.threshold ? mean / 4 : sp_s.threshold);
    }
    block_sync();
    const SplitParams sp = sp_s;
    const uint32_t light = light_s;
    // pass 2: the scans; the next step's counts are on their way while this one's are summed.
    // One block's chain of loads, sums and stores: with those loads after the barriers and
    // 4-byte stores, the scan of the uneven batch's 25k tiles took 40 us, so 20; 2k tiles 9.0
    // and 6.1.
    uint32_t n1[4], n2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        n1[k] = c1_0[k];
        n2[k] = c2_0[k];
    }
    for (uint32_t base = 0; base < n; base += 4 * 1024) {
        const uint32_t i0 = base + 4 * tid;
        uint32_t c[4], c1[4], c2[4], cls[4], ns[4], loc[kV] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            c1[k] = n1[k];
            c2[k] = n2[k];
        }
        if (base + 4 * 1024 < n) load_counts4(bb, n, i0 + 4 * 1024, n1, n2);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            c[k] = c1[k] + c2[k];
            cls[k] = c[k] > sp.threshold ? 1u : (c[k] < light ? 3u : 2u);
            loc[0] += c[k];
            ns[k] = tile_slices(c[k], sp);
#pragma unroll
            for (uint32_t q = 1; q < kV; ++q) loc[q] += cls[k] == q ? ns[k] : 0u;
        }
        uint32_t v[kV];
#pragma unroll
        for (int q = 0; q < kV; ++q) v[q] = loc[q];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
            for (int q = 0; q < kV; ++q) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, v[q], d);
                if (lane >= d) v[q] += o;
            }
        }
        if (lane == 31)
#pragma unroll
            for (int q = 0; q < kV; ++q) ws[q][wid] = v[q];
        block_sync();
        if (wid == 0) {
            uint32_t a[kV];
#pragma unroll
            for (int q = 0; q < kV; ++q) a[q] = ws[q][lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
                for (int q = 0; q < kV; ++q) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, a[q], d);
                    if (lane >= d) a[q] += o;
                }
            }
#pragma unroll
            for (int q = 0; q < kV; ++q) ws[q][lane] = a[q];
        }
        block_sync();
        uint32_t p[kV];
#pragma unroll
        for (int q = 0; q < kV; ++q) p[q] = carry[q] + v[q] - loc[q] + (wid > 0 ? ws[q][wid - 1] : 0u);
        // the first-tile entries take [offset, offset + c1) by their counted slots, the others
        // the slots after them from the cursor
        uint32_t off[4], cur[4], so[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            off[k] = p[0];
            cur[k] = p[0] + c1[k];
            so[k] = cls[k] == 1u ? p[1] : cls[k] == 2u ? p[2] : p[3];
            p[0] += c[k];
#pragma unroll
            for (uint32_t q = 1; q < kV; ++q) p[q] += cls[k] == q ? ns[k] : 0u;
        }
        if (i0 + 4 <= n) {
            *reinterpret_cast<uint4 *>(bb.tile_offset + i0) = make_uint4(off[0], off[1], off[2], off[3]);
            *reinterpret_cast<uint4 *>(bb.tile_cursor + i0) = make_uint4(cur[0], cur[1], cur[2], cur[3]);
            *reinterpret_cast<uint4 *>(bb.tile_count + i0) = make_uint4(c[0], c[1], c[2], c[3]);
            *reinterpret_cast<uint4 *>(bb.slice_offset + i0) = make_uint4(so[0], so[1], so[2], so[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i0 + k < n) {
                    bb.tile_offset[i0 + k] = off[k];
                    bb.tile_cursor[i0 + k] = cur[k];
                    bb.tile_count[i0 + k] = c[k];
                    bb.slice_offset[i0 + k] = so[k];
                }
        }
        block_sync();                    // every thread has read the carries
        if (tid == blockDim.x - 1)
#pragma unroll
            for (int q = 0; q < kV; ++q) carry[q] = p[q];
        block_sync();
    }
    if (tid == 0) {
        bb.tile_offset[n] = entry_total(te);   // carry[0] where that fits
        bb.slice_offset[n] = carry[1] + carry[2] + carry[3];
        bb.slice_offset[n + 1] = sp.threshold;
        bb.slice_offset[n + 2] = sp.slice;
        bb.slice_offset[n + 3] = carry[1];
        bb.slice_offset[n + 4] = carry[1] + carry[2];
        bb.slice_offset[n + 5] = light;
    }
}

// Tile t: the raster items (tile, slice) of the tile, and for a tile that is
// rasterized in slices, its keys cleared (unless they hold keys of earlier draws since
// the clear) and its generation set before the slices fold into them.  When the draw's
// entries outgrew the buffer (the raster folds its triangles without tiles), every tile
// gets that treatment instead.
__device__ __forceinline__ void bin_tile_items(uint32_t t, uint32_t n, const FrameGeom &g, const FrameBuffers &fb,
                                               const BinBuffers &bb)
{
    const bool live = t < n, outgrew = bb.tile_offset[n] > bb.capacity;
    const SplitParams sp = split_params(bb, n);
    const uint32_t cnt = live ? bb.tile_count[t] : 0u;
    if (live && !outgrew) {
        const uint32_t ns = tile_slices(cnt, sp), off = item_offset(bb.slice_offset, n, t, cnt, sp.threshold);
        for (uint32_t k = 0; k < ns && off + k < bb.item_capacity; ++k) bb.items[off + k] = make_uint2(t, k);
    }
    const bool empty = live && (outgrew || cnt > sp.threshold) && fb.tile_gen[t] != fb.gen;
    const int tr = (int)t / g.ntx, tc = (int)t - tr * g.ntx;
    empty_tiles_warp(empty, fb.keys + (size_t)tr * g.th * g.pitch + (size_t)tc * g.tw, g);
    if (empty) fb.tile_gen[t] = fb.gen;
}

// A fill's blocks, part after part: newline chunks, large triangles, tiles' raster items,
// the rest the small triangles.  The parts read what setup and the scan left and do not
// touch each other, so they share one launch: as four launches on three streams, with the
// events between them, they and the waits around them left the GPU idle for a tenth of a
// frame of a million triangles.  The longest blocks start first.
struct FillParts {
    uint32_t newline, large, items;
};

__global__ void __launch_bounds__(kSetupThreads, kFillMinBlocks)
bin_fill_kernel(uint32_t ntri, const uint32_t *__restrict__ order, uint32_t tri_base, uint32_t ntiles, FrameGeom g,
                FrameBuffers fb, BinBuffers bb, FillParts parts)
{
    extern __shared__ int32_t stree[];
    uint32_t blk = blockIdx.x + pdl_begin();
    if (blk < parts.newline) {
        const uint32_t lo = blk * kNewlineFillChunk;
        newline_block<true>(stree, g.nl_size, lo, min(ntri, lo + kNewlineFillChunk), order, fb.rows + tri_base, tri_base,
                            fb.nltree);
        return;
    }
    blk -= parts.newline;
    if (blk < parts.large) {
        bin_large_items<true>(tri_base, g, fb, bb, (blk * blockDim.x + threadIdx.x) >> 5,
                              (parts.large * blockDim.x) >> 5);
        return;
    }
    blk -= parts.large;
    if (blk < parts.items) {
        bin_tile_items(blk * blockDim.x + threadIdx.x, ntiles, g, fb, bb);
        return;
    }
    blk -= parts.items;
    // the small triangles setup listed
    const uint32_t n = bb.large_count[2], step = (gridDim.x - parts.newline - parts.large - parts.items) * blockDim.x;
    for (uint32_t i = blk * blockDim.x + threadIdx.x; i < n; i += step) {
        const uint4 e = bb.fill_list[i];
        const uint32_t meta = bb.fill_meta[i];
        if (!(meta & kFillReread)) {
            fill_listed(e, meta, bb.tile_offset, bb.tile_cursor, bb.entries, bb.capacity);
        } else {
            const Viewport vp = vp_of(g);
            const TriRecord r = load_record(fb.records, e.x);
            fill_small(r, e.x, vp, tile_span(vp, r), bb.tile_offset, bb.tile_cursor, bb.entries, bb.capacity, e.y, 0u);
        }
    }
}

cudaError_t launch_bin_count_large(uint32_t tri_base, const FrameGeom &g, const FrameBuffers &fb,
                                   const BinBuffers &bb, cudaStream_t s)
{
    // up to eight CTAs of 8 warps per SM; the warps stride over the items
    return launch_pdl(bin_count_large_kernel, dim3(8u * (unsigned)device_sm_count()), dim3(256), 0, s, tri_base, g, fb,
                      bb);
}

cudaError_t launch_bin_scan(uint32_t ntiles, const BinBuffers &bb, cudaStream_t s)
{
    return launch_pdl(bin_scan_kernel, dim3(1), dim3(1024), 0, s, ntiles, bb);
}

bool newline_in_fill(uint32_t ntri, const FrameGeom &g)
{
    return g.image && ntri <= kNewlinePartTriangles && newline_tree_bytes(g.nl_size) <= kNewlinePartBytes;
}

cudaError_t launch_bin_fill(uint32_t ntri, const uint32_t *order, uint32_t tri_base, uint32_t ntiles,
                            const FrameGeom &g, const FrameBuffers &fb, const BinBuffers &bb, cudaStream_t s)
{
    const uint32_t sms = (uint32_t)device_sm_count();
    FillParts parts{};
    parts.newline = newline_in_fill(ntri, g) ? (ntri + kNewlineFillChunk - 1) / kNewlineFillChunk : 0u;
    parts.large = 4u * sms;
    parts.items = (ntiles + kSetupThreads - 1) / kSetupThreads;
    const uint32_t small = std::min(2u * kFillMinBlocks * sms, (ntri + kSetupThreads - 1) / kSetupThreads);
    const size_t smem = parts.newline ? newline_tree_bytes(g.nl_size) : 0;
    return launch_pdl(bin_fill_kernel, dim3(parts.newline + parts.large + parts.items + std::max(small, 1u)),
                      dim3(kSetupThreads), smem, s, ntri, order, tri_base, ntiles, g, fb, bb, parts);
}

}  // namespace sloth
