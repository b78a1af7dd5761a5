// raster.cu -- per-tile rasterization of one frame (raster_common.cuh), one CTA per tile,
// instantiated for every supported tile shape.
#include "fold.cuh"
#include "launch.cuh"
#include "raster_common.cuh"

namespace sloth {

// Overflow fallback of a draw whose tile entries outgrew the entry buffer (its fill wrote
// what fitted): the warps of the grid fold the covered samples of its binned triangles -- the
// fill list and the large queue hold them all -- straight into the global keys (fold.cuh),
// the same minimum as the tile raster's.  The fill has made every tile's keys current.  Not
// inlined: the raster keeps its registers (its parameters are grid constants, so that
// passing them on copies none).
__device__ __noinline__ void overflow_fold(uint32_t tri_base, const FrameGeom &g, const FrameBuffers &fb,
                                           const BinBuffers &bb)
{
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    uint32_t frags = 0;
    const uint32_t n = bb.large_count[2];
    for (uint32_t i = warp; i < n; i += nwarps) frags += fold_queued<32, false, 1>(bb.fill_list[i].x, 0u, 1u, true, g, fb);
    const OverflowItems items(bb.large_count[0], bb.large_count[1], bb.large_cap);
    for (uint64_t i = warp; i < items.all; i += nwarps) {
        uint32_t part;
        const uint32_t q = items.entry(i, part);
        frags += fold_queued<8, false, 1>(tri_base + bb.large_queue[q], part, kOverflowParts, true, g, fb);
    }
    add_frags_warp(frags, fb.fragments);
}

// One CTA per raster item (tile, slice); CTAs past the item count return at once.  When the
// draw's entries outgrew the buffer, every CTA of the grid takes part in overflow_fold
// instead.
template <int TW, int TH>
__global__ void __launch_bounds__(kRasterThreads, kRasterMinBlocks)
raster_kernel(const __grid_constant__ FrameGeom g, const __grid_constant__ FrameBuffers fb,
              const __grid_constant__ BinBuffers bb, uint32_t ntiles, int depth_cull, uint32_t tri_base)
{
    __shared__ TileSmem<TW, TH> S;
    const uint32_t blk = blockIdx.x + pdl_begin(), total = bb.tile_offset[ntiles];
    if (total > bb.capacity) {
        if (blk == 0 && threadIdx.x == 0 && bb.outgrew) *bb.outgrew = total;
        overflow_fold(tri_base, g, fb, bb);
        return;
    }
    if (blk >= bb.slice_offset[ntiles] || blk >= bb.item_capacity) return;
    const uint2 it = bb.items[blk];
    const uint32_t all = bb.tile_count[it.x];
    const uint32_t thr = bb.slice_offset[ntiles + 1], slice = bb.slice_offset[ntiles + 2];
    const bool split = all > thr;
    const uint32_t first = split ? it.y * slice : 0u;
    const uint32_t cnt = split ? min(slice, all - first) : all;
    uint32_t phase = 0;
    raster_tile<TW, TH>(S, g, fb, (int)it.x, cnt, bb.entries + bb.tile_offset[it.x] + first, depth_cull, phase,
                        split);
}

cudaError_t launch_raster(const FrameGeom &g, const FrameBuffers &fb, const BinBuffers &bb,
                          int depth_cull, uint32_t tri_base, cudaStream_t s)
{
    const uint32_t ntiles = (uint32_t)(g.ntx * g.nty);
    if (ntiles == 0) return cudaSuccess;
    const uint32_t grid = bb.item_capacity;
#define SLOTH_RASTER_CASE(W_, H_)                                                              \
    if (g.tw == W_ && g.th == H_) {                                                            \
        return launch_pdl(raster_kernel<W_, H_>, dim3(grid), dim3(kRasterThreads), 0, s, g, fb, bb, ntiles, \
                          depth_cull, tri_base);                                               \
    }
    SLOTH_TILE_SHAPES(SLOTH_RASTER_CASE)
#undef SLOTH_RASTER_CASE
    return cudaErrorInvalidValue;
}

}  // namespace sloth
